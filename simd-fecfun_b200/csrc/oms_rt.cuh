// Layered int8 offset min-sum over run-time code tables: any code shape
// (802.11n/ay, 802.16e, 802.3ca, 5G NR base graphs 1 and 2, ...) and several
// codes in one launch.  The reference's int8 arithmetic bit for bit
// (decode_functions.cpp:11-103, LDPCdecode.cpp:79-201; oms_f16.cuh spells it
// out), with
//   - four codewords per 32-bit word: word v of a quad holds u = P + 128 of
//     posterior v of codewords 0..3, one byte each, and a check message word
//     R + 128 of each.  A row works on them as two f16x2 words (two codewords
//     each): bytes become halves and halves bytes by one byte permutation, and
//     every address, table word, load, store and the syndrome's XOR is shared
//     by four codewords;
//   - the layer loop over tables in shared memory (row weights and
//     circulants), rows as straight-line code (rt_dispatch);
//   - the offset beta8 per layer (a single beta is the reference's case; a
//     table of offsets serves learned offsets);
//   - the check messages in shared memory (RSMEM) or, for large codes, in a
//     per-CTA global scratch area (L2-resident at these sizes);
//   - fewer codewords than a launch has room for go two per word (half quads);
//   - work given as chunks (a job's codeword range): CTA b decodes chunks
//     b, b + grid, ...; within a chunk the persistent slot refill of
//     oms_f16_kernel keeps every slot busy.
//
// What bounds it: the ALU pipe (64 lanes per clock: 22 of a quad's 40 operations
// per edge) at 12-20 warps per SM, and between iterations the latency of the
// syndrome and of the slot phase.  Against two codewords per word and a test per
// edge (73 warp instructions per pair's edge in all, issue 53 %):
//   802.11n 2/3 Z = 81, 33333 codewords   1.55 -> 1.02 ms
//   5G NR base graph 1, Z = 384, 6001     11.5 -> 6.4 ms
//   18 802.11 codes, 50000 each           24.0 -> 15.4 ms
// of which in the same order: four per word 1.55 -> 1.29, constants in registers
// (no change at 12 warps), rows and syndrome by runs of one weight, messages of a
// new codeword masked instead of cleared, counters in registers, 32-bit indices
// 1.29 -> 1.03 (5G: 9.7 -> 7.5), wide loads from global memory 7.5 -> 6.6 (reads of
// finished codewords before refills: 6.7), row instances shared by neighbouring
// weights 6.7 -> 6.4 (802.11 codes: 20.4 -> 15.4).
#pragma once
#include <stddef.h>

#include <type_traits>

#include "msg_areas.cuh"
#include "oms_f16.cuh"

namespace ldpc {

// Offset (half2 bits) and beta = 0 quirk mask of layer l for the two
// codewords of a pair, at iterations it0 (low lane) and it1 (high lane).
__device__ __forceinline__ void rt_offsets(const RtCode& C, int l, int it0, int it1, uint32_t& beta2, uint32_t& quirk) {
    if (!C.beta_tab) {
        beta2 = C.beta2[l];
        quirk = C.quirk2[l];
        return;
    }
    const int last = C.tab_rows - 1;
    const uint32_t b0 = C.beta_tab[(it0 < last ? it0 : last) * C.L + l];
    const uint32_t b1 = C.beta_tab[(it1 < last ? it1 : last) * C.L + l];
    beta2 = b0 | (b1 << 16);
    quirk = (b0 ? 0u : 0x0000d800u) | (b1 ? 0u : 0xd8000000u);
}

// Rows run as straight-line code, one instance per width: f(lo, w) is called
// with the instance of weights lo <= d <= w.  d is the same for every thread of
// the CTA, so the branch is uniform.
//
// A row's code is about 700 bytes per edge, so what an SM executes in an
// iteration may not stay in its instruction caches: a layer that goes to
// another instance than the one before waits for instructions (802.11ad 13/16,
// weights 14, 15 and 16, three layers: 6300 cycles with an instance for every
// two weights, 3700 with one for all three).  Two sets of kernels, so that the
// unused instances of one do not spread the code of the other apart:
//   EXACT   an instance for each weight up to 12: codes whose layers come in runs
//           of a weight (rt_exact)
//   !EXACT  an instance for two neighbouring weights up to 12, four up to 24, eight
//           above, with tests for the edges that not all of them have: other codes
template <int DMAX, bool EXACT, class F>
__device__ __forceinline__ void rt_dispatch(int d, F&& f) {
#define RT_WIDTH(LO, W)                                                                   \
    if constexpr (DMAX >= W) {                                                            \
        if (d <= W) {                                                                     \
            f(std::integral_constant<int, LO>{}, std::integral_constant<int, W>{});       \
            return;                                                                       \
        }                                                                                 \
    }
    if constexpr (EXACT) {
        static_assert(DMAX <= 12);
        RT_WIDTH(2, 2) RT_WIDTH(3, 3) RT_WIDTH(4, 4) RT_WIDTH(5, 5) RT_WIDTH(6, 6) RT_WIDTH(7, 7) RT_WIDTH(8, 8)
        RT_WIDTH(9, 9) RT_WIDTH(10, 10) RT_WIDTH(11, 11) RT_WIDTH(12, 12)
    } else {
        RT_WIDTH(2, 4) RT_WIDTH(5, 6) RT_WIDTH(7, 8) RT_WIDTH(9, 10) RT_WIDTH(11, 12) RT_WIDTH(13, 16)
        RT_WIDTH(17, 20) RT_WIDTH(21, 24) RT_WIDTH(25, 32)
    }
#undef RT_WIDTH
}

// Posterior word of check t in circulant e: tb and zb are t and Z in bytes, Pg
// the quad's posteriors.
__device__ __forceinline__ uint32_t* rt_at(SpEdge e, char* Pg, uint32_t tb, uint32_t zb) {
    const uint32_t w = tb + e.off;
    return reinterpret_cast<uint32_t*>(Pg + (e.col + min(w, w + zb)));
}

// Constants of a row's update, kept in registers: as literals each use of one
// that its instruction cannot encode is a move of its own (5 of 45 operations
// per quad's edge).
struct RtConst {
    uint32_t lo, hi;        // -128, 127
    uint32_t mag;           // 0x64 in every byte
    uint32_t sub, top;      // -0x6500, 255 in both halves
    // zero: 0, of a value that the compiler does not know
    __device__ __forceinline__ explicit RtConst(uint32_t zero)
        : lo(H2_M128 ^ zero), hi(H2_P127 ^ zero), mag(0x64646464u ^ zero), sub(0x9b009b00u ^ zero), top(0x00ff00ffu ^ zero) {}
};

// 1024 + b for two of a word's four bytes (h = 0: bytes 0, 1; h = 1: bytes 2, 3), as f16x2
template <int h>
__device__ __forceinline__ uint32_t rt_widen(uint32_t w, const RtConst& k) {
    return __byte_perm(w, k.mag, h ? 0x4342 : 0x4140);
}

// One row's update for a quad of codewords (d edges from table entry ed, LO <=
// d <= W; messages R[j * rstride], offsets per f16x2 word).  NH = 1: only
// codewords 0 and 1 are in use; bytes 2 and 3 stay at P = R = 0.  fresh: bytes
// of codewords in their first iteration, whose messages count as 0.
//
// All halves are small integers, so half arithmetic on them is exact.  What it
// costs is the ALU pipe (minima, logic and permutations: 64 lanes per clock,
// half the issue rate) beside the half-precision multiply-add pipe (as much),
// so what can be a multiply-add is one:
//   Q = sat8(P - R): (1024 + u) - (1024 + R + 128), then both bounds;
//   the smaller or second value of the row: e = clamp(|Q_j| - mn1, 0, 1) is 0
//     for an edge at the minimum and 1 elsewhere, f_j = c2 + e (c1 - c2), its
//     sign by one logic operation;
//   R' + 1408 has R' + 128 as its low byte, and Q + (R' + 1408) lies in
//     1024..2047, where a half's bits are an integer with unit steps: one
//     integer add-minimum-relu subtracts the bias and applies both bounds of
//     sat8.
template <int LO, int W, bool QUIRK, int NH>
__device__ __forceinline__ void rt_row(const SpEdge* ed, int d, char* Pg, uint32_t* R, int rstride, uint32_t tb, uint32_t zb,
                                       const uint32_t (&beta2)[2], const uint32_t (&quirk)[2], uint32_t maxv2,
                                       uint32_t fresh, const RtConst& k) {
    constexpr uint32_t SGN = 0x80008000u;
    uint32_t* p[W];
    uint32_t q[NH][W];
#pragma unroll
    for (int j = 0; j < W; ++j) {
        const int e = j < LO ? j : min(j, d - 1);
        p[j] = rt_at(ed[e], Pg, tb, zb);
        const uint32_t w = *p[j], r = (R[e * rstride] & ~fresh) | (fresh & 0x80808080u);
        q[0][j] = hmin2(hmax2(hsub2(rt_widen<0>(w, k), rt_widen<0>(r, k)), k.lo), k.hi);
        if (NH == 2) q[NH - 1][j] = hmin2(hmax2(hsub2(rt_widen<1>(w, k), rt_widen<1>(r, k)), k.lo), k.hi);
    }
    uint32_t mn1[NH], f2[NH], df[NH];
#pragma unroll
    for (int h = 0; h < NH; ++h) {
        uint32_t a[W], mn2, sx = 0;
#pragma unroll
        for (int j = 0; j < W; ++j) {
            const bool has = j < LO || j < d;
            if (QUIRK) {
                a[j] = hfma2(heq2(q[h][j], H2_M128), quirk[h], habs2(q[h][j]));
                if (has) sx ^= q[h][j];
            } else {
                a[j] = q[h][j];
            }
            if (!has) a[j] = H2_1024;
        }
        Min2<W>::of(a, mn1[h], mn2);
        if (!QUIRK) sx = mn1[h];
        mn1[h] = habs2(mn1[h]);
        const uint32_t c1 = hmin2(hmax2(hsub2(mn1[h], beta2[h]), H2_ZERO), maxv2);
        const uint32_t c2 = hmin2(hmax2(hsub2(mn2, beta2[h]), H2_ZERO), maxv2);
        f2[h] = c2 ^ (sx & SGN);
        df[h] = hsub2(c1, c2) ^ (sx & SGN);
    }
#pragma unroll
    for (int j = 0; j < W; ++j) {
        uint32_t rb[NH], un[NH];
#pragma unroll
        for (int h = 0; h < NH; ++h) {
            const uint32_t a = QUIRK ? hfma2(heq2(q[h][j], H2_M128), quirk[h], habs2(q[h][j])) : habs2_f(q[h][j]);
            const uint32_t e = hsub2_sat(a, mn1[h]);
            rb[h] = hadd2(hfma2(e, df[h], f2[h]) ^ (q[h][j] & SGN), H2_1408);
            un[h] = __viaddmin_s16x2_relu(hadd2(q[h][j], rb[h]), k.sub, k.top);
        }
        if (j < LO || j < d) {
            *p[j] = NH == 2 ? __byte_perm(un[0], un[NH - 1], 0x6420) : __byte_perm(un[0], 0x80808080u, 0x4420);
            R[j * rstride] = NH == 2 ? __byte_perm(rb[0], rb[NH - 1], 0x6420) : __byte_perm(rb[0], 0x80808080u, 0x4420);
        }
    }
}

// Syndrome of this thread's check rows with early exit (as oms_syndrome), four
// codewords at once: bit 7 of a posterior's byte is set where it is not
// negative, so a check fails where the XOR of its words' bits 7 differs from
// its weight's parity.  all: bits 7 of the bytes in use.  EXACT: two rows of a
// run at a time, so that their loads are in flight together; with short runs the
// code for a row that is left over costs more than that gains (5G NR n1000, 10
// rows: 6300 against 4900 cycles).
template <int DMAX, bool EXACT>
__device__ __forceinline__ void rt_syndrome(const RtCode& C, char* Pg, uint32_t tb, uint32_t zb, uint32_t all, uint32_t* synd) {
    uint32_t seen = 0;
    for (int l = 0; l < C.L;) {
        const int first = C.rw[l], end = C.run[l];
        const SpEdge* ed = C.edge + C.ebase[l];
        rt_dispatch<DMAX, EXACT>(first, [&](auto lo_, auto w_) {
            constexpr int LO = decltype(lo_)::value, W = decltype(w_)::value, STEP = EXACT ? 2 : 1;
            auto row = [&](const SpEdge* t, int d) {
                uint32_t x = (d & 1) ? 0x80808080u : 0u;
#pragma unroll
                for (int j = 0; j < W; ++j) {
                    const uint32_t v = *rt_at(t[j < LO ? j : min(j, d - 1)], Pg, tb, zb);
                    if (j < LO || j < d) x ^= v;
                }
                return x;
            };
            do {
                const int d = LO == W ? W : C.rw[l];
                uint32_t x = STEP == 2 && l + 1 < end ? row(ed, W) | row(ed + W, W) : row(EXACT ? ed : C.edge + C.ebase[l], d);
                x &= all;
                if (x & ~seen) {
                    atomicOr(synd, x);
                    seen |= x;
                }
                if (((seen | *reinterpret_cast<volatile uint32_t*>(synd)) & all) == all) {
                    l = C.L;
                    return;
                }
                ed += STEP * W;
                l += STEP;
            } while (l < end);
            l = end;
        });
    }
}

// Shared memory: [RtCode copy, E circulants of it][posteriors G x stride words][LLR staging 4G x nstage bytes unless
// nostage][messages (E | 1) x blockDim words if RSMEM]
__host__ __device__ constexpr int rt_code_bytes(int E) { return ((int)offsetof(RtCode, edge) + E * (int)sizeof(SpEdge) + 15) & ~15; }

// Where slot k's codeword sits: quad k >> sh, byte k & ((1 << sh) - 1) of its words (sh = 2, or 1 for half quads).
__device__ __forceinline__ int rt_byte(int k, int sh) { return k & ((1 << sh) - 1); }
__device__ __forceinline__ uint8_t* rt_slot(uint32_t* Ps, int stride, int k, int sh) {
    return reinterpret_cast<uint8_t*>(Ps + (k >> sh) * stride) + rt_byte(k, sh);
}

// LLRs st[i] into a slot, from element i0 in steps of `step`: u = P + 128 flips the top bit.
__device__ __forceinline__ void rt_fill(uint8_t* pk, const int8_t* st, int n, int i0, int step) {
#pragma unroll 8
    for (int i = i0; i < n; i += step) pk[4 * i] = (uint8_t)st[i] ^ 0x80u;
}

// The same straight from global memory, four elements per load where the codeword allows it: the
// loads of a 26112-element codeword are under way together (byte by byte their latency was a third
// of 5G NR base graph 1's iteration).
__device__ __forceinline__ void rt_fill_global(uint8_t* pk, const int8_t* src, int n, int i0, int step) {
    if (((reinterpret_cast<unsigned long long>(src) | (unsigned)n) & 3) != 0) {
        rt_fill(pk, src, n, i0, step);
        return;
    }
#pragma unroll 8
    for (int i = 4 * i0; i < n; i += 4 * step) {
        const uint32_t w = __ldg(reinterpret_cast<const uint32_t*>(src + i)) ^ 0x80808080u;
        pk[4 * i] = (uint8_t)w;
        pk[4 * i + 4] = (uint8_t)(w >> 8);
        pk[4 * i + 8] = (uint8_t)(w >> 16);
        pk[4 * i + 12] = (uint8_t)(w >> 24);
    }
}

// A slot's posteriors to memory.
__device__ __forceinline__ void rt_post(int8_t* dst, const uint8_t* pk, int n, int i0, int step) {
#pragma unroll 4
    for (int i = i0; i < n; i += step) dst[i] = (int8_t)(pk[4 * i] ^ 0x80u);
}

// Codeword cw on its way to L2 (slots refilled straight from global memory).
__device__ __forceinline__ void rt_prefetch_l2(const int8_t* llr, long long cw, int n, int lane) {
    const int8_t* src = llr + cw * (long long)n;
    for (int i = 128 * lane; i < n; i += 4096) asm volatile("prefetch.global.L2 [%0];" ::"l"(src + i));
}

// a / b and a mod b, 32-bit where both fit (a third of the 64-bit operation's chain)
__device__ __forceinline__ long long rt_div(long long a, long long b) {
    return ((a | b) >> 32) == 0 ? (long long)((uint32_t)a / (uint32_t)b) : a / b;
}
__device__ __forceinline__ long long rt_mod(long long a, long long b) {
    return ((a | b) >> 32) == 0 ? (long long)((uint32_t)a % (uint32_t)b) : a % b;
}

// Counters of the codewords that one warp writes out, in lane 0's registers
// until the bucket changes (a slot's codewords mostly share one), then to the
// CTA's counters: four shared-memory atomics per bucket instead of per codeword.
struct RtTally {
    int bucket = -1;
    unsigned cws = 0, its = 0, bits = 0, errs = 0;
    __device__ __forceinline__ void flush(unsigned long long (*s_cnt)[4]) {
        if (!cws) return;
        atomicAdd(&s_cnt[bucket][0], (unsigned long long)cws);
        atomicAdd(&s_cnt[bucket][1], (unsigned long long)its);
        if (bits) atomicAdd(&s_cnt[bucket][2], (unsigned long long)bits);
        if (errs) atomicAdd(&s_cnt[bucket][3], (unsigned long long)errs);
        cws = its = bits = errs = 0;
    }
    // a flush every 2^13 codewords at the latest: at most 255 iterations and 2^17 bits each
    __device__ __forceinline__ void add(unsigned long long (*s_cnt)[4], int b, int it, unsigned errw, int cw_errs) {
        if (b != bucket || cws >= 8192) flush(s_cnt);
        bucket = b;
        ++cws;
        its += it;
        bits += errw;
        errs += cw_errs;
    }
};

// Slot phase with the whole CTA on each finished codeword (used when the CTA
// has more warps than codeword slots, where one warp per slot would leave the
// others idle: 5G NR and other long codes).  Every thread derives the same
// set of finished slots from shared state.  Element i of a finished codeword is
// read (hard bit, error, posterior out) by thread i mod blockDim; warp w's lanes
// hold elements 32 (w + m nwarps) + lane, one hard-decision word per ballot.
// With staging buffers that thread then writes the next codeword's LLR i there,
// so no element is read by one thread and overwritten by another.  Without them
// a thread loads four neighbouring LLRs at a time, over elements that others
// read: all finished slots are read first, then, after a barrier, refilled.
// Then, after a barrier, warp k mod nwarps does slot k's bookkeeping, claim
// and prefetch.  Entered after a barrier that follows every thread's
// cp.async wait; the caller commits the prefetches and ends with a barrier.
// it_rd / it_wr: the slots' iteration counts of this iteration parity and of
// the next (-1 = empty slot).
__device__ __forceinline__ void rt_slots_coop(const RtCode& C, const RtJob& job, uint32_t* Ps, int8_t* stage_base, int stride,
                                           int nstage, int nslots, int sh, long long hi, int par, long long* s_cur,
                                           long long* s_next, const int* it_rd, int* it_wr, uint32_t (*s_synd)[16],
                                           uint32_t (*s_zero_mask)[16], int* s_busy, unsigned long long& s_head,
                                           unsigned long long (*s_cnt)[4], unsigned* s_err_bits, unsigned* s_err_slots) {
    const int tid = threadIdx.x, nthr = blockDim.x, warp = tid >> 5, lane = tid & 31, nwarps = nthr >> 5;
    const int n = C.n, z = C.z;
    unsigned fin = 0, refill = 0;   // slots, the same for every thread
    for (int k = 0; k < nslots; ++k) {
        if (s_cur[k] < 0) continue;
        if (!((s_synd[par][k >> sh] >> (8 * rt_byte(k, sh))) & 0x80u) || it_rd[k] + 1 >= C.max_iter) fin |= 1u << k;
    }
    for (unsigned f = fin; f; f &= f - 1) {
        const int k = __ffs(f) - 1;
        const long long cw = s_cur[k];
        uint8_t* pk = rt_slot(Ps, stride, k, sh);
        const uint32_t* ref = job.ref_bits ? job.ref_bits + (cw % job.ref_period) * C.hard_words : nullptr;
        unsigned errw = 0, errslots = 0;
        for (int i0 = warp * 32; i0 < C.kbits; i0 += nthr) {
            const int i = i0 + lane;
            const bool b = (i < C.kbits) && pk[4 * i] < 128;
            const uint32_t word = __ballot_sync(0xffffffffu, b);
            if (lane == 0 && job.hard_out) job.hard_out[cw * C.hard_words + (i0 >> 5)] = word;
            if (ref) {
                uint32_t e = word ^ ref[i0 >> 5];
                if (i0 + 32 > C.kbits) e &= (1u << (C.kbits - i0)) - 1u;
                errw += __popc(e);
                if (C.num_par == 1) {
                    if (e) errslots = 1u;
                } else if ((e >> lane) & 1u) {
                    errslots |= 1u << ((i % z) % C.num_par);
                }
            }
        }
        if (ref && job.counters) {
            errslots = __reduce_or_sync(0xffffffffu, errslots);
            if (lane == 0 && errw) {
                atomicAdd(&s_err_bits[k], errw);
                atomicOr(&s_err_slots[k], errslots);
            }
        }
        if (job.post_out) rt_post(job.post_out + cw * (long long)n, pk, n, tid, nthr);
        if (s_next[k] >= 0) {
            if (C.nostage) refill |= 1u << k;
            else rt_fill(pk, stage_base + k * nstage, n, tid, nthr);
        }
    }
    if (refill) {
        __syncthreads();   // every warp has read the finished posteriors
        for (unsigned f = refill; f; f &= f - 1) {
            const int k = __ffs(f) - 1;
            rt_fill_global(rt_slot(Ps, stride, k, sh), job.llr + s_next[k] * (long long)n, n, tid, nthr);
        }
    }
    // every thread has taken its decision from s_cur / it_rd / s_synd, summed
    // its errors and read the staging buffers before the bookkeeping changes them
    __syncthreads();
    for (int k = warp; k < nslots; k += nwarps) {
        const long long cw = s_cur[k];
        if (cw < 0) {
            if (lane == 0) it_wr[k] = -1;
            continue;
        }
        const int it = it_rd[k] + 1;
        if (!((fin >> k) & 1u)) {
            if (lane == 0) {
                it_wr[k] = it;
                s_busy[par] = 1;
            }
            continue;
        }
        const long long nxt = s_next[k];
        unsigned long long c = 0;
        if (lane == 0) {
            if (job.iters_out) job.iters_out[cw] = (uint8_t)it;
            if (job.counters) {
                int bk = (int)(cw / job.bucket_size);
                bk = bk < job.n_buckets ? bk : job.n_buckets - 1;
                atomicAdd(&s_cnt[bk][0], 1ull);
                atomicAdd(&s_cnt[bk][1], (unsigned long long)it);
                if (s_err_bits[k]) {
                    atomicAdd(&s_cnt[bk][2], (unsigned long long)s_err_bits[k]);
                    atomicAdd(&s_cnt[bk][3], (unsigned long long)__popc(s_err_slots[k]));
                    s_err_bits[k] = 0;
                    s_err_slots[k] = 0;
                }
            }
            if (nxt >= 0) c = atomicAdd(&s_head, 1ull);
        }
        if (nxt >= 0) {
            c = __shfl_sync(0xffffffffu, c, 0);
            const long long fresh = (long long)c < hi ? (long long)c : -1;
            if (fresh >= 0) {
                if (C.nostage) rt_prefetch_l2(job.llr, fresh, n, lane);
                else prefetch_llr(stage_base + k * nstage, job.llr, fresh, n, lane);
            }
            if (lane == 0) {
                s_next[k] = fresh;
                s_busy[par] = 1;
            }
        }
        if (lane == 0) {
            s_cur[k] = nxt;
            it_wr[k] = nxt >= 0 ? 0 : -1;
            atomicOr(&s_zero_mask[par][k >> sh], 0xffu << (8 * rt_byte(k, sh)));
        }
    }
}

template <int DMAX, bool EXACT, bool QUIRK, bool RSMEM>
__global__ void __launch_bounds__(512) oms_rt_kernel(const __grid_constant__ RtLaunch lp) {
    extern __shared__ __align__(16) unsigned char rt_smem[];
    __shared__ long long s_cur[32];
    __shared__ long long s_next[32];
    // iterations done by slot k (-1 = empty), one copy per iteration parity:
    // the slot phase of parity p reads s_it[p] and writes s_it[p ^ 1], so
    // every warp sees the same slot states while others update them
    __shared__ int s_it[2][32];
    __shared__ uint32_t s_synd[2][16];        // per quad: bit 7 of byte k: a check of codeword k fails
    __shared__ uint32_t s_zero_mask[2][16];   // per quad: byte k set: clear the messages of codeword k
    __shared__ int s_busy[2];
    __shared__ unsigned long long s_head;
    __shared__ unsigned long long s_cnt[OMS_MAX_BUCKETS][4];
    __shared__ int s_code_idx;
    __shared__ unsigned s_err_bits[32], s_err_slots[32];   // cooperative write-out: per slot error sums

    const RtCode& C = *reinterpret_cast<const RtCode*>(rt_smem);
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int warp = tid >> 5, lane = tid & 31, nwarps = nthr >> 5;
    const RtConst kc(lp.zero);
    __shared__ int s_area;
    const int area = RSMEM ? 0 : take_area(lp.areas, s_area);
    if (area < 0) return;
    if (tid == 0) s_code_idx = -1;

    const int n_chunks = lp.jobs ? lp.n_chunks : (int)gridDim.x;
    __shared__ int s_claim;
    // chunk b first, then the next unclaimed chunk (batch plans) or chunk
    // b + grid: CTAs that drew cheap chunks take more of them
    auto next_chunk = [&](int ci) -> int {
        if (!lp.claim) return ci + (int)gridDim.x;
        __syncthreads();
        if (tid == 0) s_claim = (int)gridDim.x + (int)atomicAdd(lp.claim, 1u);
        __syncthreads();
        return s_claim;
    };
    for (int ci = blockIdx.x; ci < n_chunks; ci = next_chunk(ci)) {
        // ---------------- chunk set-up ----------------
        RtJob job;
        long long lo, hi;
        if (lp.jobs) {
            const RtChunk ch = lp.chunks[ci];
            job = lp.jobs[ch.job];
            lo = ch.lo;
            hi = ch.hi;
        } else {
            job = lp.job0;
            lo = job.ncw * ci / gridDim.x;
            hi = job.ncw * (ci + 1) / gridDim.x;
        }
        __syncthreads();   // the previous chunk is finished with the shared tables
        if (s_code_idx != job.code) {
            const uint4* src = reinterpret_cast<const uint4*>(lp.codes + job.code);
            uint4* dst = reinterpret_cast<uint4*>(rt_smem);
            const int m = rt_code_bytes(lp.codes[job.code].E) / 16;
            for (int i = tid; i < m; i += nthr) dst[i] = src[i];
            __syncthreads();
            if (tid == 0) s_code_idx = job.code;
        }
        const int z = C.z, n = C.n, G = C.G, stride = C.stride, E = C.E;
        uint32_t* const Ps = reinterpret_cast<uint32_t*>(rt_smem + rt_code_bytes(E));
        const int sh = lp.half ? 1 : 2, nslots = G << sh;
        const uint32_t in_use = lp.half ? 0x00008080u : 0x80808080u;
        const int nstage = C.nostage ? 0 : (n + 15) & ~15;
        int8_t* const stage_base = reinterpret_cast<int8_t*>(Ps) + ((G * stride * 4 + 15) & ~15);
        const int t = tid / G, g = tid - (tid / G) * G;
        const bool active = t < z;
        char* const Pg = reinterpret_cast<char*>(Ps + g * stride);
        const uint32_t tb = 4u * (uint32_t)t, zb = 4u * (uint32_t)z;
        // check messages: in shared memory each thread's E words are contiguous
        // at an odd stride (E | 1, so a warp's 32 lanes fall in 32 banks) and
        // edge j of a layer is the layer's base plus an immediate; the global
        // scratch keeps edge-major words (coalesced)
        const int rstride = RSMEM ? 1 : nthr;
        uint32_t* const Rt = RSMEM ? reinterpret_cast<uint32_t*>(stage_base + nslots * nstage) + tid * (E | 1)
                                   : lp.r_scratch + (long long)area * lp.r_words_per_cta + tid;

        for (int i = tid; i < OMS_MAX_BUCKETS * 4; i += nthr) (&s_cnt[0][0])[i] = 0;
        for (int i = tid; i < G * stride; i += nthr) Ps[i] = 0x80808080u;   // P = 0
        if (tid < 32) {
            const long long c0 = lo + tid, c1 = lo + nslots + tid;
            const bool ok = tid < nslots;
            s_cur[tid] = ok && c0 < hi ? c0 : -1;
            s_next[tid] = ok && c1 < hi ? c1 : -1;
            s_it[0][tid] = ok && c0 < hi ? 0 : -1;
            s_it[1][tid] = -1;
            s_err_bits[tid] = s_err_slots[tid] = 0;
            if (tid < 16) {
                s_synd[0][tid] = s_synd[1][tid] = 0;
                s_zero_mask[0][tid] = s_zero_mask[1][tid] = 0;
            }
            if (tid < 2) s_busy[tid] = 0;
        }
        if (tid == 0) s_head = (unsigned long long)(lo + 2 * nslots);
        __syncthreads();
        // first round through the staging buffers (16-byte copies), then the
        // prefetch of the second round (each warp its own slots)
        if (C.nostage) {
            for (int k = 0; k < nslots; ++k) {
                if (s_cur[k] >= 0) rt_fill_global(rt_slot(Ps, stride, k, sh), job.llr + s_cur[k] * (long long)n, n, tid, nthr);
                if (s_next[k] >= 0 && warp == k % nwarps) rt_prefetch_l2(job.llr, s_next[k], n, lane);
            }
        } else {
            for (int k = warp; k < nslots; k += nwarps)
                if (s_cur[k] >= 0) prefetch_llr(stage_base + k * nstage, job.llr, s_cur[k], n, lane);
            cp_async_commit();
            cp_async_wait_all();
            __syncwarp();
            for (int k = warp; k < nslots; k += nwarps) {
                if (s_cur[k] >= 0) rt_fill(rt_slot(Ps, stride, k, sh), stage_base + k * nstage, n, lane, 32);
                __syncwarp();
                if (s_next[k] >= 0) prefetch_llr(stage_base + k * nstage, job.llr, s_next[k], n, lane);
            }
        }
        cp_async_commit();
        __syncthreads();

        RtTally tally;
        uint32_t fresh = 0xffffffffu;   // bytes whose codeword entered this thread's quad since the last iteration
        for (int par = 0;; par ^= 1) {
            // ---------------- one layered iteration ----------------
            // iteration index of this thread's four codewords (offset tables)
            int its[4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
                its[k] = active && k < (1 << sh) ? max(s_it[par][(g << sh) + k], 0) : 0;
            for (int l = 0; l < C.L;) {
                // a run of layers of one instance
                const int first = C.rw[l], end = C.run[l];
                auto rows = [&](auto lo_, auto w_, auto nh_) {
                    do {
                        if (active) {
                            const int eb = C.ebase[l], d = C.rw[l];
                            uint32_t beta2[2], quirk[2];
                            rt_offsets(C, l, its[0], its[1], beta2[0], quirk[0]);
                            rt_offsets(C, l, its[2], its[3], beta2[1], quirk[1]);
                            rt_row<decltype(lo_)::value, decltype(w_)::value, QUIRK, decltype(nh_)::value>(
                                C.edge + eb, d, Pg, Rt + eb * rstride, rstride, tb, zb, beta2, quirk, C.maxv2, fresh, kc);
                        }
                        __syncthreads();
                    } while (++l < end);
                };
                if (lp.half)
                    rt_dispatch<DMAX, EXACT>(first, [&](auto lo_, auto w_) { rows(lo_, w_, std::integral_constant<int, 1>{}); });
                else
                    rt_dispatch<DMAX, EXACT>(first, [&](auto lo_, auto w_) { rows(lo_, w_, std::integral_constant<int, 2>{}); });
            }
            if (tid < 16) {
                s_synd[par ^ 1][tid] = 0;
                s_zero_mask[par ^ 1][tid] = 0;
            }
            if (tid == 0) s_busy[par ^ 1] = 0;
            if (active) rt_syndrome<DMAX, EXACT>(C, Pg, tb, zb, in_use, &s_synd[par][g]);
            cp_async_wait_all();   // this thread's prefetches (issued in an earlier slot phase)
            __syncthreads();       // syndrome bits final, every prefetched byte visible

            if (nslots < nwarps) {
                // ------- more warps than slots (large codes): the whole CTA writes each
                // finished codeword out and refills its slot -------
                rt_slots_coop(C, job, Ps, stage_base, stride, nstage, nslots, sh, hi, par, s_cur, s_next, s_it[par],
                              s_it[par ^ 1], s_synd, s_zero_mask, s_busy, s_head, s_cnt, s_err_bits, s_err_slots);
            } else {
                // ------- per-warp slots: lane k of every warp evaluates slot k; the
                // finished slots are dealt out in slot order, the j-th to warp
                // j mod nwarps (two codewords finishing together go to different
                // warps) -------
                unsigned done_mask;
                {
                    const int itk = lane < nslots ? s_it[par][lane] : -1;
                    const bool live = itk >= 0;
                    const bool dn = live && (!((s_synd[par][lane >> sh] >> (8 * rt_byte(lane, sh))) & 0x80u) || itk + 1 >= C.max_iter);
                    done_mask = __ballot_sync(0xffffffffu, dn);
                    if (warp == 0 && lane < nslots && !dn) {
                        s_it[par ^ 1][lane] = live ? itk + 1 : -1;
                        if (live) s_busy[par] = 1;
                    }
                }
                int j = 0;
                for (unsigned m = done_mask; m; m &= m - 1, ++j) {
                    if (j % nwarps != warp) continue;
                    const int k = __ffs(m) - 1;
                    const long long cw = s_cur[k];
                    const int it = s_it[par][k] + 1;
                    uint8_t* pk = rt_slot(Ps, stride, k, sh);
                    const uint32_t* ref = job.ref_bits ? job.ref_bits + rt_mod(cw, job.ref_period) * C.hard_words : nullptr;
                    unsigned errw, errslots;
                    warp_hard_decisions<true>([&](int i) { return pk[4 * i] < 128; }, C.kbits,
                                               C.hard_words, z, C.num_par,
                                               job.hard_out ? job.hard_out + cw * C.hard_words : nullptr, ref, lane, errw,
                                               errslots);
                    if (job.post_out) rt_post(job.post_out + cw * (long long)n, pk, n, lane, 32);
                    if (lane == 0 && job.iters_out) job.iters_out[cw] = (uint8_t)it;
                    if (job.counters && lane == 0) tally.add(s_cnt, (int)min(rt_div(cw, job.bucket_size), (long long)job.n_buckets - 1), it, errw, __popc(errslots));
                    __syncwarp();
                    const long long nxt = s_next[k];
                    if (nxt >= 0) {
                        if (C.nostage) rt_fill_global(pk, job.llr + nxt * (long long)n, n, lane, 32);
                        else rt_fill(pk, stage_base + k * nstage, n, lane, 32);
                        __syncwarp();
                        unsigned long long c = 0;
                        if (lane == 0) c = atomicAdd(&s_head, 1ull);
                        c = __shfl_sync(0xffffffffu, c, 0);
                        const long long fresh = (long long)c < hi ? (long long)c : -1;
                        if (fresh >= 0) {
                            if (C.nostage) rt_prefetch_l2(job.llr, fresh, n, lane);
                            else prefetch_llr(stage_base + k * nstage, job.llr, fresh, n, lane);
                        }
                        if (lane == 0) {
                            s_next[k] = fresh;
                            s_busy[par] = 1;
                        }
                    }
                    if (lane == 0) {
                        s_cur[k] = nxt;
                        s_it[par ^ 1][k] = nxt >= 0 ? 0 : -1;
                        atomicOr(&s_zero_mask[par][k >> sh], 0xffu << (8 * rt_byte(k, sh)));
                    }
                }
            }
            cp_async_commit();
            __syncthreads();
            fresh = active ? s_zero_mask[par][g] : 0u;
            if (!s_busy[par]) break;
        }
        cp_async_wait_all();
        if (job.counters) {
            if (lane == 0) tally.flush(s_cnt);
            __syncthreads();
            for (int i = tid; i < job.n_buckets * 4; i += nthr) {
                const unsigned long long v = (&s_cnt[0][0])[i];
                if (v) atomicAdd(job.counters + i, v);
            }
        }
    }
    if (!RSMEM) give_area(lp.areas, s_area);
}

}  // namespace ldpc
