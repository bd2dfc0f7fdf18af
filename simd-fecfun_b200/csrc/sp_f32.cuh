// Layered float decoders: sum-product (tanh / product tree / 2 atanh) and
// offset min-sum, in float (bit-exact with the reference's SIMD_ELEM_BW=-32
// builds LDPCtop_Vec16f_prod / Vec16f_min) and in double (the SIMD_ELEM_BW=-64
// builds LDPCtop_Vec8d_prod / Vec8d_min):
//   Q = P - R                                  decode_functions.cpp:53
//   a = max(|Q| - beta, 0)                     :56-62
//   x = tanh(a/2) (sum-product) or a           min_find.pl:37-41
//   f_j = combine over k != j, fixed tree      min_find.pl:52-164 (gen_trees.cuh)
//         clamped at Max_val, then 2 atanh(.)  min_find.pl:99-107, 44-45
//   R' = f_j with the sign of prod_{k!=j} Q_k  decode_functions.cpp:85-87
//   P  = Q + R'                                :91
// with the oracle's results in the same order (no fused multiply-adds outside
// tanh/atanh, whose branch-free forms in sp_math.cuh equal ldpc_math.h's on
// every argument), so posteriors agree bit for bit.
//
// What bounds it: instruction issue.  802.16e Z = 96 sum-product, 20011
// codewords at Eb/N0 1.5 dB: 11.7 ms with branches and library division, two
// tests and two constant loads per edge (307 warp instructions per edge, issue
// 65 %); 4.45 ms in this form (131 per edge, issue 73 %, ALU 40 %, FMA 42 %,
// reciprocals 22 %).  802.11ad double sum-product, 30000 codewords: 5.5 ->
// 2.9 ms, bound by dependent FP64 chains and instruction fetch (FP64 44 %).
//
// Work layout: G codewords per CTA, one per group of Z threads (thread
// (t, g) = check row t of every layer).  Posteriors in shared memory, check
// messages in shared memory (RSMEM) or, for large codes, in a global scratch
// area; the layer loop runs over run-time tables, so any code shape works.
// The iteration boundary (syndrome, write-out, refill from a prefetched
// staging buffer) follows the int8 kernel.  Codes whose posteriors and
// staging do not both fit shared memory (double, 5G NR base graph 1 at large
// Z) run without the staging buffer (tb.nostage): a finished codeword's slot
// is refilled straight from global memory.
#pragma once
#include <stdint.h>

#include <type_traits>

#include "gen_trees.cuh"
#include "msg_areas.cuh"
#include "sp_math.cuh"
#include "tables.h"
#include "writeout.cuh"

namespace ldpc {

__device__ __forceinline__ void sp_cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void sp_cp_async4(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem) : "memory");
}

__device__ __forceinline__ void sp_cp_async8(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s), "l"(gmem) : "memory");
}

// element operations of the float and double decoders: IEEE round to nearest,
// never contracted into fused multiply-adds
__device__ __forceinline__ float sp_sub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sp_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float sp_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double sp_add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float sp_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double sp_mul(double a, double b) { return __dmul_rn(a, b); }
// max(a, 0) and the lesser of two magnitudes.  sp_max0 turns NaN into 0 as
// "a > 0 ? a : 0" does, so no magnitude is NaN and the hardware minimum (one
// instruction for float) equals "a < b ? a : b".
__device__ __forceinline__ float sp_max0(float a) { return fmaxf(a, 0.0f); }
__device__ __forceinline__ double sp_max0(double a) { return a > 0.0 ? a : 0.0; }
__device__ __forceinline__ float sp_min(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ double sp_min(double a, double b) { return a < b ? a : b; }
__device__ __forceinline__ float sp_abs(float a) { return fabsf(a); }
__device__ __forceinline__ double sp_abs(double a) { return fabs(a); }
// the 32-bit word that holds the sign (bit 31)
__device__ __forceinline__ uint32_t sp_signw(float v) { return __float_as_uint(v); }
__device__ __forceinline__ uint32_t sp_signw(double v) { return (uint32_t)__double2hiint(v); }
// v with its sign flipped where bit 31 of sg is set (sign_combine)
__device__ __forceinline__ float sp_flip(float v, uint32_t sg) { return __uint_as_float(__float_as_uint(v) ^ sg); }
__device__ __forceinline__ double sp_flip(double v, uint32_t sg) {
    return __hiloint2double(__double2hiint(v) ^ (int)sg, __double2loint(v));
}

template <class T>
__device__ __forceinline__ void sp_prefetch(T* stage, const T* llr, long long cw, int n, int lane) {
    constexpr int V = 16 / (int)sizeof(T);   // elements per 16-byte copy
    const T* src = llr + cw * (long long)n;
    const unsigned long long base = reinterpret_cast<unsigned long long>(src);
    if ((n % V) == 0 && (base & 15) == 0) {
        for (int i = V * lane; i < n; i += 32 * V) sp_cp_async16(stage + i, src + i);
    } else if (sizeof(T) == 8) {
        for (int i = lane; i < n; i += 32) sp_cp_async8(stage + i, src + i);
    } else {
        for (int i = lane; i < n; i += 32) sp_cp_async4(stage + i, src + i);
    }
}

// Posterior of check t in circulant e: tb_ and zb are t and Z in bytes, Pg the
// codeword's posteriors.
template <class T>
__device__ __forceinline__ T* sp_at(SpEdge e, char* Pg, uint32_t tb_, uint32_t zb) {
    const uint32_t w = tb_ + e.off;
    return reinterpret_cast<T*>(Pg + (e.col + min(w, w + zb)));
}

// Calls f(lo, w) (integral constants) with the range lo..w of row weights
// that d falls in: each weight up to 8 by itself, then pairs, then fours.  d
// is the same for every thread, so the branch is uniform; inside, the edges
// are straight-line code whose chains the compiler interleaves (a test per
// edge, as before, kept the chains of tanh and atanh one after the other).
template <int DMAX, class F>
__device__ __forceinline__ void sp_widths(int d, F&& f) {
#define SP_WIDTH(LO, W)                                                                   \
    if constexpr (DMAX >= W) {                                                            \
        if (d <= W) {                                                                     \
            f(std::integral_constant<int, LO>{}, std::integral_constant<int, W>{});       \
            return;                                                                       \
        }                                                                                 \
    }
    SP_WIDTH(2, 2) SP_WIDTH(3, 3) SP_WIDTH(4, 4) SP_WIDTH(5, 5) SP_WIDTH(6, 6) SP_WIDTH(7, 7) SP_WIDTH(8, 8)
    SP_WIDTH(9, 10) SP_WIDTH(11, 12) SP_WIDTH(13, 14) SP_WIDTH(15, 16) SP_WIDTH(17, 18) SP_WIDTH(19, 20)
    SP_WIDTH(21, 24) SP_WIDTH(25, 28) SP_WIDTH(29, 32)
#undef SP_WIDTH
}

// One row's update: d edges (LO <= d <= W) from table entry ed, messages
// R[j * rstride].  Edges beyond d are computed on the last edge's operands
// and dropped.
template <int LO, int W, bool PROD, class T>
__device__ __forceinline__ void sp_row(const SpEdge* ed, int d, char* Pg, T* R, int rstride, uint32_t tb_, uint32_t zb,
                                       T beta, T maxv) {
    T q[W], x[W], f[W];
    T* p[W];
    uint32_t rx = 0;
#pragma unroll
    for (int j = 0; j < W; ++j) {
        const int e = j < LO ? j : min(j, d - 1);
        p[j] = sp_at<T>(ed[e], Pg, tb_, zb);
        q[j] = sp_sub(*p[j], R[e * rstride]);
    }
#pragma unroll
    for (int j = 0; j < W; ++j) {
        T a = sp_sub(sp_abs(q[j]), beta);
        a = sp_max0(a);
        x[j] = PROD ? spm_tanh_half(a) : a;
        f[j] = x[j];
        if (j < LO || j < d) rx ^= sp_signw(q[j]);
    }
    run_tree<LO, W>(d, x, f, [](T a, T b) { return PROD ? sp_mul(a, b) : sp_min(a, b); },
                    [maxv](T v) { return sp_min(maxv, v); });
#pragma unroll
    for (int j = 0; j < W; ++j) {
        const T fj = PROD ? spm_atanh_twice(f[j]) : f[j];
        const T rn = sp_flip(fj, (rx ^ sp_signw(q[j])) & 0x80000000u);
        if (j < LO || j < d) {
            *p[j] = sp_add(q[j], rn);
            R[j * rstride] = rn;
        }
    }
}

// Bytes of the shared-memory copy of a code's circulants.
__host__ __device__ constexpr int sp_edge_bytes(int E) { return (E * (int)sizeof(SpEdge) + 15) & ~15; }

// Decode codewords [lo, hi) of job with the CTA: the whole decoder; edges is
// the code's circulants in shared memory, sm_f the CTA's dynamic shared memory
// (16-byte aligned) for posteriors, staging and (RSMEM) messages, r_cta its
// global message area otherwise.  T = float or double.
template <int DMAX, bool PROD, bool RSMEM, class T>
__device__ __forceinline__ void sp_decode_range(const SpTables& tb, const SpEdge* edges, const SpJobT<T>& job,
                                                long long lo, long long hi, T* sm_f, T* r_cta) {
    constexpr int V = 16 / (int)sizeof(T);
    __shared__ long long s_cur[32];
    __shared__ long long s_next[32];
    __shared__ int s_it[32];
    __shared__ uint32_t s_synd[2];        // bit g: a check of group g's codeword fails (per iteration parity)
    __shared__ uint32_t s_zero[2];        // bit g: clear group g's messages
    __shared__ int s_busy[2];
    __shared__ unsigned long long s_head;
    __shared__ unsigned long long s_cnt[OMS_MAX_BUCKETS][4];

    const int z = tb.z, n = tb.n, G = tb.G, stride = tb.stride;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5;
    const int nthr = blockDim.x;
    const int t = tid / G, g = tid - (tid / G) * G;
    const bool active = t < z;
    const int gbase = g * stride;
    const bool staged = !tb.nostage;
    T* Ps = sm_f;
    T* stage = sm_f + ((G * stride + V - 1) & ~(V - 1));            // [G][nstage], 16-byte aligned
    const int nstage = (n + V - 1) & ~(V - 1);
    T* Rbase = RSMEM ? stage + (staged ? G * nstage : 0) : r_cta;
    // check messages: in shared memory each thread's E values are contiguous
    // at an odd stride (E | 1: a warp's lanes fall in distinct banks), so edge
    // e is the thread's base plus e; the global scratch keeps edge-major
    // values (coalesced), edge e at Rt[e * nthr]
    const int rstride = RSMEM ? 1 : nthr;
    T* Rt = RSMEM ? Rbase + tid * (tb.E | 1) : Rbase + tid;
    const T beta = job.beta, maxv = job.maxv;

    for (int i = tid; i < OMS_MAX_BUCKETS * 4; i += nthr) (&s_cnt[0][0])[i] = 0;
    for (int i = tid; i < G * stride; i += nthr) Ps[i] = T(0);
    for (int e = 0; e < tb.E; ++e) Rt[e * rstride] = T(0);
    if (tid < 32) {
        const long long c0 = lo + tid, c1 = lo + G + tid;
        s_cur[tid] = tid < G && c0 < hi ? c0 : -1;
        s_next[tid] = tid < G && c1 < hi ? c1 : -1;
        s_it[tid] = 0;
    }
    if (tid < 2) { s_synd[tid] = 0; s_zero[tid] = 0; s_busy[tid] = 0; }
    if (tid == 0) s_head = (unsigned long long)(lo + 2 * G);
    __syncthreads();
    for (int k = warp; k < G; k += nwarps) {
        if (s_cur[k] >= 0) {
            const T* src = job.llr + s_cur[k] * (long long)n;
            for (int i = lane; i < n; i += 32) Ps[k * stride + i] = src[i];
        }
        if (staged && s_next[k] >= 0) sp_prefetch(stage + k * nstage, job.llr, s_next[k], n, lane);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    __syncthreads();

    char* const Pg = reinterpret_cast<char*>(Ps + gbase);
    const uint32_t tb_ = (uint32_t)t * (uint32_t)sizeof(T), zb = (uint32_t)z * (uint32_t)sizeof(T);

    for (int par = 0;; par ^= 1) {
        // ================= one layered iteration =================
        for (int l = 0; l < tb.L; ++l) {
            if (active) {
                const int d = tb.rw[l], eb = tb.ebase[l];
                sp_widths<DMAX>(d, [&](auto lo_, auto w_) {
                    sp_row<decltype(lo_)::value, decltype(w_)::value, PROD>(edges + eb, d, Pg, Rt + eb * rstride, rstride,
                                                                            tb_, zb, beta, maxv);
                });
            }
            __syncthreads();
        }
        if (tid == 0) { s_synd[par ^ 1] = 0; s_zero[par ^ 1] = 0; s_busy[par ^ 1] = 0; }

        // ================= syndrome (early exit once this codeword fails) =================
        if (active) {
            for (int l = 0; l < tb.L; ++l) {
                if (*reinterpret_cast<volatile uint32_t*>(&s_synd[par]) & (1u << g)) break;
                const int d = tb.rw[l], eb = tb.ebase[l];
                uint32_t xr = 0;
#pragma unroll 4
                for (int j = 0; j < d; ++j) xr ^= sp_signw(*sp_at<T>(edges[eb + j], Pg, tb_, zb));
                if (xr & 0x80000000u) {
                    atomicOr(&s_synd[par], 1u << g);
                    break;
                }
            }
        }
        __syncthreads();

        // ====== each warp: its codewords -- decide, write out, promote, claim, prefetch ======
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
        for (int k = warp; k < G; k += nwarps) {
            const long long cw = s_cur[k];
            if (cw < 0) continue;
            const int it = s_it[k] + 1;
            const bool done = !(s_synd[par] & (1u << k)) || it >= job.max_iter;
            if (!done) {
                if (lane == 0) { s_it[k] = it; s_busy[par] = 1; }
                continue;
            }
            const T* pk = Ps + k * stride;
            const uint32_t* ref = job.ref_bits ? job.ref_bits + (cw % job.ref_period) * tb.hard_words : nullptr;
            unsigned errw, errslots;
            warp_hard_decisions<true>([&](int i) { return pk[i] < T(0); }, tb.kbits, tb.hard_words, z, job.num_par,
                                job.hard_out ? job.hard_out + cw * tb.hard_words : nullptr, ref, lane, errw, errslots);
            if (job.post_out) {
                T* dst = job.post_out + cw * (long long)n;
                for (int i = lane; i < n; i += 32) dst[i] = pk[i];
            }
            if (lane == 0 && job.iters_out) job.iters_out[cw] = (uint8_t)it;
            if (job.counters && lane == 0) {
                int bk = (int)(cw / job.bucket_size);
                bk = bk < job.n_buckets ? bk : job.n_buckets - 1;
                atomicAdd(&s_cnt[bk][0], 1ull);
                atomicAdd(&s_cnt[bk][1], (unsigned long long)it);
                if (errw) {
                    atomicAdd(&s_cnt[bk][2], (unsigned long long)errw);
                    atomicAdd(&s_cnt[bk][3], (unsigned long long)__popc(errslots));
                }
            }
            __syncwarp();
            const long long nxt = s_next[k];
            if (nxt >= 0) {
                const T* st = staged ? stage + k * nstage : job.llr + nxt * (long long)n;
                for (int i = lane; i < n; i += 32) Ps[k * stride + i] = st[i];
                __syncwarp();
                unsigned long long c = 0;
                if (lane == 0) c = atomicAdd(&s_head, 1ull);
                c = __shfl_sync(0xffffffffu, c, 0);
                const long long fresh = (long long)c < hi ? (long long)c : -1;
                if (staged && fresh >= 0) sp_prefetch(stage + k * nstage, job.llr, fresh, n, lane);
                if (lane == 0) { s_next[k] = fresh; s_busy[par] = 1; }
            }
            if (lane == 0) {
                s_cur[k] = nxt;
                s_it[k] = 0;
                atomicOr(&s_zero[par], 1u << k);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        __syncthreads();
        if (active && (s_zero[par] & (1u << g)))
            for (int e = 0; e < tb.E; ++e) Rt[e * rstride] = T(0);
        if (!s_busy[par]) break;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (job.counters) {
        __syncthreads();
        for (int i = tid; i < job.n_buckets * 4; i += nthr) {
            const unsigned long long v = (&s_cnt[0][0])[i];
            if (v) atomicAdd(job.counters + i, v);
        }
    }
}

// Register budget of a float kernel instance.  Sum-product on rows of weight
// <= 8 with its check messages in global scratch is held to 80 registers
// (no spills): 128-thread CTAs then fit 6 per SM instead of 5 and 384-thread
// CTAs 2 instead of 1, which pays in this latency-bound case (tanh/atanh
// chains).  Every other instance keeps the 128 that a 512-thread CTA allows.
__host__ __device__ constexpr int sp_max_regs(int dmax, bool prod, bool rsmem) {
    return dmax == 8 && prod && !rsmem ? 80 : 128;
}

// A code's circulants from the kernel parameters into the front of the CTA's
// dynamic shared memory: one broadcast load per edge there, against two
// indexed constant loads.
__device__ __forceinline__ const SpEdge* sp_load_edges(const SpTables& tb, void* sm) {
    SpEdge* e = reinterpret_cast<SpEdge*>(sm);
    for (int i = threadIdx.x; i < tb.E; i += blockDim.x) e[i] = tb.edge[i];
    return e;   // visible after sp_decode_range's first barrier
}

template <int DMAX, bool PROD, bool RSMEM, int MAXT>
__global__ void __maxnreg__(sp_max_regs(DMAX, PROD, RSMEM)) sp_f32_kernel(const __grid_constant__ SpTables tb, const __grid_constant__ SpJob job) {
    extern __shared__ __align__(16) float sm_f[];
    const long long lo = job.ncw * blockIdx.x / gridDim.x, hi = job.ncw * (blockIdx.x + 1) / gridDim.x;
    const SpEdge* edges = sp_load_edges(tb, sm_f);
    __shared__ int s_area;
    const int area = RSMEM ? 0 : take_area(job.areas, s_area);
    if (area < 0) return;
    sp_decode_range<DMAX, PROD, RSMEM>(tb, edges, job, lo, hi, sm_f + sp_edge_bytes(tb.E) / 4,
                                       RSMEM ? nullptr : job.r_scratch + (long long)area * tb.E * blockDim.x);
    if (!RSMEM) give_area(job.areas, s_area);
}

template <int DMAX, bool PROD, bool RSMEM, int MAXT>
__global__ void __launch_bounds__(MAXT) sp_f64_kernel(const __grid_constant__ SpTables tb,
                                                      const __grid_constant__ SpJobT<double> job) {
    extern __shared__ __align__(16) double sm_d[];
    const long long lo = job.ncw * blockIdx.x / gridDim.x, hi = job.ncw * (blockIdx.x + 1) / gridDim.x;
    const SpEdge* edges = sp_load_edges(tb, sm_d);
    __shared__ int s_area;
    const int area = RSMEM ? 0 : take_area(job.areas, s_area);
    if (area < 0) return;
    sp_decode_range<DMAX, PROD, RSMEM>(tb, edges, job, lo, hi, sm_d + sp_edge_bytes(tb.E) / 8,
                                       RSMEM ? nullptr : job.r_scratch + (long long)area * tb.E * blockDim.x);
    if (!RSMEM) give_area(job.areas, s_area);
}

}  // namespace ldpc
