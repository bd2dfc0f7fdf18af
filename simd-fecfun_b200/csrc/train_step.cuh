// Loss and offset gradient of the learned-offset decoder in one kernel: the
// forward unrolling, the loss and the adjoint of train.cuh, per codeword in
// one CTA, so that what the adjoint needs never leaves the CTA's own scratch.
//
//   forward   per iteration and layer as train.cuh; every edge's Q goes to the
//             scratch, and after each iteration the loss of the posteriors and
//             its adjoint (the adjoint to the scratch)
//   adjoint   iterations and layers in reverse, from the stored Q: nothing is
//             recomputed.  Of a row's edges only the two that hold the smallest
//             and the second smallest magnitude pass a gradient through the
//             minimum (ga in train.cuh is 0 elsewhere), so gP changes there
//             alone and the offset's gradient is minus those two.
//
// What bounds it: instruction issue and the scratch's traffic together.
// 802.16e 1/2 Z = 96, 10 iterations: 292 KB of Q and 92 KB of loss adjoint per
// codeword, written once and read once in the opposite order (so that L2
// serves the younger part), against 384 KB of posteriors and messages written
// to checkpoints, read back, and the layers recomputed from them.  65536
// codewords: 105 ms (13 forward, 84 adjoint, 8 for the loss in torch) -> 19.3 ms;
// issue 58 %, DRAM 29 %, 15 warps per SM (shared memory).  Q loaded one row
// ahead: 25.4 -> 22.6 ms; sent bits in shared memory: -> 18.8 ms; the loss in full
// float precision (expf, the product of 1 + e^-|x| kept less 1, a quotient with
// residual step): -> 19.3 ms.
//
// Layout: G codewords per CTA, thread (g, t) = check row t of every layer of
// codeword g, as the decoders.  The messages R (forward) and their adjoint
// (backward) sit per thread at an odd stride.  Scratch of a CTA, coalesced:
// Q at [(it * E + e) * NT + tid], loss adjoint at [(it * mcol + c) * NT + tid]
// behind it; thread (g, t) owns element t of every column in these passes.
// NT = 128 for CTAs of up to 128 threads, so that a row's addresses are a base
// plus immediates; 512 otherwise.
#pragma once
#include <stdint.h>

#include "sp_f32.cuh"
#include "tables.h"
#include "train.cuh"

namespace ldpc {

struct TrainStepJob {
    const float* llr;                // [ncw][n]
    const uint8_t* cw_bits;          // [ncw][n] sent code bits
    long long ncw;
    int iters;
    const float* beta;               // [iters][L]
    const float* loss_w;             // [iters]
    float maxv;                      // row clamp
    float inv_norm;
    float* scratch;                  // [gridDim][iters * (E + mcol) * NT], or null: loss only
    float* gbeta_part;               // [gridDim * warps][iters * L] (with scratch)
    double* loss_part;               // [gridDim]
};

__host__ __device__ constexpr int train_step_smem(int G, int stride, int E, int mcol, int threads, int n_beta) {
    return sp_edge_bytes(E) + 4 * (((G * stride + 3) & ~3) + ((E | 1) + (mcol + 31) / 32) * threads + n_beta);
}

// One row forward (weights LO..W, as sp_widths).  Q to qs[j * NT] if KEEP.
template <int LO, int W, int NT, bool KEEP>
__device__ __forceinline__ void ts_row_fwd(const SpEdge* ed, int d, char* Pg, float* R, uint32_t tb_, uint32_t zb,
                                           float beta, float maxv, float* qs) {
    float q[W], a[W];
    float* p[W];
    float mn1 = __int_as_float(0x7f800000), mn2 = mn1;
    uint32_t rx = 0;
#pragma unroll
    for (int j = 0; j < W; ++j) {
        const int e = j < LO ? j : min(j, d - 1);
        p[j] = sp_at<float>(ed[e], Pg, tb_, zb);
        q[j] = __fsub_rn(*p[j], R[e]);
    }
#pragma unroll
    for (int j = 0; j < W; ++j) {
        const bool has = j < LO || j < d;
        a[j] = fmaxf(__fsub_rn(fabsf(q[j]), beta), 0.0f);
        if (KEEP && has) qs[j * NT] = q[j];
        if (!has) a[j] = __int_as_float(0x7f800000);
        else rx ^= __float_as_uint(q[j]);
        mn2 = fminf(mn2, fmaxf(mn1, a[j]));
        mn1 = fminf(mn1, a[j]);
    }
    const float f1 = fminf(maxv, mn1), f2 = fminf(maxv, mn2);
#pragma unroll
    for (int j = 0; j < W; ++j) {
        const float f = a[j] == mn1 ? f2 : f1;   // several at mn1: mn2 = mn1
        const float rn = sp_flip(f, (rx ^ __float_as_uint(q[j])) & 0x80000000u);
        if (j < LO || j < d) {
            *p[j] = __fadd_rn(q[j], rn);
            R[j] = rn;
        }
    }
}

// One row of the adjoint: q from the scratch (loaded by the caller before the
// barrier).  R holds, per edge, the adjoint of Q of the following iteration
// (the adjoint of R' is gP - that).  Returns the row's gradient of its offset.
template <int LO, int W>
__device__ __forceinline__ float ts_row_bwd(const SpEdge* ed, int d, char* Gg, float* R, uint32_t tb_, uint32_t zb,
                                            float beta, float maxv, const float (&q)[W]) {
    float m[W], gp[W];
    float* p[W];
    float mn1 = __int_as_float(0x7f800000), mn2 = mn1;
    uint32_t rx = 0;
#pragma unroll
    for (int j = 0; j < W; ++j) {
        const bool has = j < LO || j < d;
        p[j] = sp_at<float>(ed[j < LO ? j : min(j, d - 1)], Gg, tb_, zb);
        gp[j] = *p[j];
        m[j] = has ? fmaxf(__fsub_rn(fabsf(q[j]), beta), 0.0f) : __int_as_float(0x7f800000);
        if (has) rx ^= __float_as_uint(q[j]);
        mn2 = fminf(mn2, fmaxf(mn1, m[j]));
        mn1 = fminf(mn1, m[j]);
    }
    // gradients pass the minimum unless the clamp holds the row's value; those at
    // or below the offset (m = 0) end there
    const bool to1 = mn1 < maxv && mn1 > 0.0f, to2 = mn2 < maxv && mn2 > 0.0f;
    if (mn1 == mn2 && to1) {
        // two edges at the minimum: the first is the minimum, the next one the second
        bool first = true;
#pragma unroll
        for (int j = 0; j < W; ++j)
            if (first && m[j] == mn1) {
                m[j] = -1.0f;
                first = false;
            }
        mn1 = -1.0f;
    }
    float gm1 = 0.0f, gm2 = 0.0f;
#pragma unroll
    for (int j = 0; j < W; ++j) {
        if (j < LO || j < d) {
            const float gf = sp_flip(__fsub_rn(gp[j], R[j]), (rx ^ __float_as_uint(q[j])) & 0x80000000u);
            if (m[j] == mn1) gm2 += gf;
            else gm1 += gf;
        }
    }
    // the value of every edge but the smallest is mn1, the smallest's is mn2
    gm1 = to1 ? gm1 : 0.0f;
    gm2 = to2 ? gm2 : 0.0f;
    const float gb = -(gm1 + gm2);
#pragma unroll
    for (int j = 0; j < W; ++j) {
        if (j < LO || j < d) {
            const bool is1 = m[j] == mn1, is2 = m[j] == mn2;
            const float ga = is1 ? gm1 : is2 ? gm2 : 0.0f;
            if (is2 && !is1) gm2 = 0.0f;         // the first of several second smallest
            const float gq = gp[j] + sp_flip(ga, __float_as_uint(q[j]) & 0x80000000u);
            if (is1 || is2) *p[j] = gq;
            R[j] = gq;
        }
    }
    return gb;
}

template <int DMAX, int NT, bool GRAD>
__global__ void __launch_bounds__(NT) oms_train_step(const __grid_constant__ SpTables tb, const __grid_constant__ TrainStepJob job) {
    extern __shared__ __align__(16) float ts_sm[];
    __shared__ double s_loss[NT / 32];
    const SpEdge* edges = sp_load_edges(tb, ts_sm);
    const int z = tb.z, n = tb.n, G = tb.G, L = tb.L, E = tb.E, mcol = tb.mcol, iters = job.iters;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int g = tid / z, t = tid - (tid / z) * z;
    float* const Ps = ts_sm + sp_edge_bytes(E) / 4;
    float* const Pg = Ps + g * tb.stride;
    float* const R = Ps + ((G * tb.stride + 3) & ~3) + tid * (E | 1);
    char* const Pb = reinterpret_cast<char*>(Pg);
    float* const betas = Ps + ((G * tb.stride + 3) & ~3) + (int)blockDim.x * (E | 1);
    for (int i = tid; i < iters * L; i += blockDim.x) betas[i] = job.beta[i];
    // sent bits of the thread's elements, 32 columns per word, word w at sent[w * blockDim.x]
    uint32_t* const sent = reinterpret_cast<uint32_t*>(betas + iters * L) + tid;
    const uint32_t tb_ = 4u * (uint32_t)t, zb = 4u * (uint32_t)z;
    float* const Qs = GRAD ? job.scratch + (long long)blockIdx.x * iters * (E + mcol) * NT + tid : nullptr;
    float* const Gs = GRAD ? Qs + (long long)iters * E * NT : nullptr;
    float* const part = GRAD ? job.gbeta_part + (long long)(blockIdx.x * nwarps + warp) * iters * L : nullptr;
    if (GRAD) {
        for (int i = lane; i < iters * L; i += 32) part[i] = 0.0f;
        __syncwarp();
    }
    double loss = 0.0;

    for (long long c0 = (long long)blockIdx.x * G; c0 < job.ncw; c0 += (long long)gridDim.x * G) {
        const long long cw = c0 + g;
        const bool active = g < G && cw < job.ncw;
        __syncthreads();   // the previous codewords are finished with the shared memory
        const uint8_t* bits = job.cw_bits + cw * (long long)n + t;
        if (active) {
            const float* src = job.llr + cw * (long long)n + t;
#pragma unroll 8
            for (int c = 0; c < mcol; ++c) Pg[c * z + t] = src[c * z];
            for (int e = 0; e < E; ++e) R[e] = 0.0f;
            for (int b = 0; b < mcol; b += 32) {
                uint32_t m = 0;
#pragma unroll 8
                for (int c = b; c < min(b + 32, mcol); ++c) m |= (bits[c * z] ? 1u : 0u) << (c - b);
                sent[(b >> 5) * blockDim.x] = m;
            }
        }
        __syncthreads();
        for (int it = 0; it < iters; ++it) {
            for (int l = 0; l < L; ++l) {
                if (active) {
                    const int d = tb.rw[l], eb = tb.ebase[l];
                    const float beta = betas[it * L + l];
                    float* qs = GRAD ? Qs + (long long)(it * E + eb) * NT : nullptr;
                    sp_widths<DMAX>(d, [&](auto lo_, auto w_) {
                        ts_row_fwd<decltype(lo_)::value, decltype(w_)::value, NT, GRAD>(edges + eb, d, Pb, R + eb, tb_, zb,
                                                                                        beta, job.maxv, qs);
                    });
                }
                __syncthreads();
            }
            // loss softplus(x), x = -s P: max(x, 0) + ln(1 + e^-|x|), the logarithms of up to 32
            // elements as one of their product.  The product is kept less 1, a sum of positive
            // terms, so that small e^-|x| count in full (a converged batch has no others; as a
            // product of rounded 1 + e^-|x| its loss was 1 % off at |P| = 12, 0 beyond 16.6).  The
            // adjoint is -s times the logistic of x.
            if (active) {
                const float w = __ldg(job.loss_w + it), wk = w * job.inv_norm;
                float* gs = GRAD ? Gs + (long long)it * mcol * NT : nullptr;
                float sum = 0.0f;
                for (int b = 0; b < mcol; b += 32) {
                    const int bn = min(32, mcol - b);
                    float prod1 = 0.0f;   // product - 1
                    uint32_t m = ~sent[(b >> 5) * blockDim.x];
#pragma unroll 8
                    for (int c = 0; c < bn; ++c, m >>= 1) {
                        const uint32_t sg = m << 31;
                        const float x = sp_flip(Pg[(b + c) * z + t], sg);
                        const float ex = expf(-fabsf(x));
                        sum += fmaxf(x, 0.0f);
                        prod1 = __fmaf_rn(prod1, ex, prod1) + ex;
                        if (GRAD) gs[(b + c) * NT] = sp_flip(wk * spm_div(x < 0.0f ? ex : 1.0f, 1.0f + ex), sg);
                    }
                    sum += log1pf(prod1);
                }
                loss += (double)w * (double)sum;
            }
            __syncthreads();
        }
        if (!GRAD) continue;

        if (active) {
            for (int c = 0; c < mcol; ++c) Pg[c * z + t] = 0.0f;
            for (int e = 0; e < E; ++e) R[e] = 0.0f;
        }
        // Q one layer ahead, as wide as the widest row, where registers allow: a
        // row's loads are under way while the row before it is computed
        constexpr bool AHEAD = DMAX <= 16;
        float qn[AHEAD ? DMAX : 1];
        if (AHEAD) {
            const float* qs = Qs + (long long)((iters - 1) * E + tb.ebase[L - 1]) * NT;
#pragma unroll
            for (int j = 0; j < (AHEAD ? DMAX : 1); ++j) qn[j] = active && j < tb.rw[L - 1] ? qs[j * NT] : 0.0f;
        }
        for (int it = iters - 1; it >= 0; --it) {
            if (active) {
                const float* gs = Gs + (long long)it * mcol * NT;
#pragma unroll 12
                for (int c = 0; c < mcol; ++c) Pg[c * z + t] += gs[c * NT];
            }
            for (int l = L - 1; l >= 0; --l) {
                const int d = tb.rw[l], eb = tb.ebase[l];
                const float beta = betas[it * L + l];
                const float* qs = Qs + (long long)(it * E + eb) * NT;
                float gb = 0.0f;
                float qc[AHEAD ? DMAX : 1];
                if (AHEAD) {
                    const int ln = l > 0 ? l - 1 : L - 1, in = l > 0 ? it : it - 1;
                    const float* nx = Qs + (long long)(in * E + tb.ebase[ln]) * NT;
                    const int dn = in >= 0 && active ? tb.rw[ln] : 0;
#pragma unroll
                    for (int j = 0; j < (AHEAD ? DMAX : 1); ++j) {
                        qc[j] = qn[j];
                        if (j < dn) qn[j] = nx[j * NT];
                    }
                }
                sp_widths<DMAX>(d, [&](auto lo_, auto w_) {
                    constexpr int LO = decltype(lo_)::value, W = decltype(w_)::value;
                    float q[W];
#pragma unroll
                    for (int j = 0; j < W; ++j)
                        q[j] = AHEAD ? qc[AHEAD ? j : 0] : active ? qs[(j < LO ? j : min(j, d - 1)) * NT] : 0.0f;
                    __syncthreads();   // the layer above (or the loss adjoint) is in gP
                    if (active) gb = ts_row_bwd<LO, W>(edges + eb, d, Pb, R + eb, tb_, zb, beta, job.maxv, q);
                });
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) gb += __shfl_xor_sync(0xffffffffu, gb, o);
                if (lane == 0) atomicAdd(part + it * L + l, gb);   // this warp alone adds here, in order
            }
            __syncthreads();
        }
    }
    // loss of the CTA, in a fixed order
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
    if (lane == 0) s_loss[warp] = loss;
    __syncthreads();
    if (tid == 0) {
        double s = 0.0;
        for (int w = 0; w < nwarps; ++w) s += s_loss[w];
        job.loss_part[blockIdx.x] = s * (double)job.inv_norm;
    }
}

}  // namespace ldpc
