// Host side of the learned-offset decoder: forward with checkpoints,
// adjoint, and evaluation with early exit.
#include <algorithm>
#include <cstring>

#include "internal.h"
#include "train.cuh"
#include "train_step.cuh"

using ldpc::fail;

namespace {

typedef void (*train_fn)(const ldpc::SpTables, const ldpc::TrainJob);

struct TrainKernels {
    int dmax;
    train_fn fwd, bwd;
};
const TrainKernels kTrain[] = {{8, ldpc::oms_train_fwd<8>, ldpc::oms_train_bwd<8>},
                               {16, ldpc::oms_train_fwd<16>, ldpc::oms_train_bwd<16>},
                               {32, ldpc::oms_train_fwd<32>, ldpc::oms_train_bwd<32>}};

constexpr int kTrainMaxSmem = 220 * 1024;

struct Geometry {
    train_fn k;
    int threads, smem, grid;
};

int geometry(ldpc_ctx* x, size_t n, bool backward, Geometry* g) {
    if (!x) return fail(LDPC_ERR_INVALID_ARG, "ctx is NULL");
    if (x->cfg.variant != LDPC_F32_OMS)
        return fail(LDPC_ERR_INVALID_ARG, "the learned-offset decoder needs a float offset min-sum context");
    const ldpc::SpTables& t = x->spt;
    const int d = x->code.max_row_weight;
    const TrainKernels* tk = nullptr;
    for (const TrainKernels& k : kTrain)
        if (d <= k.dmax) {
            tk = &k;
            break;
        }
    if (!tk) return fail(LDPC_ERR_UNSUPPORTED, "learned decoder: row weight %d > 32", d);
    const size_t n4 = (size_t)((t.n + 3) & ~3), ez4 = (size_t)((t.E * t.z + 3) & ~3);
    const size_t smem = backward ? 2 * (n4 + ez4) * 4 : (n4 + ez4) * 4;
    if (smem > (size_t)kTrainMaxSmem)
        return fail(LDPC_ERR_UNSUPPORTED, "learned decoder: %zu B of shared memory per codeword (N=%d, %d edges)", smem, t.n,
                    t.E * t.z);
    g->k = backward ? tk->bwd : tk->fwd;
    g->threads = ((t.z + 31) / 32) * 32;
    g->smem = (int)smem;
    CUDA_TRY(ldpc::allow_dynamic_smem((const void*)g->k, kTrainMaxSmem));
    int per_sm = 0;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)g->k, g->threads, g->smem));
    if (per_sm < 1) return fail(LDPC_ERR_UNSUPPORTED, "learned decoder: launch does not fit an SM");
    g->grid = (int)std::max<long long>(1, std::min<long long>((long long)n, (long long)per_sm * x->sms));
    return LDPC_OK;
}

// Loss (and gradient) kernel: codewords per CTA as the float decoders choose
// them, fewer while the CTA's shared memory is above what lets five share an SM.
typedef void (*step_fn)(const ldpc::SpTables, const ldpc::TrainStepJob);
struct StepKernels {
    int dmax, nt;
    step_fn grad, loss;
};
#define TSK(D_, N_) {D_, N_, ldpc::oms_train_step<D_, N_, true>, ldpc::oms_train_step<D_, N_, false>}
const StepKernels kStep[] = {TSK(8, 128), TSK(16, 128), TSK(32, 128), TSK(8, 512), TSK(16, 512), TSK(32, 512)};
#undef TSK

struct StepGeometry {
    step_fn k;
    int threads, smem, grid, nt;
    ldpc::SpTables t;
};

int step_geometry(ldpc_ctx* x, size_t n, int iters, bool grad, StepGeometry* g) {
    Geometry unused;
    // the codes that the separate forward and adjoint kernels take
    if (int rc = geometry(x, n, grad, &unused)) return rc;
    const ldpc_code& c = x->code;
    int G = std::max(1, std::min(32, 128 / c.z));
    auto smem = [&](int k) {
        ldpc::fill_sp_tables(c, k, (int)sizeof(float), &g->t);
        return ldpc::train_step_smem(k, g->t.stride, g->t.E, g->t.mcol, ((k * c.z + 31) / 32) * 32, iters * g->t.L);
    };
    while (G > 1 && smem(G) > 45 * 1024) --G;
    g->smem = smem(G);
    g->threads = ((G * c.z + 31) / 32) * 32;
    g->nt = g->threads <= 128 ? 128 : 512;
    g->k = nullptr;
    for (const StepKernels& k : kStep)
        if (!g->k && k.nt == g->nt && c.max_row_weight <= k.dmax) g->k = grad ? k.grad : k.loss;
    if (g->smem > kTrainMaxSmem)
        return fail(LDPC_ERR_UNSUPPORTED, "learned decoder: %d B of shared memory per codeword", g->smem);
    CUDA_TRY(ldpc::allow_dynamic_smem((const void*)g->k, kTrainMaxSmem));
    int per_sm = 0;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)g->k, g->threads, g->smem));
    if (per_sm < 1) return fail(LDPC_ERR_UNSUPPORTED, "learned decoder: launch does not fit an SM");
    const long long want = ((long long)n + G - 1) / G;
    g->grid = (int)std::max<long long>(1, std::min<long long>(want, (long long)per_sm * x->sms));
    return LDPC_OK;
}

int check_iters(int iters) {
    if (iters < 1 || iters > ldpc::TRAIN_MAX_ITERS)
        return fail(LDPC_ERR_INVALID_ARG, "iterations %d outside 1..%d", iters, ldpc::TRAIN_MAX_ITERS);
    return LDPC_OK;
}

}  // namespace

extern "C" {

int ldpc_learned_grid(ldpc_ctx* x, size_t n, int* bwd_grid) {
    Geometry g;
    if (int rc = geometry(x, n, true, &g)) return rc;
    if (bwd_grid) *bwd_grid = g.grid;
    return LDPC_OK;
}

int ldpc_learned_forward(ldpc_ctx* x, const float* llr, size_t n, int iters, const float* beta, float* ckpt_p,
                         float* ckpt_r, void* stream) {
    if (int rc = check_iters(iters)) return rc;
    if (n && (!llr || !beta || !ckpt_p || !ckpt_r)) return fail(LDPC_ERR_INVALID_ARG, "NULL buffer");
    Geometry g;
    if (int rc = geometry(x, n, false, &g)) return rc;
    if (n == 0) return LDPC_OK;
    CUDA_TRY(cudaSetDevice(x->device));
    ldpc::TrainJob j;
    memset(&j, 0, sizeof(j));
    j.llr = llr;
    j.ncw = (long long)n;
    j.iters = iters;
    j.beta = beta;
    j.maxv = x->maxf;
    j.ckpt_p = ckpt_p;
    j.ckpt_r = ckpt_r;
    g.k<<<g.grid, g.threads, g.smem, (cudaStream_t)stream>>>(x->spt, j);
    CUDA_TRY(cudaGetLastError());
    return LDPC_OK;
}

int ldpc_learned_backward(ldpc_ctx* x, size_t n, int iters, const float* beta, const float* ckpt_p, const float* ckpt_r,
                          const uint8_t* cw_bits, const float* loss_w, float inv_norm, float* gbeta_part,
                          float* grad_llr, void* stream) {
    if (int rc = check_iters(iters)) return rc;
    if (n && (!beta || !ckpt_p || !ckpt_r || !cw_bits || !loss_w || !gbeta_part))
        return fail(LDPC_ERR_INVALID_ARG, "NULL buffer");
    Geometry g;
    if (int rc = geometry(x, n, true, &g)) return rc;
    if (n == 0) return LDPC_OK;
    CUDA_TRY(cudaSetDevice(x->device));
    ldpc::TrainJob j;
    memset(&j, 0, sizeof(j));
    j.ncw = (long long)n;
    j.iters = iters;
    j.beta = beta;
    j.maxv = x->maxf;
    j.ckpt_p = const_cast<float*>(ckpt_p);
    j.ckpt_r = const_cast<float*>(ckpt_r);
    j.cw_bits = cw_bits;
    j.loss_w = loss_w;
    j.inv_norm = inv_norm;
    j.gbeta_part = gbeta_part;
    j.grad_llr = grad_llr;
    g.k<<<g.grid, g.threads, g.smem, (cudaStream_t)stream>>>(x->spt, j);
    CUDA_TRY(cudaGetLastError());
    return LDPC_OK;
}

int ldpc_learned_loss_size(ldpc_ctx* x, size_t n, int iters, int want_grad, int* loss_rows, int* grad_rows,
                           size_t* scratch_floats) {
    if (int rc = check_iters(iters)) return rc;
    StepGeometry g;
    if (int rc = step_geometry(x, n, iters, want_grad != 0, &g)) return rc;
    if (loss_rows) *loss_rows = g.grid;
    if (grad_rows) *grad_rows = g.grid * (g.threads / 32);
    if (scratch_floats) *scratch_floats = (size_t)g.grid * iters * (g.t.E + g.t.mcol) * g.nt;
    return LDPC_OK;
}

int ldpc_learned_loss(ldpc_ctx* x, const float* llr, const uint8_t* cw_bits, size_t n, int iters, const float* beta,
                      const float* loss_w, float inv_norm, float* scratch, float* gbeta_part, double* loss_part,
                      void* stream) {
    if (int rc = check_iters(iters)) return rc;
    if (!loss_part || (n && (!llr || !cw_bits || !beta || !loss_w)) || (!scratch != !gbeta_part))
        return fail(LDPC_ERR_INVALID_ARG, "NULL buffer");
    StepGeometry g;
    if (int rc = step_geometry(x, n, iters, scratch != nullptr, &g)) return rc;
    CUDA_TRY(cudaSetDevice(x->device));
    ldpc::TrainStepJob j;
    memset(&j, 0, sizeof(j));
    j.llr = llr;
    j.cw_bits = cw_bits;
    j.ncw = (long long)n;
    j.iters = iters;
    j.beta = beta;
    j.loss_w = loss_w;
    j.maxv = x->maxf;
    j.inv_norm = inv_norm;
    j.scratch = scratch;
    j.gbeta_part = gbeta_part;
    j.loss_part = loss_part;
    g.k<<<g.grid, g.threads, g.smem, (cudaStream_t)stream>>>(g.t, j);
    CUDA_TRY(cudaGetLastError());
    return LDPC_OK;
}

int ldpc_learned_decode(ldpc_ctx* x, const float* llr, size_t n, int iters, const float* beta, float* post_out,
                        uint32_t* hard_out, uint8_t* iters_out, void* stream) {
    if (int rc = check_iters(iters)) return rc;
    if (n && (!llr || !beta)) return fail(LDPC_ERR_INVALID_ARG, "NULL buffer");
    Geometry g;
    if (int rc = geometry(x, n, false, &g)) return rc;
    if (n == 0) return LDPC_OK;
    CUDA_TRY(cudaSetDevice(x->device));
    ldpc::TrainJob j;
    memset(&j, 0, sizeof(j));
    j.llr = llr;
    j.ncw = (long long)n;
    j.iters = iters;
    j.beta = beta;
    j.maxv = x->maxf;
    j.early_exit = 1;
    j.post_out = post_out;
    j.hard_out = hard_out;
    j.iters_out = iters_out;
    g.k<<<g.grid, g.threads, g.smem, (cudaStream_t)stream>>>(x->spt, j);
    CUDA_TRY(cudaGetLastError());
    return LDPC_OK;
}

}  // extern "C"
