// One encoder layer for training (network/sp_layer.py:52-104 of the reference, drop rates 0): the attention block's forward and the
// whole layer's backward less the three products named below, the launches issued from native code.
//   Q, K, V = [pos] LayerNorm(x W + b),  a = attention merged over heads,  x1 = x + a Wfc + bfc,  h = relu(x1 W1 + b1),  y = x1 + h W2 + b2.
// As single autograd ops a layer took 14 launches forward and 45 backward, each with its own Python, allocations and weight images,
// and a library product plus a reduction per dense layer for the weight and bias gradients.
// The caller makes the dense layers' forward products and dh = (dy W2^T) [h > 0], dx1 = dy + dh W1^T, da = dx1 Wfc^T in plain fp32: which
// hidden values pass the ReLU is decided by their last bits, and a chain of 24 products in 3xTF32, whose accumulation truncates,
// moved a training step's gradients further from fp64 (5.0e-6 against 3.1e-6).  The projections stay on the warp-MMA kernel: the
// tcgen05 one is as close to fp64 (9.1e-7 both before the LayerNorm, 5.0e-7 after it), but its other roundings put other single
// hidden values on the other side of the ReLU, each worth 1e-5 to 2e-4 of a step's gradients.
// Here: weight images (they change every step; one launch), projections and attention; then attention and LayerNorm backward to
// dqkv = [dq dk dv], dx = dx1 + dq Wq^T + dk Wk^T + dv Wv^T, one product x^T dqkv for the three projections' weights and one per dense
// layer (from 128 rows on, below which the caller's fp32 products are closer to fp64), with the bias gradients as its column sums.  LayerNorm's input is recomputed from x.
// 141 x 141 nodes, batch 4, whole training step: 14.6 -> 10.2 ms.
#include "tc_common.cuh"

namespace spgt {

int tc_weight_prepare_jobs(const TcPrepJobs& jobs, int n, cudaStream_t st);                          // tc_gemm.cu
int tn_gemm(const float* A, int lda, const float* B, int ldb, float* C, int ldc, int64_t panel, float* colsum, bool sum_a, int M, int N, int rows,
            void* workspace, size_t workspace_bytes, cudaStream_t st);                               // tc_tn.cu
int galerkin_attn_bwd(const float* Q, const float* K, const float* V, const float* d_out, float* dQ, float* dK, float* dV, int B, int H, int dpk,
                      int S, bool merged, void* workspace, size_t workspace_bytes, cudaStream_t st); // attention_bwd.cu
int projpos_qkv_mma(const float* x, const float* wq, const float* bq, const float* wk, const float* bk, const float* wv, const float* bv,
                    const float* lnwk, const float* lnbk, const float* lnwv, const float* lnbv, float eps, const float* pos, float* q, float* k, float* v,
                    int B, int S, int d_pos, cudaStream_t st);                                       // gemm.cu
size_t projpos_bwd_qkv_workspace_bytes(int B, int S);                                                // projection_bwd.cu
int projpos_bwd_qkv(const float* grad_q, const float* grad_k, const float* grad_v, const float* h, const float* lnwk, const float* lnwv, float eps,
                    float* dh, float* const* db, float* const* dlnw, float* const* dlnb, int B, int S, int d_pos, float* workspace, cudaStream_t st);

// Weight images (floats): per 128-wide column tile and 32-k block 2 * 128 * 32.
constexpr int ET_D = 128, ET_A = 136, ET_F = 256, ET_DP = 2, ET_W = 4 * 2 * 128 * 32;
constexpr int ET_KV = 0, ET_QKV_T = 2 * ET_W, ET_BKV = 5 * ET_W, ET_IMG = ET_BKV + 2 * ET_D;

// Kept for the backward: weight images, q, k, v.  Offsets in floats, multiples of four.
struct TrainSaved {
    size_t q, k, v, total;
    TrainSaved(size_t rows) { q = ET_IMG; k = q + rows * ET_A; v = k + rows * ET_A; total = v + rows * ET_A; }
};
// Scratch of the backward: K and V before their LayerNorm, gradients of q, k, v, and of the three projections side by side.
struct TrainScratch {
    size_t hkv, dq, dk, dv, dqkv, ws, ws_bytes, total;
    TrainScratch(int B, int S) {
        const size_t rows = (size_t)B * S;
        hkv = 0; dq = rows * ET_F; dk = dq + rows * ET_A; dv = dk + rows * ET_A; dqkv = dv + rows * ET_A; ws = dqkv + rows * 3 * ET_D;
        ws_bytes = spgt_galerkin_attn_bwd_workspace_bytes(B, 4, 34, S);
        const int n = (int)rows;
        for (const size_t need : {projpos_bwd_qkv_workspace_bytes(B, S), spgt_tn_gemm_workspace_bytes(ET_D, ET_F, n), spgt_tn_gemm_workspace_bytes(ET_F, ET_D, n),
                                  spgt_tn_gemm_workspace_bytes(ET_D, ET_A, n), spgt_tn_gemm_workspace_bytes(ET_D, 3 * ET_D, n)})
            if (need > ws_bytes) ws_bytes = need;
        total = ws + (ws_bytes + 3) / 4;
    }
};
static bool train_sizes_ok(int B, int S) { return B > 0 && S > 0 && (int64_t)B * S <= 0x7fffffffLL / 4; }

static int train_images(const spgt_encoder_params* p, float* img, cudaStream_t st) {
    TcPrepJobs jobs;
    int n = 0;
    auto add = [&](int kind, const float* w, float* dst) { jobs.job[n++] = {w, dst, kind, ET_D, ET_D, ET_D, ET_D, 128}; };
    add(0, p->wk, img + ET_KV);                            // [128 in][128 out]
    add(0, p->wv, img + ET_KV + ET_W);
    add(1, p->wq, img + ET_QKV_T);
    add(1, p->wk, img + ET_QKV_T + ET_W);
    add(1, p->wv, img + ET_QKV_T + 2 * ET_W);
    add(2, p->bk, img + ET_BKV);
    add(2, p->bv, img + ET_BKV + ET_D);
    return tc_weight_prepare_jobs(jobs, n, st);
}

static bool train_params_ok(const spgt_encoder_params* p) {
    for (const float* v : {p->wq, p->wk, p->wv, p->bq, p->bk, p->bv, p->lnwk, p->lnbk, p->lnwv, p->lnbv})
        if (!v) return false;
    return true;
}

}  // namespace spgt

using namespace spgt;

extern "C" size_t spgt_encoder_train_saved_bytes(int B, int S) { return train_sizes_ok(B, S) ? TrainSaved((size_t)B * S).total * sizeof(float) : 0; }
extern "C" size_t spgt_encoder_train_workspace_bytes(int B, int S) { return train_sizes_ok(B, S) ? TrainScratch(B, S).total * sizeof(float) : 0; }

#define SPGT_TRY(call) if (const int e_ = (call)) return e_

extern "C" int spgt_encoder_train_fwd(const spgt_encoder_params* p, const float* x, const float* pos, float* attention, int B, int S, float eps,
                                      void* saved, size_t saved_bytes, spgt_stream_t stream) {
    if (!p || !x || !pos || !attention || !saved || !train_params_ok(p)) return SPGT_ERR_NULL;
    if (!train_sizes_ok(B, S)) return SPGT_ERR_SHAPE;
    const TrainSaved t((size_t)B * S);
    if (saved_bytes < t.total * sizeof(float)) return SPGT_ERR_WORKSPACE;
    for (const void* v : {(const void*)x, (const void*)attention, (const void*)saved, (const void*)p->wq, (const void*)p->wk, (const void*)p->wv})
        if (!aligned16(v)) return SPGT_ERR_ALIGN;
    float* s = (float*)saved;
    SPGT_TRY(train_images(p, s, (cudaStream_t)stream));
    SPGT_TRY(projpos_qkv_mma(x, p->wq, p->bq, p->wk, p->bk, p->wv, p->bv, p->lnwk, p->lnbk, p->lnwv, p->lnbv, eps, pos, s + t.q, s + t.k, s + t.v, B, S,
                             ET_DP, (cudaStream_t)stream));
    return spgt_galerkin_attn_fwd(s + t.q, s + t.k, s + t.v, attention, nullptr, B, 4, 34, S, 1, stream);
}

extern "C" int spgt_encoder_train_bwd(const spgt_encoder_params* p, const spgt_encoder_grads* g, const float* x, const float* attention,
                                      const float* x1, const float* h, const float* dy, const float* dh, const float* dx1, const float* da,
                                      float* dx, int B, int S, float eps, const void* saved, size_t saved_bytes, void* workspace,
                                      size_t workspace_bytes, spgt_stream_t stream) {
    if (!p || !g || !x || !attention || !x1 || !h || !dy || !dh || !dx1 || !da || !dx || !saved || !workspace || !train_params_ok(p)) return SPGT_ERR_NULL;
    for (const float* v : {g->wqkv, g->bq, g->bk, g->bv, g->lnwk, g->lnbk, g->lnwv, g->lnbv})
        if (!v) return SPGT_ERR_NULL;
    const bool dense = g->wfc != nullptr;                  // (all six or none)
    for (const float* v : {g->bfc, g->w1, g->b1, g->w2, g->b2})
        if ((v != nullptr) != dense) return SPGT_ERR_NULL;
    if (!train_sizes_ok(B, S)) return SPGT_ERR_SHAPE;
    const TrainSaved t((size_t)B * S);
    const TrainScratch c(B, S);
    if (saved_bytes < t.total * sizeof(float) || workspace_bytes < c.total * sizeof(float)) return SPGT_ERR_WORKSPACE;
    for (const void* v : {(const void*)x, (const void*)attention, (const void*)x1, (const void*)h, (const void*)dy, (const void*)dh, (const void*)dx1,
                          (const void*)da, (const void*)dx, saved, (const void*)workspace})
        if (!aligned16(v)) return SPGT_ERR_ALIGN;
    const float* s = (const float*)saved;
    float* w = (float*)workspace;
    const int rows = B * S;
    const cudaStream_t st = (cudaStream_t)stream;
    void* tw = w + c.ws;
    // dense layers: dW = dy^T x as torch keeps it, [out][in]
    if (dense) {
        SPGT_TRY(tn_gemm(dy, ET_D, h, ET_F, g->w2, ET_F, 128, g->b2, true, ET_D, ET_F, rows, tw, c.ws_bytes, st));
        SPGT_TRY(tn_gemm(dh, ET_F, x1, ET_D, g->w1, ET_D, 128, g->b1, true, ET_F, ET_D, rows, tw, c.ws_bytes, st));
        SPGT_TRY(tn_gemm(dx1, ET_D, attention, ET_A, g->wfc, ET_A, 128, g->bfc, true, ET_D, ET_A, rows, tw, c.ws_bytes, st));
    }
    // attention, LayerNorm, projections
    SPGT_TRY(galerkin_attn_bwd(s + t.q, s + t.k, s + t.v, da, w + c.dq, w + c.dk, w + c.dv, B, 4, 34, S, true, tw, c.ws_bytes, st));
    SPGT_TRY(spgt_linear_tc_fwd(x, ET_D, s + ET_KV, s + ET_BKV, nullptr, ET_F, w + c.hkv, ET_F, rows, ET_D, ET_F, SPGT_ACT_NONE, stream));
    float *const db[3] = {g->bq, g->bk, g->bv}, *const dlnw[2] = {g->lnwk, g->lnwv}, *const dlnb[2] = {g->lnbk, g->lnbv};
    SPGT_TRY(projpos_bwd_qkv(w + c.dq, w + c.dk, w + c.dv, w + c.hkv, p->lnwk, p->lnwv, eps, w + c.dqkv, db, dlnw, dlnb, B, S, ET_DP, (float*)tw, st));
    SPGT_TRY(tn_gemm(x, ET_D, w + c.dqkv, 3 * ET_D, g->wqkv, ET_D, ET_D * ET_D, nullptr, false, ET_D, 3 * ET_D, rows, tw, c.ws_bytes, st));
    // (three products of 128 terms each on top of one another in fp32: one truncating chain of 384 is three times less accurate)
    for (int i = 0; i < 3; ++i)
        SPGT_TRY(spgt_linear_tc_fwd(w + c.dqkv + i * ET_D, 3 * ET_D, s + ET_QKV_T + i * ET_W, nullptr, i ? dx : dx1, ET_D, dx, ET_D, rows, ET_D, ET_D,
                                    SPGT_ACT_NONE, stream));
    return SPGT_OK;
}
