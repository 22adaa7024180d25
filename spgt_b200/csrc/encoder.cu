// Host side of the fused encoder layer: workspace, launches, status (kernels: encoder_kv.cu, encoder_fold.cu, encoder_out.cu).
#include "encoder_common.cuh"

namespace spgt {

int encoder_kv(const float* x, const void* wkv, const float* bk, const float* bv, float eps, const float* pos, float* partial, int S,
               const EncoderSplit& sp, cudaStream_t st);
int encoder_fold(const float* partial, const spgt_encoder_weights& w, float* m_img, float* pc, int B, int S, const EncoderSplit& sp, cudaStream_t st);
int encoder_out(const float* x, const float* m_img, const float* pc, const float* pos, const void* w1, const float* b1, const void* w2,
                const float* b2, float* y, int B, int S, int act, bool ffn, bool residual, cudaStream_t st);

int tc_weight_prepare_jobs(const TcPrepJobs& jobs, int n, cudaStream_t st);                          // tc_gemm.cu

static size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

}  // namespace spgt

using namespace spgt;

// Images of wkv, w1 and w2, one after the other: each 2 column tiles x 4 k-blocks (w2: 1 x 8) of 2 * 128 * 32 floats.
constexpr size_t EN_IMAGE = (size_t)8 * 2 * 128 * 32 * sizeof(float);

extern "C" size_t spgt_encoder_weights_bytes(int ffn) { return (ffn ? 3 : 1) * EN_IMAGE; }

extern "C" int spgt_encoder_weights_prepare(const float* wk, const float* wv, const float* w1, const float* w2, void* images, size_t bytes,
                                            spgt_stream_t stream) {
    if (!wk || !wv || !images || (w1 != nullptr) != (w2 != nullptr)) return SPGT_ERR_NULL;
    if (bytes < spgt_encoder_weights_bytes(w1 != nullptr)) return SPGT_ERR_WORKSPACE;
    if (!aligned16(images)) return SPGT_ERR_ALIGN;
    float* img = (float*)images;
    TcPrepJobs jobs;
    jobs.job[0] = {wk, img, 3, EN_D, EN_D, 2 * EN_D, EN_D, 128, wv};
    jobs.job[1] = {w1, img + EN_IMAGE / sizeof(float), 1, EN_D, EN_D, 2 * EN_D, EN_D, 128, nullptr};
    jobs.job[2] = {w2, img + 2 * (EN_IMAGE / sizeof(float)), 1, 2 * EN_D, 2 * EN_D, EN_D, 2 * EN_D, 128, nullptr};
    return tc_weight_prepare_jobs(jobs, w1 ? 3 : 1, (cudaStream_t)stream);
}

extern "C" size_t spgt_encoder_workspace_bytes(int B, int S) {
    if (B <= 0 || S <= 0 || (int64_t)B * ceil_div(S, EN_ROWS) > 0x7fffffffLL / EN_ROWS) return 0;
    const EncoderSplit sp = encoder_split(B, S, num_sms());
    return align256((size_t)B * EN_PAIRS * sp.max_parts * EN_P_FLOATS * 4) + (size_t)B * (2 * EN_D * EN_D) * 4 + align256((size_t)B * 3 * EN_D * 4);
}

extern "C" int spgt_encoder_layer_fwd(const spgt_encoder_weights* w, const float* x, const float* pos, float* y, int B, int S, float eps, int act,
                                      int ffn, int residual, void* workspace, size_t workspace_bytes, spgt_stream_t stream) {
    if (!w || !x || !pos || !y || !workspace || !w->wkv || !w->wq || !w->lnwk || !w->lnbk || !w->lnwv || !w->lnbv || !w->wfc) return SPGT_ERR_NULL;
    if (ffn && (!w->w1 || !w->b1 || !w->w2)) return SPGT_ERR_NULL;
    if (act < 0 || act > 3) return SPGT_ERR_SHAPE;
    const size_t need = spgt_encoder_workspace_bytes(B, S);
    if (need == 0) return SPGT_ERR_SHAPE;
    if (workspace_bytes < need) return SPGT_ERR_WORKSPACE;
    if (!aligned16(x) || (reinterpret_cast<uintptr_t>(pos) & 7u) || !aligned16(y) || !aligned16(workspace) || !aligned16(w->wkv) || !aligned16(w->wq) || !aligned16(w->wfc) ||
        (ffn && (!aligned16(w->w1) || !aligned16(w->w2))))
        return SPGT_ERR_ALIGN;
    const EncoderSplit sp = encoder_split(B, S, num_sms());
    float* partial = (float*)workspace;
    float* m_img = (float*)((char*)workspace + align256((size_t)B * EN_PAIRS * sp.max_parts * EN_P_FLOATS * 4));
    float* pc = m_img + (size_t)B * (2 * EN_D * EN_D);
    const cudaStream_t st = (cudaStream_t)stream;
    const ChainScope chain;
    if (int e = encoder_kv(x, w->wkv, w->bk, w->bv, eps, pos, partial, S, sp, st)) return e;
    if (int e = encoder_fold(partial, *w, m_img, pc, B, S, sp, st)) return e;
    return encoder_out(x, m_img, pc, pos, w->w1, w->b1, w->w2, w->b2, y, B, S, act, ffn != 0, residual != 0, st);
}
