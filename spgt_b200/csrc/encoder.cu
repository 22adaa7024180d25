// Host side of the fused encoder layer: workspace, launches, status (kernels: encoder_kv.cu, encoder_fold.cu, encoder_out.cu).
#include "encoder_common.cuh"

namespace spgt {

int encoder_kv(const float* x, const void* wkv, const float* bk, const float* bv, float eps, const float* pos, float* partial, int S,
               const EncoderSplit& sp, cudaStream_t st);
int encoder_fold(const float* partial, const spgt_encoder_weights& w, float* m_img, float* pc, int B, int S, const EncoderSplit& sp, cudaStream_t st);
int encoder_out(const float* x, const float* m_img, const float* pc, const float* pos, const void* w1, const float* b1, const void* w2,
                const float* b2, float* y, int B, int S, int act, bool ffn, bool residual, cudaStream_t st);

static size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

}  // namespace spgt

using namespace spgt;

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
