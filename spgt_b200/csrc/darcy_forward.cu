// The whole Darcy forward as one call: the launches of every stage issued from native code into one caller-provided
// workspace.  Issued op by op from Python a forward of small batches is bound by the host (about 27 us per op against 5 - 15 us
// of GPU time: 1.18 ms for one 141 x 141 field); from here a launch costs about 2 us of host time.
#include "common.cuh"

namespace spgt {

int decoder_head_tc(const float* x, const void* w1prep, const float* b1, const float* w2, float b2, const float* b2_dev, float scale, float shift,
                    const float* scale_map, const float* shift_map, int dirichlet, float* out, int B, int Hh, int Ww, int K, int N1, int act,
                    cudaStream_t st);      // tc_gemm.cu

static int pad4(int c) { return (c + 3) & ~3; }

// Workspace: the encoder's activations, which outlive the phases, then one region that the phases (down-scaler, encoder layer,
// up-scaler + decoder) reuse one after the other.  Offsets in floats, each a multiple of 64 floats.
struct DarcyPlan {
    size_t xa, phase, total;
    size_t d0, d1, d2, d3;                      // down-scaler: conv0 output and the three convolution outputs
    size_t es, es_bytes;                        // encoder layer scratch
    size_t up, uc, uw, y[2], ws, ws_bytes;      // up-scaler and decoder
};

static bool darcy_plan(const spgt_darcy_model* m, int B, DarcyPlan& p) {
    if (!m || B <= 0 || m->r <= 0 || m->mid <= 0 || m->ra <= 0 || m->n_encoder < 0 || m->n_decoder < 0) return false;
    if (m->n_encoder > SPGT_MAX_LAYERS || m->n_decoder > SPGT_MAX_LAYERS || m->d_pos != 2) return false;
    if (m->c1 <= 0 || m->c2 <= 0 || m->c3 <= 0 || m->c1 + m->c2 + m->c3 != 128) return false;
    const size_t b = (size_t)B, S = (size_t)m->ra * m->ra, M = (size_t)m->mid * m->mid, R = (size_t)m->r * m->r;
    p.ws_bytes = m->n_decoder > 0 ? spgt_spectral_workspace_bytes(B, m->r, m->modes, 32) : 0;
    if (m->n_decoder > 0 && p.ws_bytes == 0) return false;
    size_t at = 0;
    auto take = [&](size_t& off, size_t floats) { off = at; at += (floats + 63) & ~(size_t)63; };
    take(p.xa, b * S * 128);
    p.phase = at;
    take(p.d0, b * M * 128);
    take(p.d1, b * M * pad4(m->c1));
    take(p.d2, b * M * pad4(m->c2));
    take(p.d3, b * M * pad4(m->c3));
    p.total = at;
    at = p.phase;
    p.es_bytes = spgt_encoder_workspace_bytes(B, (int)S);
    if (p.es_bytes == 0) return false;
    take(p.es, (p.es_bytes + 3) / 4);
    if (at > p.total) p.total = at;
    at = p.phase;
    take(p.up, b * M * 128);
    take(p.uc, b * M * 128);
    take(p.uw, b * M * 32);
    take(p.y[0], b * R * 32);
    take(p.y[1], b * R * 32);
    take(p.ws, (p.ws_bytes + 3) / 4);
    if (at > p.total) p.total = at;
    return true;
}

}  // namespace spgt

using namespace spgt;

extern "C" size_t spgt_darcy_workspace_bytes(const spgt_darcy_model* m, int B) {
    DarcyPlan p;
    return darcy_plan(m, B, p) ? p.total * sizeof(float) : 0;
}

extern "C" int spgt_darcy_launches(const spgt_darcy_model* m, int B) {
    DarcyPlan p;
    if (!darcy_plan(m, B, p)) return 0;
    return 5 + 3 * m->n_encoder + 4 + m->n_decoder * spgt_spectral_launches(B, m->r, m->modes) + 1;
}

extern "C" int spgt_darcy_forward(const spgt_darcy_model* m, const float* node, const float* position, const float* grid, float* out,
                                  int B, float* const* taps, void* workspace, size_t workspace_bytes, spgt_stream_t stream) {
    return spgt_darcy_forward_devbias(m, nullptr, node, position, grid, out, B, taps, workspace, workspace_bytes, stream);
}

extern "C" int spgt_darcy_forward_devbias(const spgt_darcy_model* m, const float* head_b2, const float* node, const float* position,
                                          const float* grid, float* out, int B, float* const* taps, void* workspace, size_t workspace_bytes,
                                          spgt_stream_t stream) {
    if (!m || !node || !position || !grid || !out || !workspace) return SPGT_ERR_NULL;
    DarcyPlan p;
    if (!darcy_plan(m, B, p)) return SPGT_ERR_SHAPE;
    if (workspace_bytes < p.total * sizeof(float)) return SPGT_ERR_WORKSPACE;
    if (!aligned16(workspace)) return SPGT_ERR_ALIGN;
    const ChainScope chain;
    float* ws = (float*)workspace;
    const int mid = m->mid, ra = m->ra, r = m->r, S = ra * ra, D = 128;
    const size_t xa_bytes = (size_t)B * S * D * sizeof(float);
    int rc;
#define SPGT_TRY(call) if ((rc = (call)) != SPGT_OK) return rc
    auto tap = [&](int i, const float* src, size_t bytes) {
        if (!taps || !taps[i]) return SPGT_OK;
        const cudaError_t e = cudaMemcpyAsync(taps[i], src, bytes, cudaMemcpyDeviceToDevice, (cudaStream_t)stream);
        if (e != cudaSuccess) { g_last_cuda_error = (int)e; return SPGT_ERR_LAUNCH; }
        return SPGT_OK;
    };
    // down-scaler
    const int p1 = pad4(m->c1), p2 = pad4(m->c2), p3 = pad4(m->c3);
    SPGT_TRY(spgt_conv0_down_fwd(node, m->conv0_w, m->conv0_b, ws + p.d0, B, r, r, mid, mid, D, m->act_down, stream));
    SPGT_TRY(spgt_conv3x3_nhwc_fwd(ws + p.d0, D, 0, D, m->conv_w[0], m->conv_b[0], ws + p.d1, p1, 0, p1, B, mid, mid, m->act_down, stream));
    SPGT_TRY(spgt_conv3x3_nhwc_fwd(ws + p.d1, p1, 0, p1, m->conv_w[1], m->conv_b[1], ws + p.d2, p2, 0, p2, B, mid, mid, m->act_down, stream));
    SPGT_TRY(spgt_conv3x3_nhwc_fwd(ws + p.d2, p2, 0, p2, m->conv_w[2], m->conv_b[2], ws + p.d3, p3, 0, p3, B, mid, mid, m->act_down, stream));
    SPGT_TRY(spgt_bilinear_concat3_fwd(ws + p.d1, ws + p.d2, ws + p.d3, p1, p2, p3, m->c1, m->c2, m->c3, ws + p.xa, B, mid, mid, ra, ra,
                                       m->act_down, stream));
    SPGT_TRY(tap(0, ws + p.xa, xa_bytes));
    // encoder
    float* x = ws + p.xa;
    for (int l = 0; l < m->n_encoder; ++l) {
        const spgt_encoder_weights& w = m->encoder[l];
        SPGT_TRY(spgt_encoder_layer_fwd(&w, x, position, x, B, S, m->eps, m->act_ffn, 1, 1, ws + p.es, p.es_bytes, stream));
        SPGT_TRY(tap(1 + l, x, xa_bytes));
    }
    // up-scaler (its last interpolation is fused with the decoder's spatial fc)
    SPGT_TRY(spgt_bilinear_fwd(x, ws + p.up, B, ra, ra, mid, mid, D, SPGT_ACT_NONE, stream));
    SPGT_TRY(spgt_conv3x3_nhwc_fwd(ws + p.up, D, 0, D, m->up_w, m->up_b, ws + p.uc, D, 0, D, B, mid, mid, m->act_up, stream));
    SPGT_TRY(tap(1 + m->n_encoder, ws + p.uc, (size_t)B * mid * mid * D * sizeof(float)));
    // decoder
    SPGT_TRY(spgt_linear_tc_fwd(ws + p.uc, D, m->fcx_w, nullptr, nullptr, 32, ws + p.uw, 32, B * mid * mid, D, 32, SPGT_ACT_NONE, stream));
    SPGT_TRY(spgt_upsample_grid_fwd(ws + p.uw, grid, m->fcg_w, m->fc_b, ws + p.y[0], B, mid, mid, r, r, 32, stream));
    for (int l = 0; l < m->n_decoder; ++l) {
        const spgt_spectral_weights& w = m->decoder[l];
        SPGT_TRY(spgt_spectral_conv2d_fwd(ws + p.y[l & 1], w.wr, w.br, w.fw0, w.fw1, m->tables, ws + p.ws, p.ws_bytes, ws + p.y[(l + 1) & 1], B, r,
                                          32, m->modes, m->act_dec, stream));
    }
    SPGT_TRY(decoder_head_tc(ws + p.y[m->n_decoder & 1], m->head_w1, m->head_b1, m->head_w2, m->b2, head_b2, m->scale, m->shift, m->scale_map,
                             m->shift_map, m->dirichlet, out, B, r, r, 32, 128, m->act_dec, (cudaStream_t)stream));
#undef SPGT_TRY
    return SPGT_OK;
}
