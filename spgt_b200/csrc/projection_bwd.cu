// Backward of the multi-head projection (+ per-head LayerNorm) + position op, element-wise part.
// Reference: multihead_projection_with_position_rrc_backward / multihead_projection_layernorm_with_position_rrc_backward
// (extension/bind/galerkin_attention.cu:26-48, 70-102) and lnorm_grad_ccc_cuda (extension/native/multihead_dim32.cu).
//
// Forward:  h = x W + b  [rows = B*S, D = H*32];  per (row, head): hat = (h - mu) * invsigma, y = hat * lnw + lnb;
//           out[b, h, d_pos + c, s] = y[b*S + s, 32 h + c]  (position rows carry no gradient).
// This kernel takes grad_out [B, H, d_pos + 32, S] and the recomputed h and produces
//   dh [rows, D]  (the gradient with respect to h, row-major: the A operand of the two GEMMs dX = dh W^T and dW = x^T dh),
//   per-block sums of  db = sum_rows dh,  dlnw = sum_rows g * hat,  dlnb = sum_rows g   (g = gathered grad_out),
// which a second kernel adds up in block order (deterministic).  Without LayerNorm (lnw == nullptr) dh = g.
// A warp works on one head, a lane on one grid node with all 32 channels in registers: the LayerNorm sums need no shuffles, and
// the parameter sums stay in registers until the block's last node (a block of one node per iteration and a warp reduction
// per row took 44 us for 65536 rows, the serial addition of its 2048 partial sums another 66 us).
#include "common.cuh"

namespace spgt {

constexpr int PB_ROWS = 32;      // grid nodes per warp and iteration

// Rows of h and dh have pitches ldh and ldd.  VEC: they start at 16-byte boundaries.
template <bool LN, bool VEC = true>
__device__ __forceinline__ void proj_bwd_body(const float* __restrict__ grad_out, const float* __restrict__ h, int ldh, const float* __restrict__ lnw,
                                              float* __restrict__ dh, int ldd, float* __restrict__ partial, int S, int H, int d_pos, float eps,
                                              int tiles_per_sample, int tiles) {
    extern __shared__ float red[];                        // [H][32][33]
    const int D = H * 32, dpk = d_pos + 32;
    const int lane = threadIdx.x & 31, head = threadIdx.x >> 5;
    float w[32], db[32], dw[32], dbt[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) { w[c] = LN ? __ldg(lnw + head * 32 + c) : 1.0f; db[c] = dw[c] = dbt[c] = 0.0f; }
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int b = tile / tiles_per_sample, s = (tile - b * tiles_per_sample) * PB_ROWS + lane;
        if (s >= S) continue;
        const int64_t row = (int64_t)b * S + s;
        const float* gp = grad_out + (((int64_t)b * H + head) * dpk + d_pos) * S + s;
        float g[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) g[c] = __ldg(gp + (int64_t)c * S);              // lanes = consecutive nodes
        if constexpr (LN) {
            float v[32], mu = 0.0f, var = 0.0f, m1 = 0.0f, m2 = 0.0f;
            const float* hp = h + row * ldh + head * 32;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 q = VEC ? __ldg(reinterpret_cast<const float4*>(hp) + j) : make_float4(__ldg(hp + 4 * j), __ldg(hp + 4 * j + 1), __ldg(hp + 4 * j + 2), __ldg(hp + 4 * j + 3));
                v[4 * j] = q.x; v[4 * j + 1] = q.y; v[4 * j + 2] = q.z; v[4 * j + 3] = q.w;
                mu += (q.x + q.y) + (q.z + q.w);
            }
            mu *= 1.0f / 32.0f;
#pragma unroll
            for (int c = 0; c < 32; ++c) { v[c] -= mu; var = fmaf(v[c], v[c], var); }
            const float inv = 1.0f / sqrtf(var * (1.0f / 32.0f) + eps);
#pragma unroll
            for (int c = 0; c < 32; ++c) {
                v[c] *= inv;                              // hat
                dw[c] = fmaf(g[c], v[c], dw[c]);
                dbt[c] += g[c];
                g[c] *= w[c];                             // gradient of hat
                m1 += g[c];
                m2 = fmaf(g[c], v[c], m2);
            }
            m1 *= 1.0f / 32.0f; m2 *= 1.0f / 32.0f;
#pragma unroll
            for (int c = 0; c < 32; ++c) g[c] = inv * (g[c] - m1 - v[c] * m2);
        }
        float* dp = dh + row * ldd + head * 32;
        if constexpr (VEC) {
#pragma unroll
            for (int j = 0; j < 8; ++j) reinterpret_cast<float4*>(dp)[j] = make_float4(g[4 * j], g[4 * j + 1], g[4 * j + 2], g[4 * j + 3]);
        } else {
#pragma unroll
            for (int c = 0; c < 32; ++c) dp[c] = g[c];
        }
#pragma unroll
        for (int c = 0; c < 32; ++c) db[c] += g[c];
    }
    // lane sums -> channel sums: through a padded square per warp
    float* sq = red + head * (32 * 33);
    float* p = partial + (int64_t)blockIdx.x * 3 * D + head * 32 + lane;
    auto columns = [&](const float (&v)[32], int which) {
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 32; ++c) sq[lane * 33 + c] = v[c];
        __syncwarp();
        float t = 0.0f;
#pragma unroll
        for (int k = 0; k < 32; ++k) t += sq[k * 33 + lane];
        p[which * D] = t;
    };
    columns(db, 0);
    if (LN) { columns(dw, 1); columns(dbt, 2); }
}

template <bool LN, bool VEC>
__global__ void __launch_bounds__(256)
proj_bwd_kernel(const float* __restrict__ grad_out, const float* __restrict__ h, const float* __restrict__ lnw,
                float* __restrict__ dh, float* __restrict__ partial, int S, int H, int d_pos, float eps, int tiles_per_sample, int tiles) {
    proj_bwd_body<LN, VEC>(grad_out, h, H * 32, lnw, dh, H * 32, partial, S, H, d_pos, eps, tiles_per_sample, tiles);
}

// Q, K and V of a layer in one launch (blockIdx.y): dh [rows, 384] = dq | dk | dv, h [rows, 256] = K | V before their LayerNorm
struct ProjBwdQkv { const float *grad[3], *h, *lnw[3]; float *dh, *partial; };
__global__ void __launch_bounds__(128)
proj_bwd_qkv_kernel(const ProjBwdQkv p, int S, int d_pos, float eps, int tiles_per_sample, int tiles) {
    const int w = blockIdx.y;
    float* partial = p.partial + (int64_t)w * gridDim.x * 384;
    if (w == 0) proj_bwd_body<false>(p.grad[0], nullptr, 0, nullptr, p.dh, 384, partial, S, 4, d_pos, eps, tiles_per_sample, tiles);
    else proj_bwd_body<true>(p.grad[w], p.h + (w - 1) * 128, 256, p.lnw[w], p.dh + w * 128, 384, partial, S, 4, d_pos, eps, tiles_per_sample, tiles);
}

// 32 columns per block, eight threads per column take every eighth partial sum
__device__ __forceinline__ void proj_bwd_reduce_body(const float* __restrict__ partial, float* __restrict__ db, float* __restrict__ dlnw,
                                                     float* __restrict__ dlnb, int D, int nblocks) {
    __shared__ float red[8][33];
    const int c = threadIdx.x & 31, k0 = threadIdx.x >> 5, i = blockIdx.x * 32 + c;
    float s = 0.0f;
#pragma unroll 8
    for (int k = k0; k < nblocks; k += 8) s += __ldg(partial + (int64_t)k * 3 * D + i);
    red[k0][c] = s;
    __syncthreads();
    if (k0 == 0) {
#pragma unroll
        for (int k = 1; k < 8; ++k) s += red[k][c];
        float* dst = i < D ? db : (i < 2 * D ? dlnw : dlnb);
        if (dst != nullptr) dst[i % D] = s;
    }
}

__global__ void __launch_bounds__(256)
proj_bwd_reduce_kernel(const float* __restrict__ partial, float* __restrict__ db, float* __restrict__ dlnw, float* __restrict__ dlnb,
                       int D, int nblocks) {
    proj_bwd_reduce_body(partial, db, dlnw, dlnb, D, nblocks);
}

struct ProjBwdQkvOut { float *db[3], *dlnw[3], *dlnb[3]; };
__global__ void __launch_bounds__(256)
proj_bwd_reduce_qkv_kernel(const float* __restrict__ partial, const ProjBwdQkvOut o, int nblocks) {
    const int w = blockIdx.y;
    if (w == 0 && blockIdx.x >= 4) return;                 // (Q has no LayerNorm)
    proj_bwd_reduce_body(partial + (int64_t)w * nblocks * 384, o.db[w], o.dlnw[w], o.dlnb[w], 128, nblocks);
}

static int proj_bwd_blocks(int B, int S, int H) {          // enough warps for eight per SM sub-partition, one tile each at least
    const int64_t tiles = (int64_t)B * ceil_div(S, PB_ROWS), most = (int64_t)num_sms() * (H <= 4 ? 2 : 1);
    return (int)(tiles < most ? tiles : most);
}

size_t projpos_bwd_qkv_workspace_bytes(int B, int S) { return (size_t)3 * proj_bwd_blocks(B, S, 4) * 384 * sizeof(float); }

// Width 128, four heads.  grad_* [B,4,d_pos+32,S], h [B*S,256] -> dh [B*S,384] and the parameter sums of the three projections.
int projpos_bwd_qkv(const float* grad_q, const float* grad_k, const float* grad_v, const float* h, const float* lnwk, const float* lnwv, float eps,
                    float* dh, float* const* db, float* const* dlnw, float* const* dlnb, int B, int S, int d_pos, float* workspace, cudaStream_t st) {
    const int tps = ceil_div(S, PB_ROWS), blocks = proj_bwd_blocks(B, S, 4);
    const ProjBwdQkv p{{grad_q, grad_k, grad_v}, h, {nullptr, lnwk, lnwv}, dh, workspace};
    proj_bwd_qkv_kernel<<<dim3((unsigned)blocks, 3), 128, (size_t)128 * 33 * sizeof(float), st>>>(p, S, d_pos, eps, tps, B * tps);
    if (int e = launch_status()) return e;
    const ProjBwdQkvOut o{{db[0], db[1], db[2]}, {nullptr, dlnw[0], dlnw[1]}, {nullptr, dlnb[0], dlnb[1]}};
    proj_bwd_reduce_qkv_kernel<<<dim3(12, 3), 256, 0, st>>>(workspace, o, blocks);
    return launch_status();
}

}  // namespace spgt

using namespace spgt;

extern "C" size_t spgt_projpos_bwd_workspace_bytes(int B, int S, int H) {
    if (B <= 0 || S <= 0 || H <= 0 || H > 8) return 0;
    return (size_t)proj_bwd_blocks(B, S, H) * 3 * H * 32 * sizeof(float);
}

extern "C" int spgt_projpos_bwd_elementwise(const float* grad_out, const float* h, const float* ln_weight, float eps, float* dh,
                                            float* db, float* dlnw, float* dlnb, int B, int S, int H, int d_head, int d_pos,
                                            void* workspace, size_t workspace_bytes, spgt_stream_t stream) {
    if (!grad_out || !dh) return SPGT_ERR_NULL;
    if (ln_weight && !h) return SPGT_ERR_NULL;
    if (B <= 0 || S <= 0 || H <= 0 || H > 8 || d_head != 32 || d_pos < 0 || d_pos > 8) return SPGT_ERR_SHAPE;
    const int tps = ceil_div(S, PB_ROWS);
    if ((int64_t)B * tps > 0x7fffffffLL) return SPGT_ERR_SHAPE;
    if (!workspace || workspace_bytes < spgt_projpos_bwd_workspace_bytes(B, S, H)) return SPGT_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    const int D = H * 32, blocks = proj_bwd_blocks(B, S, H);
    const bool vec = (!h || aligned16(h)) && aligned16(dh);
    auto kern = ln_weight ? (vec ? proj_bwd_kernel<true, true> : proj_bwd_kernel<true, false>) : (vec ? proj_bwd_kernel<false, true> : proj_bwd_kernel<false, false>);
    kern<<<(unsigned)blocks, H * 32, (size_t)H * 32 * 33 * sizeof(float), st>>>(grad_out, h, ln_weight, dh, (float*)workspace, S, H, d_pos, eps, tps,
                                                                             B * tps);
    if (int e = launch_status()) return e;
    proj_bwd_reduce_kernel<<<(ln_weight ? 3 : 1) * D / 32, 256, 0, st>>>((const float*)workspace, db, ln_weight ? dlnw : nullptr,
                                                                         ln_weight ? dlnb : nullptr, D, blocks);
    return launch_status();
}
