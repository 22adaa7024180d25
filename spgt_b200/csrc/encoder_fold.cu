// Folds T, Wq and Wfc of one encoder layer into the per-sample affine map of encoder_common.cuh: M (as the W image that
// encoder_out_kernel streams), P and c.
//
// One cluster of eight blocks per sample.  Block `rank` adds the partial sums of half a head (17 rows of T, in block order), applies
// the LayerNorm's weight and bias and hands its rows to the others through distributed shared memory; then it produces 16 of
// the 128 output columns: G = T Wfc (136 x 34 x 16) and M = Wq G' (128 x 128 x 16), both 3xTF32 on warp-level MMAs (with
// fp32 FMAs the operand reads from shared memory took 16000 of 29000 cycles).  Wq goes from global memory straight into operand
// fragments, loaded before the partial sums are needed.  Bound by the latency of its steps: on its own 13 us for 8 samples, 30 for 64.
#include "encoder_common.cuh"

namespace spgt {

constexpr int FO_CL = 8, FO_N = EN_D / FO_CL, FO_THREADS = 256, FO_ROWS = 17;
constexpr int FO_TP = 44, FO_WP = 24, FO_GP = 18;              // pitches of T, Wfc and G' rows: fragment reads without bank conflicts
// a block's sums: its 17 rows of products, then (pos 0, pos 1, 1) sums of K [3][32] and V [3][32] of its head, position sums
constexpr int FO_K = FO_ROWS * 32, FO_V = FO_K + 96, FO_POS = FO_V + 96, FO_SUMS = FO_POS + 8;
constexpr size_t FO_SMEM = (size_t)(FO_SUMS + FO_ROWS * FO_TP + 4 * 48 * FO_TP + 4 * 40 * FO_WP + EN_D * FO_GP + 8 * FO_N + 128 + 128 + 256) * sizeof(float);

__device__ __forceinline__ float4 ld_dsmem_f32x4(const float* local_smem_ptr, uint32_t rank) {
    uint32_t remote;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_u32(local_smem_ptr)), "r"(rank));
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote));
    return v;
}

__global__ void __cluster_dims__(FO_CL, 1, 1) __launch_bounds__(FO_THREADS, 2)
encoder_fold_kernel(const float* __restrict__ partial, const float* __restrict__ wq, const float* __restrict__ bq, const float* __restrict__ lnwk,
                    const float* __restrict__ lnbk, const float* __restrict__ lnwv, const float* __restrict__ lnbv,
                    const float* __restrict__ wfc, const float* __restrict__ bfc, float* __restrict__ m_img, float* __restrict__ pc, int S,
                    EncoderSplit sp) {
    extern __shared__ __align__(16) float fsm[];
    float* s_sum = fsm;                           // [FO_SUMS]
    float* s_own = s_sum + FO_SUMS;               // this block's rows of T
    float* s_t = s_own + FO_ROWS * FO_TP;         // T: four heads of 48 rows, 34 used
    float* s_wfc = s_t + 4 * 48 * FO_TP;          // four heads of 40 rows
    float* s_g = s_wfc + 4 * 40 * FO_WP;          // G': the 128 channel rows of G
    float* s_gp = s_g + EN_D * FO_GP;             // its position rows [head][2][16]
    float *s_ln = s_gp + 8 * FO_N, *s_bq = s_ln + 128, *s_red = s_bq + 128;
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, fg = lane >> 2, ft = lane & 3, b = blockIdx.x / FO_CL;
    const uint32_t rank = cluster_ctarank();
    const int n0 = (int)rank * FO_N, h = (int)rank >> 1, hh = h & 1, r0 = ((int)rank & 1) * FO_ROWS;      // head, head in its pair, first row of T_h
    // Wq rows 16 warp + fg and + 8 as A fragments: chunk kb covers 16 channels, of which this lane holds 4 ft .. 4 ft + 3; k-step e (0, 1)
    // of the chunk takes channels 4 ft + 2 e as k = ft and 4 ft + 2 e + 1 as k = ft + 4 (the order of a sum's terms is free).
    float4 wa[8], wb[8];
#pragma unroll
    for (int kb = 0; kb < 8; ++kb) {
        wa[kb] = __ldg(reinterpret_cast<const float4*>(wq + (warp * 16 + fg) * EN_D + kb * 16) + ft);
        wb[kb] = __ldg(reinterpret_cast<const float4*>(wq + (warp * 16 + fg + 8) * EN_D + kb * 16) + ft);
    }
    // Wfc columns n0 .. n0 + 15, from the weight as torch keeps it: [128 out][136 in]; rows 34 - 39 of a head are zero
    for (int i = t; i < FO_N * 34; i += FO_THREADS) {
        const int n = i / 34, j4 = i - n * 34;
        const float4 w = __ldg(reinterpret_cast<const float4*>(wfc + (n0 + n) * 136) + j4);
        const float ws[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) { const int j = 4 * j4 + e; s_wfc[((j / 34) * 40 + j % 34) * FO_WP + n] = ws[e]; }
    }
    for (int i = t; i < 4 * 6 * FO_N; i += FO_THREADS) s_wfc[((i / 96) * 40 + 34 + (i % 96) / FO_N) * FO_WP + i % FO_N] = 0.0f;
    if (t < 128) {
        const float* ln = t < 32 ? lnwk : t < 64 ? lnbk : t < 96 ? lnwv : lnbv;        // this head's LayerNorm: wk | bk | wv | bv
        s_ln[t] = __ldg(ln + h * 32 + (t & 31));
        s_bq[t] = bq ? __ldg(bq + t) : 0.0f;
    }
    pdl_wait();
    pdl_launch_next();
    const int first = sp.owner(b * sp.tps), parts = sp.owner(b * sp.tps + sp.tps - 1) - first + 1;
    static_assert(FO_SUMS % 4 == 0 && FO_SUMS / 4 <= FO_THREADS, "one sum of four values per thread");
    if (t < FO_SUMS / 4) {
        const int i = 4 * t;
        int e;                                    // element of a partial-sum record
        if (i < FO_K) { const int row = r0 - 2 + (i >> 5); e = row < 0 ? 0 : EN_P_CORE + (hh * 32 + row) * 32 + (i & 31); }      // (rows below 0: unused)
        else if (i < FO_V) e = EN_P_K + ((i - FO_K) >> 5) * 64 + hh * 32 + (i & 31);
        else if (i < FO_POS) e = EN_P_V + ((i - FO_V) >> 5) * 64 + hh * 32 + (i & 31);
        else e = EN_P_POS + i - FO_POS;
        const float4* src = reinterpret_cast<const float4*>(partial + (int64_t)(b * EN_PAIRS + (h >> 1)) * sp.max_parts * EN_P_FLOATS + e);
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int k = 0; k < parts; ++k) {
            const float4 v = __ldca(src + (int64_t)k * (EN_P_FLOATS / 4));
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        *reinterpret_cast<float4*>(s_sum + i) = s;
    }
    __syncthreads();
    // rows r0 .. r0 + 16 of T_h, with the LayerNorm's weight and bias and 1 / S; columns 34 - 39 are zero
    {
        const float inv_s = 1.0f / (float)S;
        const float *K = s_sum + FO_K, *V = s_sum + FO_V, *P = s_sum + FO_POS;
        for (int i = t; i < FO_ROWS * FO_TP; i += FO_THREADS) {
            const int q = i / FO_TP, j = i - q * FO_TP, r = r0 + q, c = r - 2, d = j - 2;
            float v;
            if (j >= 34) v = 0.0f;
            else if (r < 2 && j < 2) v = P[r + j];
            else if (r < 2) v = s_ln[64 + d] * V[r * 32 + d] + s_ln[96 + d] * P[3 + r];
            else if (j < 2) v = s_ln[c] * K[j * 32 + c] + s_ln[32 + c] * P[3 + j];
            else v = s_ln[c] * (s_ln[64 + d] * s_sum[q * 32 + d] + s_ln[96 + d] * K[64 + c]) + s_ln[32 + c] * (s_ln[64 + d] * V[64 + d] + s_ln[96 + d] * (float)S);
            s_own[i] = v * inv_s;
        }
    }
    cluster_sync_all();
#pragma unroll
    for (int i = t; i < FO_CL * FO_ROWS * (FO_TP / 4); i += FO_THREADS) {
        const int r = i / (FO_ROWS * FO_TP / 4), e = i - r * (FO_ROWS * FO_TP / 4);
        *reinterpret_cast<float4*>(s_t + ((r >> 1) * 48 + (r & 1) * FO_ROWS) * FO_TP + 4 * e) = ld_dsmem_f32x4(s_own + 4 * e, (uint32_t)r);
    }
    cluster_sync_all();                           // (every block has read before any leaves)
    // G = T Wfc: twelve 16-row tiles (three per head, rows from 34 on are not used), 16 columns, k = 40
    for (int mt = warp; mt < 12; mt += FO_THREADS / 32) {
        const int gh = mt / 3, m0 = (mt - gh * 3) * 16;
        const float* A = s_t + (gh * 48 + m0 + fg) * FO_TP + ft;
        const float* B = s_wfc + (gh * 40 + ft) * FO_WP + fg;
        float c[2][4] = {};
#pragma unroll
        for (int k8 = 0; k8 < 5; ++k8) {
            uint32_t ah[4], al[4];
            split_tf32(A[k8 * 8], ah[0], al[0]); split_tf32(A[8 * FO_TP + k8 * 8], ah[1], al[1]);
            split_tf32(A[k8 * 8 + 4], ah[2], al[2]); split_tf32(A[8 * FO_TP + k8 * 8 + 4], ah[3], al[3]);
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                uint32_t bh[2], bl[2];
                split_tf32(B[k8 * 8 * FO_WP + n * 8], bh[0], bl[0]); split_tf32(B[(k8 * 8 + 4) * FO_WP + n * 8], bh[1], bl[1]);
                mma_3xtf32(c[n], ah, al, bh, bl);
            }
        }
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = m0 + fg + (e >> 1) * 8, col = n * 8 + 2 * ft + (e & 1);
                if (r < 2) s_gp[(gh * 2 + r) * FO_N + col] = c[n][e];
                else if (r < 34) s_g[(gh * 32 + r - 2) * FO_GP + col] = c[n][e];
            }
    }
    __syncthreads();
    // M rows 16 warp .. + 15, 16 columns
    {
        float c[2][4] = {};
#pragma unroll
        for (int kb = 0; kb < 8; ++kb) {
            const float a0[4] = {wa[kb].x, wa[kb].y, wa[kb].z, wa[kb].w}, a1[4] = {wb[kb].x, wb[kb].y, wb[kb].z, wb[kb].w};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                uint32_t ah[4], al[4];
                split_tf32(a0[2 * e], ah[0], al[0]); split_tf32(a1[2 * e], ah[1], al[1]);
                split_tf32(a0[2 * e + 1], ah[2], al[2]); split_tf32(a1[2 * e + 1], ah[3], al[3]);
                const float* B = s_g + (kb * 16 + 4 * ft + 2 * e) * FO_GP + fg;
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    uint32_t bh[2], bl[2];
                    split_tf32(B[n * 8], bh[0], bl[0]); split_tf32(B[FO_GP + n * 8], bh[1], bl[1]);
                    mma_3xtf32(c[n], ah, al, bh, bl);
                }
            }
        }
        float* img = m_img + (int64_t)b * (EN_D * EN_D * 2);
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int k = warp * 16 + fg + (e >> 1) * 8;
                tc_img_store(img + (k >> 5) * 8192, 128, n0 + n * 8 + 2 * ft + (e & 1), k & 31, c[n][e]);
            }
    }
    // bq G': eight channels per thread, then P and c
    {
        const int n = t & 15, g = t >> 4;
        float v = 0.0f;
#pragma unroll
        for (int e = 0; e < 8; ++e) v += s_bq[g * 8 + e] * s_g[(g * 8 + e) * FO_GP + n];
        s_red[g * 16 + n] = v;
    }
    __syncthreads();
    if (t < 3 * FO_N) {
        const int which = t / FO_N, n = t - which * FO_N;
        float v = 0.0f;
        if (which < 2) {
#pragma unroll
            for (int k = 0; k < 4; ++k) v += s_gp[(k * 2 + which) * FO_N + n];
        } else {
#pragma unroll
            for (int g = 0; g < 16; ++g) v += s_red[g * 16 + n];
            v += bfc ? __ldg(bfc + n0 + n) : 0.0f;
        }
        pc[((int64_t)b * 3 + which) * EN_D + n0 + n] = v;
    }
}

int encoder_fold(const float* partial, const spgt_encoder_weights& w, float* m_img, float* pc, int B, int S, const EncoderSplit& sp, cudaStream_t st) {
    static SmemOptIn configured;
    if (int e = smem_opt_in(encoder_fold_kernel, FO_SMEM, configured)) return e;
    return launch_chained(encoder_fold_kernel, B * FO_CL, FO_THREADS, FO_SMEM, st, partial, w.wq, w.bq, w.lnwk, w.lnbk, w.lnwv, w.lnbv, w.wfc, w.bfc, m_img, pc, S, sp);
}

}  // namespace spgt
