// Backward of the Galerkin attention op  out[s][j] = sum_i Q[i][s] T[i][j],  T[i][j] = (1/S) sum_s K[i][s] V[j][s]
// (reference: multihead_galerkin_attention_cccr_backward, extension/bind/galerkin_attention.cu:126-173, which runs
// three split-K and three small-K SGEMMs).  Exact fp32 FMA arithmetic:
//   reduce  T and  dT[i][j] = sum_s Q[i][s] dOut[s][j]:  a block streams a chunk of the S columns of one (batch, head) through
//           shared memory; a thread owns 6 x 6 entries and a seventh of the columns of every tile;
//   sum     chunk partials in chunk order (deterministic);
//   apply   up to four grid nodes per thread:  dQ[i][s] = sum_j T[i][j] dOut[s][j],   dK[i][s] = (1/S) sum_j dT[i][j] V[j][s],
//           dV[j][s] = (1/S) sum_i dT[i][j] K[i][s].
// Both are bound by the values shared memory hands to registers (128 bytes per cycle and SM): with 6 x 6 entries twelve 16-byte
// reads feed 144 FMAs, with four nodes nine feed 144.  Batch 16, 4 heads, S = 4096: 540 us with five single entries and one
// node per thread.
// Layouts as in the forward: Q, K, V, dQ, dK, dV [B*H, dpk, S] (S fastest), dOut [B*H, S, dpk] or, merged heads, [B, S, H * dpk].
#include <type_traits>
#include "common.cuh"

namespace spgt {

constexpr int AB_MAXD = 35, AB_TP = 36;        // dpk <= 35; pitch of the dpk x dpk matrices
constexpr int AB_MAT = AB_TP * AB_TP;
constexpr int AB_GROUPS = 7, AB_COLS = AB_GROUPS * 16, AB_CP = AB_COLS + 4;      // columns per tile, pitch (an odd number of 16-byte units)
constexpr int AB_THREADS = 256;                // 7 groups x 36 threads work, all load

// Rows of dOut: pitch ld, rows of (batch, head) bh start at `at(bh)`.
struct AbOut {
    int ld, H, D, S;                           // merged heads: H > 0, ld = H * D
    __device__ __forceinline__ int64_t at(int64_t bh) const {
        return H > 0 ? bh / H * S * ld + bh % H * D : bh * (int64_t)D * S;
    }
};

// partial [bh][which: T, dT][chunk][36][36].  The next tile's copies are in flight while a tile is multiplied, two blocks per SM: with
// plain loads between two barriers and one block per SM the kernel waited for memory (batch 16, 4 heads, S = 4096: 302 us, now 70 us).
// VEC: rows of Q, K, V in 16-byte copies (S a multiple of four, aligned bases), else 4-byte ones; dOut, whose rows are nodes, is
// transposed by 4-byte copies.  magic = 2^20 / D + 1: i / D = i * magic >> 20 for i < 2^12.
// NA: entries a thread owns along each side, the whole 36 x 36 with 6; fewer where D <= 6 NA.
constexpr int AB_STAGE = 2 * AB_TP * AB_CP;
template <bool VEC, int NA>
__global__ void __launch_bounds__(AB_THREADS, 2)
attn_bwd_reduce_kernel(const float* __restrict__ Q, const float* __restrict__ K, const float* __restrict__ V, const float* __restrict__ dOut,
                       float* __restrict__ partial, int D, int S, int chunks, uint32_t magic, AbOut od) {
    extern __shared__ __align__(16) float smem[];          // two stages of A rows, B rows
    const int t = threadIdx.x, chunk = blockIdx.x % chunks, which = blockIdx.y;
    const int64_t bh = blockIdx.x / chunks, base = bh * (int64_t)D * S;
    const int tiles = (S + AB_COLS - 1) / AB_COLS;
    const int t_begin = (int)(((int64_t)chunk * tiles) / chunks), t_end = (int)(((int64_t)(chunk + 1) * tiles) / chunks);
    const float* A = (which ? Q : K) + base;
    const float* B = which ? dOut + od.at(bh) : V + base;
    const int g = t / 36, tt = t - g * 36, i0 = tt / 6, j0 = tt - i0 * 6;          // entries (i0 + 6 a, j0 + 6 b), a, b < NA
    // groups that have columns, in any tile of this block: a single short tile leaves the others nothing to add up
    const int cols = t_end - t_begin > 1 || S - t_begin * AB_COLS >= AB_COLS ? AB_COLS : (S - t_begin * AB_COLS + 15) / 16 * 16, groups = cols / 16;
    for (int i = t; i < (AB_TP - D) * AB_CP; i += AB_THREADS)
#pragma unroll
        for (int k = 0; k < 4; ++k) smem[k * AB_TP * AB_CP + D * AB_CP + i] = 0.0f;
    auto copy_rows = [&](const float* src, float* dst, int s0, int ns) {
        if constexpr (VEC) {
            for (int i = t; i < D * (AB_COLS / 4); i += AB_THREADS) {
                const int r = i / (AB_COLS / 4), c = (i - r * (AB_COLS / 4)) * 4;
                if (c >= cols) continue;
                cp_async_zfill<16>(dst + r * AB_CP + c, c < ns ? src + (int64_t)r * S + s0 + c : src, c < ns);
            }
        } else {
            for (int i = t; i < D * AB_COLS; i += AB_THREADS) {
                const int r = i / AB_COLS, c = i - r * AB_COLS;
                if (c >= cols) continue;
                cp_async_zfill<4>(dst + r * AB_CP + c, c < ns ? src + (int64_t)r * S + s0 + c : src, c < ns);
            }
        }
    };
    auto load = [&](int tile, int stage) {
        const int s0 = tile * AB_COLS, ns = S - s0 < AB_COLS ? S - s0 : AB_COLS;
        float *as = smem + stage * AB_STAGE, *bs = as + AB_TP * AB_CP;
        copy_rows(A, as, s0, ns);
        if (!which) copy_rows(B, bs, s0, ns);
        else
            for (int i = t; i < D * cols; i += AB_THREADS) {
                const int c = (int)(((uint32_t)i * magic) >> 20), j = i - c * D;
                cp_async_zfill<4>(bs + j * AB_CP + c, c < ns ? B + (int64_t)(s0 + c) * od.ld + j : B, c < ns);
            }
        cp_async_commit();
    };
    float acc[NA][NA] = {};
    load(t_begin, 0);
    for (int tile = t_begin; tile < t_end; ++tile) {
        const int stage = (tile - t_begin) & 1;
        if (tile + 1 < t_end) { load(tile + 1, stage ^ 1); cp_async_wait<1>(); } else cp_async_wait<0>();
        __syncthreads();
        if (g < groups) {
            const float* pa = smem + stage * AB_STAGE + i0 * AB_CP + g * 16;
            const float* pb = smem + stage * AB_STAGE + (AB_TP + j0) * AB_CP + g * 16;
#pragma unroll
            for (int s = 0; s < 16; s += 4) {
                float4 b[NA];
#pragma unroll
                for (int e = 0; e < NA; ++e) b[e] = *reinterpret_cast<const float4*>(pb + 6 * e * AB_CP + s);
#pragma unroll
                for (int e = 0; e < NA; ++e) {
                    const float4 a = *reinterpret_cast<const float4*>(pa + 6 * e * AB_CP + s);
#pragma unroll
                    for (int f = 0; f < NA; ++f) {
                        acc[e][f] = fmaf(a.x, b[f].x, acc[e][f]); acc[e][f] = fmaf(a.y, b[f].y, acc[e][f]);
                        acc[e][f] = fmaf(a.z, b[f].z, acc[e][f]); acc[e][f] = fmaf(a.w, b[f].w, acc[e][f]);
                    }
                }
            }
        }
        __syncthreads();
    }
    // the column groups, in order
    float* out = partial + ((bh * 2 + which) * chunks + chunk) * AB_MAT;
    float* red = smem;
    for (int k = 0; k < groups; ++k) {
        __syncthreads();
        if (g == k)
#pragma unroll
            for (int e = 0; e < NA; ++e)
#pragma unroll
                for (int f = 0; f < NA; ++f) {
                    const int at = (i0 + 6 * e) * AB_TP + j0 + 6 * f;
                    red[at] = k == 0 ? acc[e][f] : red[at] + acc[e][f];
                }
    }
    __syncthreads();
    for (int i = t; i < AB_MAT; i += AB_THREADS) out[i] = NA == 6 || (i / AB_TP < 6 * NA && i % AB_TP < 6 * NA) ? red[i] : 0.0f;
}

// sums [bh][T | dT | dT transposed][36][36]: chunk partials in chunk order, 1 / S included
__global__ void __launch_bounds__(256)
attn_bwd_sum_kernel(const float* __restrict__ partial, float* __restrict__ sums, int chunks, float inv_s) {
    const int64_t bh = blockIdx.x;
    const int which = blockIdx.y;
    const float* src = partial + (bh * 2 + which) * chunks * AB_MAT;
    float* dst = sums + bh * 3 * AB_MAT;
    for (int i = threadIdx.x; i < AB_MAT; i += blockDim.x) {
        float s = 0.0f;
#pragma unroll 8
        for (int k = 0; k < chunks; ++k) s += __ldg(src + (int64_t)k * AB_MAT + i);
        s *= inv_s;
        if (which == 0) dst[i] = s;
        else { dst[AB_MAT + i] = s; dst[2 * AB_MAT + (i % AB_TP) * AB_TP + i / AB_TP] = s; }
    }
}

constexpr int AP_THREADS = 128;

// JQ: quads of channels, 9 for any D <= 36
template <int AP_NODES, int JQ>
__global__ void __launch_bounds__(AP_THREADS, 3)
attn_bwd_apply_kernel(const float* __restrict__ K, const float* __restrict__ V, const float* __restrict__ dOut, const float* __restrict__ sums,
                      float* __restrict__ dQ, float* __restrict__ dK, float* __restrict__ dV, int D, int S, int col_tiles, AbOut od) {
    __shared__ __align__(16) float mats[3 * AB_MAT];       // T | dT | dT transposed
    const int t = threadIdx.x;
    const int64_t bh = blockIdx.x / col_tiles, base = bh * (int64_t)D * S;
    const int s0 = (int)(blockIdx.x % col_tiles) * (AP_THREADS * AP_NODES) + t;
    for (int i = t; i < 3 * AB_MAT / 4; i += AP_THREADS)
        reinterpret_cast<float4*>(mats)[i] = __ldg(reinterpret_cast<const float4*>(sums + bh * 3 * AB_MAT) + i);
    __syncthreads();
    float x[4 * JQ][AP_NODES];
    auto multiply = [&](const float* m, float* dst) {      // dst[i][s] = sum_j m[i][j] x[j]
#pragma unroll 1
        for (int i = 0; i < D; ++i) {
            const float4* row = reinterpret_cast<const float4*>(m + i * AB_TP);
            float acc[AP_NODES] = {};
#pragma unroll
            for (int j = 0; j < JQ; ++j) {
                const float4 w = row[j];
#pragma unroll
                for (int n = 0; n < AP_NODES; ++n) {
                    acc[n] = fmaf(w.x, x[4 * j][n], acc[n]); acc[n] = fmaf(w.y, x[4 * j + 1][n], acc[n]);
                    acc[n] = fmaf(w.z, x[4 * j + 2][n], acc[n]); acc[n] = fmaf(w.w, x[4 * j + 3][n], acc[n]);
                }
            }
#pragma unroll
            for (int n = 0; n < AP_NODES; ++n)
                if (s0 + n * AP_THREADS < S) dst[base + (int64_t)i * S + s0 + n * AP_THREADS] = acc[n];
        }
    };
    auto load_columns = [&](const float* src) {
#pragma unroll
        for (int j = 0; j < 4 * JQ; ++j)
#pragma unroll
            for (int n = 0; n < AP_NODES; ++n)
                x[j][n] = j < D && s0 + n * AP_THREADS < S ? __ldg(src + base + (int64_t)j * S + s0 + n * AP_THREADS) : 0.0f;
    };
    load_columns(V);
    multiply(mats + AB_MAT, dK);
    load_columns(K);
    multiply(mats + 2 * AB_MAT, dV);
    const float* rows = dOut + od.at(bh);
#pragma unroll
    for (int n = 0; n < AP_NODES; ++n)
#pragma unroll
        for (int j = 0; j < 4 * JQ; ++j)
            x[j][n] = j < D && s0 + n * AP_THREADS < S ? __ldg(rows + (int64_t)(s0 + n * AP_THREADS) * od.ld + j) : 0.0f;
    multiply(mats, dQ);
}

// blocks per (batch, head) and matrix: four waves of two per SM, one tile each at least
static int attn_bwd_chunks(int64_t BH, int S) {
    const int tiles = ceil_div(S, AB_COLS);
    int64_t c = (int64_t)8 * num_sms() / (2 * BH);
    if (c > tiles) c = tiles;
    return (int)(c < 1 ? 1 : c);
}

}  // namespace spgt

using namespace spgt;

extern "C" size_t spgt_galerkin_attn_bwd_workspace_bytes(int B, int H, int dpk, int S) {
    if (B <= 0 || H <= 0 || S <= 0 || dpk <= 0 || dpk > AB_MAXD) return 0;
    const int64_t BH = (int64_t)B * H;
    return (size_t)BH * (2 * attn_bwd_chunks(BH, S) + 3) * AB_MAT * sizeof(float);
}

namespace spgt {
// merged: d_out is [B, S, H * dpk], as the output projection takes it
int galerkin_attn_bwd(const float* Q, const float* K, const float* V, const float* d_out, float* dQ, float* dK, float* dV, int B, int H, int dpk,
                      int S, bool merged, void* workspace, size_t workspace_bytes, cudaStream_t st) {
    if (!Q || !K || !V || !d_out || !dQ || !dK || !dV) return SPGT_ERR_NULL;
    if (B <= 0 || H <= 0 || S <= 0 || dpk <= 0 || dpk > AB_MAXD) return SPGT_ERR_SHAPE;
    const int64_t BH = (int64_t)B * H;
    // four nodes per thread where that still makes a block per SM (small problems are bound by the length of one thread's work) and where
    // there are nodes for them: 1024 x 4 heads of 16 nodes took 659 us with four, three of them past the end, and all seven column
    // groups added up; now 231 (495 before)
    const int chunks = attn_bwd_chunks(BH, S);
    int nodes = 4;
    while (nodes > 1 && (BH * ceil_div(S, AP_THREADS * nodes) < num_sms() || S <= AP_THREADS * nodes / 2)) nodes >>= 1;
    const int col_tiles = ceil_div(S, AP_THREADS * nodes);
    if (BH * chunks > 0x7fffffffLL || BH * col_tiles > 0x7fffffffLL) return SPGT_ERR_SHAPE;
    if (!workspace || workspace_bytes < spgt_galerkin_attn_bwd_workspace_bytes(B, H, dpk, S)) return SPGT_ERR_WORKSPACE;
    const AbOut od{merged ? H * dpk : dpk, merged ? H : 0, dpk, S};
    float* partial = (float*)workspace;
    float* sums = partial + BH * 2 * chunks * AB_MAT;
    const bool vec = (S & 3) == 0 && aligned16(Q) && aligned16(K) && aligned16(V);
    const size_t smem = (size_t)2 * AB_STAGE * sizeof(float);
    const float inv_s = 1.0f / (float)S;
    // Narrow heads (the model's have 34 rows) leave most of the 36 x 36 entries empty: 2 x 4 heads of 8 rows, 4096 nodes took 40 us with all of
    // them, now 32 (16 for a kernel that looped over the rows there are); 16 x 4 of 16 rows: 127 and 86 (124).
    auto run = [&](auto na_, auto jq_) {
        constexpr int NA = decltype(na_)::value, JQ = decltype(jq_)::value;
        static SmemOptIn opt_v, opt_s;
        if (int e = vec ? smem_opt_in(attn_bwd_reduce_kernel<true, NA>, smem, opt_v) : smem_opt_in(attn_bwd_reduce_kernel<false, NA>, smem, opt_s)) return e;
        auto reduce = vec ? attn_bwd_reduce_kernel<true, NA> : attn_bwd_reduce_kernel<false, NA>;
        reduce<<<dim3((unsigned)(BH * chunks), 2), AB_THREADS, smem, st>>>(Q, K, V, d_out, partial, dpk, S, chunks, (1u << 20) / (uint32_t)dpk + 1, od);
        if (int e = launch_status()) return e;
        attn_bwd_sum_kernel<<<dim3((unsigned)BH, 2), 256, 0, st>>>(partial, sums, chunks, inv_s);
        if (int e = launch_status()) return e;
        auto apply = nodes == 4 ? attn_bwd_apply_kernel<4, JQ> : nodes == 2 ? attn_bwd_apply_kernel<2, JQ> : attn_bwd_apply_kernel<1, JQ>;
        apply<<<(unsigned)(BH * col_tiles), AP_THREADS, 0, st>>>(K, V, d_out, sums, dQ, dK, dV, dpk, S, col_tiles, od);
        return launch_status();
    };
    using std::integral_constant;
    if (dpk <= 12) return run(integral_constant<int, 2>{}, integral_constant<int, 3>{});
    if (dpk <= 24) return run(integral_constant<int, 4>{}, integral_constant<int, 6>{});
    return run(integral_constant<int, 6>{}, integral_constant<int, 9>{});
}
}  // namespace spgt

extern "C" int spgt_galerkin_attn_bwd(const float* Q, const float* K, const float* V, const float* d_out, float* dQ, float* dK,
                                      float* dV, int B, int H, int dpk, int S, void* workspace, size_t workspace_bytes,
                                      spgt_stream_t stream) {
    return galerkin_attn_bwd(Q, K, V, d_out, dQ, dK, dV, B, H, dpk, S, false, workspace, workspace_bytes, (cudaStream_t)stream);
}
