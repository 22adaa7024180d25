// C[M, N] = A^T B  for row-major A [rows, lda], B [rows, ldb] (weight gradients: dW = x^T dy), 3xTF32 on tcgen05, and the column
// sums of B (bias gradients).
//
// The reduction runs over the rows, so both operands are needed K-major with the rows as k: raw blocks of 32 rows arrive row-major
// (cp.async, padded pitch), and eight warps store them TRANSPOSED - one operand row per matrix column, 32 long - as
// hi / lo tiles, both parts rounded to nearest.  Per 8 rows one MMA A_hi x [B_hi | B_lo] and one A_lo x B_hi, the latter on top of
// the B_lo columns.
// What it replaces are fp32 products, so its error has to stay below theirs.  The accumulate step of an MMA truncates towards zero: the
// large A_hi B_hi sums have an accumulator of their own, and all are added to fp32 registers after every block of 32 rows.  Error
// relative to fp64 (normal entries, 128 x 256, against the library's fp32 product): 200 rows 1.4e-7 (2.0e-7), 1849 rows 1.4e-7 (2.8e-7),
// 65536 rows 1.8e-7 (7.7e-7); entries of one sign, 7396 rows 1.3e-7 (1.5e-7).  With sums of 128 rows and a truncated hi part it was 3.5e-7,
// 3.7e-7, 3.9e-7 and 6.6e-7, above fp32 up to about 4000 rows; the shorter sums and the rounding cost 10 % of the time (7396 rows: 16.8 ->
// 18.6 us; 65536 rows: 39 -> 45; library product and sum: 70 and 240).  Below 128 rows fp32 is closer (64 rows: 1.1e-7 against 1.3e-7).
// 65536 rows, 256 x 128: the kernel takes 47 us, 100 MB of DRAM reads, tensor pipe and shared-memory data pipe 30 % busy each, 2.3
// instructions per cycle: paced by the transposing warps and the hand-offs.
// Blocks split the rows; their partial results are added by a second kernel in an order fixed by their number: deterministic.
//   warps 0-1 raw loaders (A, B), 2 MMA issuer, 4-11 transposers (A: 4-7, B: 8-11), 12-19 accumulation.
// Every wait is a bounded mbarrier poll that records a code on expiry.
#include "tc_common.cuh"

namespace spgt {

__device__ int g_tn_status = 0;

constexpr int TN_T = 128, TN_ROWS = 32, TN_THREADS = 640;
constexpr int TN_RAW_PITCH = TN_T + 4, TN_RAW = TN_ROWS * TN_RAW_PITCH * 4, TN_NR = 2, TN_NS = 2;
constexpr int TN_HALF = TN_T * 128, TN_STAGE = 4 * TN_HALF;              // A_hi | A_lo | B_hi | B_lo
constexpr int TN_OFF_RAW = TN_NS * TN_STAGE, TN_OFF_BAR = TN_OFF_RAW + TN_NR * 2 * TN_RAW;
constexpr size_t TN_SMEM = TN_OFF_BAR + 256;
static_assert(TN_SMEM <= 227 * 1024, "shared memory budget");

struct TnParams {
    const float *a, *b;
    float *partial, *colsum;            // [split][tile][128][128]; [split][128-column tile of the summed matrix][128], or NULL
    int lda, ldb, M, N, rows, nt, sum_a;
};

__global__ void __launch_bounds__(TN_THREADS, 1) tn_gemm_kernel(const TnParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t smem_base = smem_u32(smem);
    if (smem_base & 1023u) {
        if (threadIdx.x == 0) atomicCAS(&g_tn_status, 0, 90);
        return;
    }
    const uint32_t bars = smem_base + TN_OFF_BAR;
    auto raw_full = [&](uint32_t s) { return bars + 8u * s; };            // [2]
    auto raw_empty = [&](uint32_t s) { return bars + 8u * (2 + s); };     // [2]
    auto st_full = [&](uint32_t s) { return bars + 8u * (6 + s); };       // [2]
    auto st_empty = [&](uint32_t s) { return bars + 8u * (8 + s); };      // [2]
    auto acc_full = [&](uint32_t s) { return bars + 8u * (10 + s); };     // [2]
    auto acc_empty = [&](uint32_t s) { return bars + 8u * (12 + s); };    // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + TN_OFF_BAR + 224);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + TN_OFF_BAR + 232);
    const int tid = threadIdx.x, warp = (int)tc_uniform(tid >> 5), lane = tid & 31;
    const int tile = blockIdx.y, m0 = tile / p.nt * TN_T, n0 = tile % p.nt * TN_T;
    const int blocks = (p.rows + TN_ROWS - 1) / TN_ROWS;
    const int k_begin = (int)((int64_t)blockIdx.x * blocks / gridDim.x), n_my = (int)((int64_t)(blockIdx.x + 1) * blocks / gridDim.x) - k_begin;
    if (tid == 0) {
        for (int s = 0; s < TN_NR; ++s) { mbar_init(raw_full(s), 64); mbar_init(raw_empty(s), 256); }
        for (int s = 0; s < 2; ++s) { mbar_init(st_full(s), 256); mbar_init(st_empty(s), 1); mbar_init(acc_full(s), 1); mbar_init(acc_empty(s), 256); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tc_uniform(*tmem_slot);

    if (warp < 2) {
        // ------------------------------------------ raw loaders: a row per instruction ------------------------------------------
        const float* src = warp ? p.b + n0 : p.a + m0;
        const int ld = warp ? p.ldb : p.lda, left = (warp ? p.N - n0 : p.M - m0) - lane * 4;
        const int bytes = left >= 4 ? 16 : (left > 0 ? left * 4 : 0);
        uint32_t s = 0, ph = 0;
        for (int k = 0; k < n_my; ++k) {
            if (!mbar_wait(raw_empty(s), ph ^ 1u, abort_flag, 91, &g_tn_status)) break;
            const int row0 = (k_begin + k) * TN_ROWS;
            const uint32_t dst = smem_base + TN_OFF_RAW + (2 * s + warp) * TN_RAW + lane * 16;
#pragma unroll 16
            for (int r = 0; r < TN_ROWS; ++r) {
                const bool ok = row0 + r < p.rows && bytes > 0;
                const float* from = ok ? src + (int64_t)(row0 + r) * ld + lane * 4 : p.a;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + r * (TN_RAW_PITCH * 4)), "l"(from), "r"(ok ? bytes : 0) : "memory");
            }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(raw_full(s)) : "memory");
            if (++s == TN_NR) { s = 0; ph ^= 1u; }
        }
        cp_async_wait_all();
    } else if (warp == 2) {
        // ------------------------------------------ MMA issuer ------------------------------------------
        if (tc_elect()) {
            constexpr uint32_t idesc2 = tc_idesc(2 * TN_T), idesc1 = tc_idesc(TN_T);
            uint32_t s = 0, ph = 0;
            for (int k = 0; k < n_my; ++k) {
                const uint32_t buf = (uint32_t)(k & 1), d = tmem_base + buf * 256;
                if (!mbar_wait(acc_empty(buf), (uint32_t)((k >> 1) & 1) ^ 1u, abort_flag, 92, &g_tn_status)) break;
                if (!mbar_wait(st_full(s), ph, abort_flag, 93, &g_tn_status)) break;
                tc_fence_after();
                const uint32_t st = smem_base + s * TN_STAGE;
                const uint64_t ah = tc_smem_desc(st), al = tc_smem_desc(st + TN_HALF), b = tc_smem_desc(st + 2 * TN_HALF);
#pragma unroll
                for (int k8 = 0; k8 < 4; ++k8) {
                    tc_mma_tf32_ss(d, ah + k8 * 2, b + k8 * 2, idesc2, k8 > 0 ? 1u : 0u);
                    tc_mma_tf32_ss(d + TN_T, al + k8 * 2, b + k8 * 2, idesc1, 1u);
                }
                tc_commit(st_empty(s));
                tc_commit(acc_full(buf));
                if (++s == TN_NS) { s = 0; ph ^= 1u; }
            }
        }
        __syncwarp();
    } else if (warp >= 4 && warp < 12) {
        // ------------------------------------------ transposers ------------------------------------------
        // lane = row of the block; warp w of four takes columns 32 w .. + 31 of its matrix
        const int isb = (warp - 4) >> 2, c0 = (warp & 3) * 32;
        uint32_t coff[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) coff[j] = (uint32_t)(j * 128 + (((lane >> 2) ^ j) << 4) + (lane & 3) * 4);
        float sums[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) sums[j] = 0.0f;
        uint32_t rs = 0, rph = 0, s = 0, ph = 0;
        bool alive = true;
        for (int k = 0; k < n_my; ++k) {
            if (!mbar_wait(raw_full(rs), rph, abort_flag, 94, &g_tn_status)) { alive = false; break; }
            const float4* src = reinterpret_cast<const float4*>(smem + TN_OFF_RAW + (2 * rs + isb) * TN_RAW + lane * (TN_RAW_PITCH * 4) + c0 * 4);
            float4 v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = src[j];
            mbar_arrive(raw_empty(rs));
            if (++rs == TN_NR) { rs = 0; rph ^= 1u; }
            if (!mbar_wait(st_empty(s), ph ^ 1u, abort_flag, 95, &g_tn_status)) { alive = false; break; }
            uint8_t* dst = smem + s * TN_STAGE + isb * 2 * TN_HALF + (c0 >> 3) * 1024;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float e[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
                uint32_t h[4];
                float l[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) { h[i] = tf32_rna_cvt(e[i]); l[i] = e[i] - __uint_as_float(h[i]); }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int c = 4 * j + i;
                    *reinterpret_cast<uint32_t*>(dst + (c >> 3) * 1024 + coff[c & 7]) = h[i];
                    *reinterpret_cast<uint32_t*>(dst + TN_HALF + (c >> 3) * 1024 + coff[c & 7]) = __float_as_uint(l[i]) + 0x1000u;
                    sums[c] += e[i];
                }
            }
            fence_proxy_async();
            mbar_arrive(st_full(s));
            if (++s == TN_NS) { s = 0; ph ^= 1u; }
        }
        // column sums of A or B: lanes (rows) together, by the blocks of the other matrix's first tile
        if (alive && isb != p.sum_a && p.colsum != nullptr && (p.sum_a ? n0 : m0) == 0) {
            float mine = 0.0f;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                float t = sums[j];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (lane == j) mine = t;
            }
            const int ct = p.sum_a ? gridDim.y / p.nt : p.nt, ci = p.sum_a ? tile / p.nt : tile % p.nt;
            p.colsum[((int64_t)blockIdx.x * ct + ci) * TN_T + c0 + lane] = mine;
        }
    } else if (warp >= 12) {
        // ------------------------------------------ accumulation ------------------------------------------
        const int q = warp & 3, half = (warp - 12) >> 2;                  // columns 64 half .. + 63 of this lane's row
        const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
        float acc[64];
#pragma unroll
        for (int j = 0; j < 64; ++j) acc[j] = 0.0f;
        bool alive = true;
        for (int k = 0; k < n_my; ++k) {
            const uint32_t buf = (uint32_t)(k & 1);
            if (!mbar_wait(acc_full(buf), (uint32_t)((k >> 1) & 1), abort_flag, 96, &g_tn_status)) { alive = false; break; }
            tc_fence_after();
#pragma unroll
            for (int j = 0; j < 64; j += 16) {
                float v[16];
                tc_ld16_sum(tmem_base + lane_addr + buf * 256 + half * 64 + j, TN_T, v);
#pragma unroll
                for (int e = 0; e < 16; ++e) acc[j + e] += v[e];
            }
            tc_fence_before();
            mbar_arrive(acc_empty(buf));
        }
        if (alive) {
            float* out = p.partial + (((int64_t)blockIdx.x * gridDim.y + tile) * TN_T + q * 32 + lane) * TN_T + half * 64;
#pragma unroll
            for (int j = 0; j < 16; ++j) reinterpret_cast<float4*>(out)[j] = make_float4(acc[4 * j], acc[4 * j + 1], acc[4 * j + 2], acc[4 * j + 3]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 2) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

// C and the column sums from the partial results.  Eight threads share a result (four columns of a row, or a column sum): thread g adds
// partial results g, g + 8, ..., and the eight sums are added in order: one thread per result left 16 blocks with 148 serial loads
// (128 x 128, 65536 rows: 16 us, now 5.5).
__global__ void __launch_bounds__(256)
tn_reduce_kernel(const float* __restrict__ partial, const float* __restrict__ colpart, float* __restrict__ C, float* __restrict__ colsum, int ldc,
                 int64_t panel, int M, int N, int tiles, int nt, int splits, int sums, int sum_tiles) {
    __shared__ float4 part[8][32];
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, c_blocks = tiles * (TN_T * TN_T / 4 / 32);
    if ((int)blockIdx.x < c_blocks) {
        const int i = blockIdx.x * 32 + lane;               // element of the padded [tiles][128][128 / 4]
        const float4* src = reinterpret_cast<const float4*>(partial) + i;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int k = g; k < splits; k += 8) {
            const float4 v = __ldg(src + (int64_t)k * tiles * (TN_T * TN_T / 4));
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        part[g][lane] = s;
        __syncthreads();
        if (g) return;
#pragma unroll
        for (int k = 1; k < 8; ++k) { const float4 v = part[k][lane]; s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w; }
        const int c4 = i % (TN_T / 4), r = i / (TN_T / 4) % TN_T, tile = i / (TN_T * TN_T / 4);
        const int row = tile / nt * TN_T + r, col = tile % nt * TN_T + c4 * 4;
        if (row < M) {
            const float o[4] = {s.x, s.y, s.z, s.w};
            float* dst = C + tile % nt * panel + (int64_t)row * ldc + c4 * 4;
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (col + e < N) dst[e] = o[e];
        }
    } else {
        const int c = (blockIdx.x - c_blocks) * 32 + lane;   // (colpart has whole 128-column tiles)
        float s = 0.0f;
        if (c < sums)
#pragma unroll 8
            for (int k = g; k < splits; k += 8) s += __ldg(colpart + ((int64_t)k * sum_tiles) * TN_T + c);
        part[g][lane].x = s;
        __syncthreads();
        if (g || c >= sums) return;
#pragma unroll
        for (int k = 1; k < 8; ++k) s += part[k][lane].x;
        colsum[c] = s;
    }
}

int tn_status(bool reset) {
    int v = 0;
    if (reset) return cudaMemcpyToSymbol(g_tn_status, &v, sizeof(int)) == cudaSuccess ? SPGT_OK : SPGT_ERR_LAUNCH;
    return cudaMemcpyFromSymbol(&v, g_tn_status, sizeof(int)) == cudaSuccess ? v : SPGT_ERR_LAUNCH;
}

// Blocks that share the rows: one wave over the SMs, at least eight row blocks each (below that the partial results cost more)
static int tn_splits(int M, int N, int rows) {
    const int tiles = ceil_div(M, TN_T) * ceil_div(N, TN_T), most = num_sms() / tiles < 1 ? 1 : num_sms() / tiles, want = ceil_div(rows, TN_ROWS * 8);
    return want < most ? want : most;
}

}  // namespace spgt

using namespace spgt;

extern "C" size_t spgt_tn_gemm_workspace_bytes(int M, int N, int rows) {
    if (M <= 0 || N <= 0 || rows <= 0 || M > 4096 || N > 4096) return 0;
    const size_t mt = ceil_div(M, TN_T), nt = ceil_div(N, TN_T), splits = (size_t)tn_splits(M, N, rows);
    return splits * (mt * nt * TN_T * TN_T + (mt > nt ? mt : nt) * TN_T) * sizeof(float);
}

namespace spgt {
// sum_a: the column sums are A's [M], not B's [N].  panel: distance between the 128-column panels of C (128: side by side).
int tn_gemm(const float* A, int lda, const float* B, int ldb, float* C, int ldc, int64_t panel, float* colsum, bool sum_a, int M, int N, int rows,
            void* workspace, size_t workspace_bytes, cudaStream_t st) {
    if (!A || !B || !C || !workspace) return SPGT_ERR_NULL;
    const size_t need = spgt_tn_gemm_workspace_bytes(M, N, rows);
    if (need == 0 || (lda & 3) || (ldb & 3)) return SPGT_ERR_SHAPE;
    if (workspace_bytes < need) return SPGT_ERR_WORKSPACE;
    if (!aligned16(A) || !aligned16(B) || !aligned16(workspace)) return SPGT_ERR_ALIGN;
    static SmemOptIn configured;
    if (int e = smem_opt_in(tn_gemm_kernel, TN_SMEM, configured)) return e;
    const int nt = ceil_div(N, TN_T), mt = ceil_div(M, TN_T), tiles = mt * nt, splits = tn_splits(M, N, rows);
    float* partial = (float*)workspace;
    float* colpart = partial + (size_t)splits * tiles * TN_T * TN_T;
    const TnParams p{A, B, partial, colsum ? colpart : nullptr, lda, ldb, M, N, rows, nt, sum_a ? 1 : 0};
    tn_gemm_kernel<<<dim3((unsigned)splits, (unsigned)tiles), TN_THREADS, TN_SMEM, st>>>(p);
    if (int e = launch_status()) return e;
    const int sums = colsum ? (sum_a ? M : N) : 0;
    tn_reduce_kernel<<<tiles * (TN_T * TN_T / 4 / 32) + ceil_div(sums, 32), 256, 0, st>>>(partial, colpart, C, colsum, ldc, panel, M, N, tiles, nt,
                                                                                        splits, sums, sum_a ? mt : nt);
    return launch_status();
}
}  // namespace spgt

extern "C" int spgt_tn_gemm(const float* A, int lda, const float* B, int ldb, float* C, int ldc, float* colsum, int M, int N, int rows,
                            void* workspace, size_t workspace_bytes, spgt_stream_t stream) {
    if (A && B && C && workspace && (lda < M || ldb < N || ldc < N)) return SPGT_ERR_SHAPE;
    return tn_gemm(A, lda, B, ldb, C, ldc, TN_T, colsum, false, M, N, rows, workspace, workspace_bytes, (cudaStream_t)stream);
}
