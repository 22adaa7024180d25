// Second half of an encoder layer (see encoder_common.cuh), one kernel:
//   y = [x +] x M + pos P + c,      out = y + act(y W1 + b1) W2 + b2          (FFN = false: out = y, the attention layer alone)
// with M, P, c of the tile's sample.  Three chained GEMMs on one 128-row tile (3xTF32); x, y and out share one row-major tile in
// shared memory, every A operand passes through two tensor-memory stages of 32 columns hi | lo, the 256 hidden
// activations never leave tensor memory.
//   GEMM 0  A = x (split by warps 0-3), B = M image,            D0 128 columns
//   GEMM 1  A = y (D0 + x + pos P + c, warps 4-11),             D1 256 columns
//   GEMM 2  A = act(D1 + b1) (warps 4-11),                      D2 128 columns, in D0's place
// D0 / D2 and D1 swap sides from tile to tile, so that GEMM 0 of the next tile and the last epilogue do not wait for one another.
// The B operands stream through a ring of 16 KB slots (an image's hi or lo half): 640 KB per tile from L2, 42 B per cycle and SM
// (measured: L2 delivers at least 79).  The tensor pipe needs 15400 cycles per tile (240 MMAs of 64); measured on its own, 64 x 2809 nodes:
// 144 us = 21700 cycles for each of at most ten tiles per SM, the pipe 67 % busy: the conversions between the chained GEMMs are in the way.
//   warps 0-3 x splitters, 4-11 converters / epilogue, 12 x tile loader, 13-14 image loaders (even / odd slots), 15 MMA issuer.
// Every wait is a bounded mbarrier poll that records a code on expiry.
#include "encoder_common.cuh"

namespace spgt {

__device__ int g_enc_out_status = 0;

constexpr int EO_THREADS = 512, EO_NW = 5, EO_SLOT = 16384, EO_PITCH = 132, EO_XT = EN_ROWS * EO_PITCH * 4, EO_PC = 3 * EN_D * 4;
constexpr int EO_OFF_X = EO_NW * EO_SLOT, EO_OFF_PC = EO_OFF_X + 2 * EO_XT, EO_OFF_CONST = EO_OFF_PC + 2 * EO_PC;
constexpr int EO_OFF_BAR = EO_OFF_CONST + (256 + 128) * 4;
constexpr size_t EO_SMEM = EO_OFF_BAR + 256;
static_assert(EO_SMEM <= 227 * 1024, "shared memory budget");
constexpr uint32_t EO_A = 384;

struct EncoderOutParams {
    const float *x, *m_img, *pc, *pos, *w1, *b1, *w2, *b2;
    float* y;
    int S, tps, n_tiles, act, residual;
};

template <bool FFN>
__global__ void __launch_bounds__(EO_THREADS, 1) encoder_out_kernel(const EncoderOutParams p) {
    constexpr int USES = FFN ? 16 : 4, SLOTS = FFN ? 40 : 8;            // A-stage uses and image slots per tile
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t smem_base = smem_u32(smem);
    if (smem_base & 1023u) {
        if (threadIdx.x == 0) atomicCAS(&g_enc_out_status, 0, 60);
        return;
    }
    float* consts = reinterpret_cast<float*>(smem + EO_OFF_CONST);      // b1 [256] | b2 [128]
    const uint32_t bars = smem_base + EO_OFF_BAR;
    auto a_full = [&](uint32_t s) { return bars + 8u * s; };            // [2]
    auto a_empty = [&](uint32_t s) { return bars + 8u * (2 + s); };     // [2]
    auto x_full = [&](uint32_t s) { return bars + 8u * (4 + s); };      // [2]
    auto x_empty = [&](uint32_t s) { return bars + 8u * (6 + s); };     // [2]
    auto d_free = [&](uint32_t s) { return bars + 8u * (8 + s); };      // [2] the last accumulator of a tile (by tile parity) has been read
    const uint32_t d0_full = bars + 8u * 10, d1_full = bars + 8u * 11, d2_full = bars + 8u * 12, x_go = bars + 8u * 13;
    auto w_full = [&](uint32_t s) { return bars + 8u * (14 + s); };     // [5]
    auto w_empty = [&](uint32_t s) { return bars + 8u * (19 + s); };    // [5]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + EO_OFF_BAR + 224);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + EO_OFF_BAR + 232);

    const int tid = threadIdx.x, warp = (int)tc_uniform(tid >> 5), lane = tid & 31;
    const int n_my = ((int)blockIdx.x < p.n_tiles) ? (p.n_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    auto tile_index = [&](int ti) { return (int)blockIdx.x + ti * (int)gridDim.x; };
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(a_full(s), 128); mbar_init(a_empty(s), 1); mbar_init(x_full(s), 32); mbar_init(x_empty(s), 256); mbar_init(d_free(s), 256);
        }
        mbar_init(d0_full, 1); mbar_init(d1_full, 1); mbar_init(d2_full, 1); mbar_init(x_go, 1);
        for (int s = 0; s < EO_NW; ++s) { mbar_init(w_full(s), 1); mbar_init(w_empty(s), 1); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 15) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (FFN)
        for (int i = tid; i < 384; i += EO_THREADS) consts[i] = i < 256 ? __ldg(p.b1 + i) : (p.b2 ? __ldg(p.b2 + i - 256) : 0.0f);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tc_uniform(*tmem_slot);
    pdl_wait();
    pdl_launch_next();

    // Split 32 values of this thread's row and store them as A stage s once its previous use (the stage's `use`-th) is over.  The
    // split comes before the wait: a stage's turn-around is what paces the short k-blocks.
    auto store_a = [&](uint32_t s, uint32_t use, uint32_t lane_addr, const float (&v)[32], int code) {
        uint32_t hi[32], lo[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) split_tf32(v[j], hi[j], lo[j]);
        if (!mbar_wait(a_empty(s), ((use >> 1) & 1u) ^ 1u, abort_flag, code, &g_enc_out_status)) return false;
        tc_fence_after();
        const uint32_t a_hi = tmem_base + lane_addr + EO_A + s * 64;
        tc_st16(a_hi, reinterpret_cast<uint32_t(&)[16]>(hi[0]));
        tc_st16(a_hi + 16, reinterpret_cast<uint32_t(&)[16]>(hi[16]));
        tc_st16(a_hi + 32, reinterpret_cast<uint32_t(&)[16]>(lo[0]));
        tc_st16(a_hi + 48, reinterpret_cast<uint32_t(&)[16]>(lo[16]));
        tc_wait_st();
        tc_fence_before();
        mbar_arrive(a_full(s));
        return true;
    };

    if (warp < 4) {
        // ------------------------------------------ x splitters ------------------------------------------
        const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
        bool alive = true;
        for (int ti = 0; ti < n_my && alive; ++ti) {
            const uint32_t buf = (uint32_t)(ti & 1);
            if (!mbar_wait(x_full(buf), (uint32_t)((ti >> 1) & 1), abort_flag, 61, &g_enc_out_status)) break;
            // The A stages are shared with the other converters; after k-block 4 of the previous tile's GEMM 2 only the last use
            // of each stage may be unconsumed when its parity wait below comes, so it cannot mistake an older phase for the wanted one.
            if (FFN && ti > 0 && !mbar_wait(x_go, (uint32_t)((ti - 1) & 1), abort_flag, 62, &g_enc_out_status)) break;
            const float4* row = reinterpret_cast<const float4*>(smem + EO_OFF_X + buf * EO_XT + (warp * 32 + lane) * (EO_PITCH * 4));
            for (int kb = 0; kb < 4; ++kb) {
                const uint32_t use = (uint32_t)(ti * USES + kb), s = use & 1u;
                float v[32];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float4 w = row[kb * 8 + j];
                    v[4 * j] = w.x; v[4 * j + 1] = w.y; v[4 * j + 2] = w.z; v[4 * j + 3] = w.w;
                }
                if (!store_a(s, use, lane_addr, v, 63)) { alive = false; break; }
            }
        }
    } else if (warp < 12) {
        // ------------------------------------------ converters / epilogue ------------------------------------------
        const int q = warp & 3;
        const uint32_t g = (uint32_t)((warp - 4) >> 2);                 // group g takes the k-blocks (32 columns) of parity g, in stage g
        const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
        const int r = q * 32 + lane;
        bool alive = true;
        auto fetch_pos = [&](int ti) {                                  // position values of this row, a tile ahead
            const int tile = tile_index(ti < n_my ? ti : 0), b = tile / p.tps, row = (tile - b * p.tps) * EN_ROWS + r;
            return row < p.S ? __ldg(reinterpret_cast<const float2*>(p.pos) + (int64_t)b * p.S + row) : make_float2(0.f, 0.f);
        };
        float2 pnext = fetch_pos(0);
        for (int ti = 0; ti < n_my && alive; ++ti) {
            const uint32_t buf = (uint32_t)(ti & 1), tph = (uint32_t)(ti & 1);
            const uint32_t d0 = tmem_base + lane_addr + (buf ? 256u : 0u), d1 = tmem_base + lane_addr + (buf ? 0u : 128u);
            const int tile = tile_index(ti), b = tile / p.tps, row0 = (tile - b * p.tps) * EN_ROWS;
            const int nrows = p.S - row0;                               // (may exceed the tile)
            float* xrow = reinterpret_cast<float*>(smem + EO_OFF_X + buf * EO_XT) + r * EO_PITCH;
            const float* pc = reinterpret_cast<const float*>(smem + EO_OFF_PC + buf * EO_PC);
            const float2 ps = pnext;
            pnext = fetch_pos(ti + 1);
            // rows of this warp, 32 columns from c0: shared memory -> coalesced stores (one 128-byte line per row)
            auto store_rows = [&](int c0) {
                __syncwarp();
                const float* sp = reinterpret_cast<const float*>(smem + EO_OFF_X + buf * EO_XT) + (q * 32 + (lane >> 3)) * EO_PITCH + c0 + (lane & 7) * 4;
                float* yp = p.y + ((int64_t)b * p.S + row0 + q * 32 + (lane >> 3)) * EN_D + c0 + (lane & 7) * 4;
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (q * 32 + i * 4 + (lane >> 3) < nrows)
                        *reinterpret_cast<float4*>(yp + i * 4 * EN_D) = *reinterpret_cast<const float4*>(sp + i * 4 * EO_PITCH);
            };
            if (!mbar_wait(x_full(buf), (uint32_t)((ti >> 1) & 1), abort_flag, 64, &g_enc_out_status)) break;
            if (!mbar_wait(d0_full, tph, abort_flag, 65, &g_enc_out_status)) break;
            tc_fence_after();
#pragma unroll 1
            for (int kb = (int)g; kb < 4; kb += 2) {
                float v[32];
                tc_ld32(d0 + kb * 32, v);
                if (!FFN && kb + 2 >= 4) { tc_fence_before(); mbar_arrive(d_free(buf)); }
                float4* xr = reinterpret_cast<float4*>(xrow + kb * 32);
                const float4* p0 = reinterpret_cast<const float4*>(pc + kb * 32);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float4 a0 = p0[j], a1 = p0[32 + j], c = p0[64 + j];
                    float4 o = make_float4(v[4 * j] + (ps.x * a0.x + ps.y * a1.x + c.x), v[4 * j + 1] + (ps.x * a0.y + ps.y * a1.y + c.y),
                                           v[4 * j + 2] + (ps.x * a0.z + ps.y * a1.z + c.z), v[4 * j + 3] + (ps.x * a0.w + ps.y * a1.w + c.w));
                    if (FFN || p.residual) { const float4 xv = xr[j]; o.x += xv.x; o.y += xv.y; o.z += xv.z; o.w += xv.w; }
                    xr[j] = o;
                    v[4 * j] = o.x; v[4 * j + 1] = o.y; v[4 * j + 2] = o.z; v[4 * j + 3] = o.w;
                }
                if constexpr (FFN) {
                    const uint32_t use = (uint32_t)(ti * USES + 4 + kb);
                    if (!store_a(g, use, lane_addr, v, 66)) { alive = false; break; }
                } else {
                    store_rows(kb * 32);
                }
            }
            if (!alive) break;
            if constexpr (FFN) {
                if (!mbar_wait(d1_full, tph, abort_flag, 67, &g_enc_out_status)) break;
                tc_fence_after();
#pragma unroll 1
                for (int kb = (int)g; kb < 8; kb += 2) {
                    const uint32_t use = (uint32_t)(ti * USES + 8 + kb);
                    float v[32];
                    tc_ld32(d1 + kb * 32, v);
                    const float4* bb = reinterpret_cast<const float4*>(consts + kb * 32);
#pragma unroll
                    for (int j = 0; j < 8; ++j) { const float4 c = bb[j]; v[4 * j] += c.x; v[4 * j + 1] += c.y; v[4 * j + 2] += c.z; v[4 * j + 3] += c.w; }
                    if (p.act == SPGT_ACT_RELU) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.0f);
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = apply_act(v[j], p.act);
                    }
                    if (!store_a(g, use, lane_addr, v, 68)) { alive = false; break; }
                }
                if (!alive) break;
                if (!mbar_wait(d2_full, tph, abort_flag, 69, &g_enc_out_status)) break;
                tc_fence_after();
#pragma unroll 1
                for (int kb = (int)g; kb < 4; kb += 2) {
                    float v[32];
                    tc_ld32(d0 + kb * 32, v);
                    if (kb + 2 >= 4) { tc_fence_before(); mbar_arrive(d_free(buf)); }
                    float4* xr = reinterpret_cast<float4*>(xrow + kb * 32);
                    const float4* bb = reinterpret_cast<const float4*>(consts + 256 + kb * 32);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float4 c = bb[j];
                        float4 o = xr[j];
                        o.x += v[4 * j] + c.x; o.y += v[4 * j + 1] + c.y; o.z += v[4 * j + 2] + c.z; o.w += v[4 * j + 3] + c.w;
                        xr[j] = o;
                    }
                    store_rows(kb * 32);
                }
            }
            mbar_arrive(x_empty(buf));
        }
    } else if (warp == 12) {
        // ------------------------------------------ x tiles and pos / constant rows of the sample ------------------------------------------
        for (int ti = 0; ti < n_my; ++ti) {
            const uint32_t buf = (uint32_t)(ti & 1);
            const int tile = tile_index(ti), b = tile / p.tps, row0 = (tile - b * p.tps) * EN_ROWS;
            const int nrows = p.S - row0 < EN_ROWS ? p.S - row0 : EN_ROWS;
            if (!mbar_wait(x_empty(buf), (uint32_t)((ti >> 1) & 1) ^ 1u, abort_flag, 70, &g_enc_out_status)) break;
            // a row per instruction (bulk copies of 512-byte rows took 5000 cycles longer); rows beyond the sample are zero
            const float* src = p.x + ((int64_t)b * p.S + row0) * EN_D + lane * 4;
            const uint32_t dst = smem_base + EO_OFF_X + buf * EO_XT + lane * 16;
#pragma unroll 16
            for (int r = 0; r < EN_ROWS; ++r) {
                const bool ok = r < nrows;
                const float* from = ok ? src + (int64_t)r * EN_D : p.x;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + r * (EO_PITCH * 4)), "l"(from), "r"(ok ? 16 : 0) : "memory");
            }
            for (int i = lane; i < EO_PC / 16; i += 32)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_base + EO_OFF_PC + buf * EO_PC + i * 16), "l"(p.pc + (int64_t)b * 3 * EN_D + i * 4) : "memory");
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(x_full(buf)) : "memory");
        }
        cp_async_wait_all();
    } else if (warp < 15) {
        // ------------------------------------------ image loaders ------------------------------------------
        // slot g of this block's stream: tile g / SLOTS; M: (k-block, part), W1: (k-block, column tile, part), W2: (k-block, part)
        if (lane == 0) {
            int ti = 0, i = warp - 13;
            uint32_t s = (uint32_t)i, ph = 0;
            while (ti < n_my) {
                if (!mbar_wait(w_empty(s), ph ^ 1u, abort_flag, 71, &g_enc_out_status)) break;
                const float* src;
                if (i < 8) src = p.m_img + (int64_t)(tile_index(ti) / p.tps) * (2 * EN_D * EN_D) + i * 4096;
                else if (i < 24) { const int j = i - 8, kb = j >> 2, nt = (j >> 1) & 1; src = p.w1 + ((nt * 4 + kb) * 2 + (j & 1)) * 4096; }
                else src = p.w2 + (i - 24) * 4096;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(w_full(s)), "r"(EO_SLOT) : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(smem_base + s * EO_SLOT), "l"(src), "r"(EO_SLOT), "r"(w_full(s)) : "memory");
                if ((i += 2) >= SLOTS) { i -= SLOTS; ++ti; }
                if ((s += 2) >= EO_NW) { s -= EO_NW; ph ^= 1u; }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------ MMA issuer ------------------------------------------
        if (tc_elect()) {
            constexpr uint32_t idesc = tc_idesc(128);
            uint32_t ws = 0, wph = 0;
            // one k-block against one 128-column image (hi slot, then lo slot)
            auto block = [&](uint32_t d, uint32_t stage, bool fresh) {
                const uint32_t ah0 = tmem_base + EO_A + stage * 64;
                if (!mbar_wait(w_full(ws), wph, abort_flag, 72, &g_enc_out_status)) return false;
                tc_fence_after();
                uint64_t db = tc_smem_desc(smem_base + ws * EO_SLOT);
#pragma unroll
                for (int k8 = 0; k8 < 4; ++k8) {
                    tc_mma_tf32_ts(d, ah0 + 32 + k8 * 8, db + k8 * 2, idesc, (fresh && k8 == 0) ? 0u : 1u);
                    tc_mma_tf32_ts(d, ah0 + k8 * 8, db + k8 * 2, idesc, 1u);
                }
                tc_commit(w_empty(ws));
                if (++ws == EO_NW) { ws = 0; wph ^= 1u; }
                if (!mbar_wait(w_full(ws), wph, abort_flag, 73, &g_enc_out_status)) return false;
                tc_fence_after();
                db = tc_smem_desc(smem_base + ws * EO_SLOT);
#pragma unroll
                for (int k8 = 0; k8 < 4; ++k8) tc_mma_tf32_ts(d, ah0 + k8 * 8, db + k8 * 2, idesc, 1u);
                tc_commit(w_empty(ws));
                if (++ws == EO_NW) { ws = 0; wph ^= 1u; }
                return true;
            };
            bool alive = true;
            for (int ti = 0; ti < n_my && alive; ++ti) {
                const uint32_t par = (uint32_t)(ti & 1);
                const uint32_t d0 = tmem_base + (par ? 256u : 0u), d1 = tmem_base + (par ? 0u : 128u);
                uint32_t use = (uint32_t)(ti * USES);
                auto stage_ready = [&]() { return mbar_wait(a_full(use & 1u), (use >> 1) & 1u, abort_flag, 74, &g_enc_out_status); };
                if (!FFN && ti > 1 && !mbar_wait(d_free(par), (uint32_t)(((ti >> 1) - 1) & 1), abort_flag, 75, &g_enc_out_status)) break;
                for (int kb = 0; kb < 4; ++kb, ++use) {
                    if (!stage_ready() || !block(d0, use & 1u, kb == 0)) { alive = false; break; }
                    tc_commit(a_empty(use & 1u));
                }
                if (!alive) break;
                tc_commit(d0_full);
                if constexpr (FFN) {
                    // D1 covers the columns of the previous tile's last accumulator
                    if (ti > 0 && !mbar_wait(d_free(par ^ 1u), (uint32_t)(((ti - 1) >> 1) & 1), abort_flag, 76, &g_enc_out_status)) break;
                    for (int kb = 0; kb < 4; ++kb, ++use) {
                        if (!stage_ready() || !block(d1, use & 1u, kb == 0) || !block(d1 + 128, use & 1u, kb == 0)) { alive = false; break; }
                        tc_commit(a_empty(use & 1u));
                    }
                    if (!alive) break;
                    tc_commit(d1_full);
                    for (int kb = 0; kb < 8; ++kb, ++use) {
                        if (!stage_ready() || !block(d0, use & 1u, kb == 0)) { alive = false; break; }
                        tc_commit(a_empty(use & 1u));
                        if (kb == 4) tc_commit(x_go);
                    }
                    if (!alive) break;
                    tc_commit(d2_full);
                }
            }
        }
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 15) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

int encoder_out(const float* x, const float* m_img, const float* pc, const float* pos, const void* w1, const float* b1, const void* w2,
                const float* b2, float* y, int B, int S, int act, bool ffn, bool residual, cudaStream_t st) {
    EncoderOutParams p{x, m_img, pc, pos, (const float*)w1, b1, (const float*)w2, b2, y, S, ceil_div(S, EN_ROWS), 0, act, residual ? 1 : 0};
    p.n_tiles = B * p.tps;
    const int grid = p.n_tiles < num_sms() ? p.n_tiles : num_sms();
    if (ffn) {
        static SmemOptIn configured;
        if (int e = smem_opt_in(encoder_out_kernel<true>, EO_SMEM, configured)) return e;
        return launch_chained(encoder_out_kernel<true>, grid, EO_THREADS, EO_SMEM, st, p);
    } else {
        static SmemOptIn configured;
        if (int e = smem_opt_in(encoder_out_kernel<false>, EO_SMEM, configured)) return e;
        return launch_chained(encoder_out_kernel<false>, grid, EO_THREADS, EO_SMEM, st, p);
    }
}

int encoder_out_status(bool reset) {
    int v = 0;
    if (reset) return cudaMemcpyToSymbol(g_enc_out_status, &v, sizeof(int)) == cudaSuccess ? SPGT_OK : SPGT_ERR_LAUNCH;
    return cudaMemcpyFromSymbol(&v, g_enc_out_status, sizeof(int)) == cudaSuccess ? v : SPGT_ERR_LAUNCH;
}

}  // namespace spgt
