// K and V projections with per-head LayerNorm and the reduction T = [pos K]^T [pos V] over the grid nodes, for two of the four
// heads per thread block, without K or V leaving the SM (see encoder_common.cuh).
//
// Per 128-row tile: GEMM  D[128 rows][64 K | 64 V channels] = x W (3xTF32, x split into tensor memory, W as hi / lo images that
// stream from L2 for every tile: its shared memory holds operand tiles of all four 32-row quarters instead), normalisation by eight
// warps that own one row each, which store the result TRANSPOSED - one row per channel, 32 grid nodes long - as operand tiles, and one MMA per 8 nodes that multiplies
//   A = [K; K_lo] (64 + 64 rows)  with  B = [V; V_lo] (64 + 64 rows)
// so that all four hi / lo products of both heads come from one 128 x 128 x 8 instruction (the blocks between different heads
// are computed and dropped: narrower shapes take no less time).  The hi operand is the plain fp32 value: the tensor core reads
// its upper 19 bits, lo is what they leave.  The sums against the position values and 1 are fp32 sums over the same tiles.
//
// The tensor pipe needs 4100 cycles per tile (48 MMAs of 64 cycles for the projection and 16 for T); two accumulator buffers let the
// GEMM of a tile overlap the normalisation of the one before, whose T products follow it.  Measured on its own, 64 x 2809 nodes: 88 us
// = 6700 cycles per tile, tensor pipe 58 % and shared-memory data pipe 50 % busy: paced by the hand-offs between the roles.
// A block works on tiles of consecutive grid nodes and leaves one partial sum per sample it touches; the order of all additions is
// fixed by the sizes.  The accumulate step of an MMA truncates, so T chains end after 512 nodes (64 MMAs) and go
// on in fp32 registers.
//   warps 0-1 x loaders, 2 weight loader, 3 MMA issuer, 4-7 x splitters, 8-15 normalisation (K: 8-11, V: 12-15), 16-19 sums.
// Every wait is a bounded mbarrier poll that records a code on expiry.
#include "encoder_common.cuh"

namespace spgt {

__device__ int g_enc_kv_status = 0;

constexpr int KV_THREADS = 32 * 20;
constexpr int KV_W_BYTES = 2 * 32768, KV_BLOCK = 32768, KV_RAW = EN_ROWS * TC_BK * 4, KV_NR = 2;
constexpr int KV_OFF_T = KV_W_BYTES, KV_OFF_RAW = KV_OFF_T + 4 * KV_BLOCK, KV_OFF_CONST = KV_OFF_RAW + KV_NR * KV_RAW;
constexpr int KV_OFF_POS = KV_OFF_CONST + 128 * 4, KV_OFF_BAR = KV_OFF_POS + 4 * 32 * 8;
constexpr size_t KV_SMEM = KV_OFF_BAR + 256;
static_assert(KV_SMEM <= 227 * 1024, "shared memory budget");
constexpr uint32_t KV_T = 256, KV_A = 384;                     // tensor memory: D buffers [0,128) [128,256), T, two A stages
constexpr int KV_CHAIN = 4;                                    // tiles whose products one T accumulator sums

// Row of channel c (0..63) in a K or V operand tile: 16 hi rows, then the 16 lo rows of the same channels, so that hi and lo of
// a channel lie 16 lanes apart in one warp's quarter of tensor memory.
__device__ __forceinline__ constexpr int kv_tile_row(int c, int lo) { return (c >> 4) * 32 + (c & 15) + 16 * lo; }

__global__ void __launch_bounds__(KV_THREADS, 1)
encoder_kv_kernel(const float* __restrict__ x, const float* __restrict__ wkv_img, const float* __restrict__ bk, const float* __restrict__ bv,
                  float eps, const float* __restrict__ pos, float* __restrict__ partial, int S, EncoderSplit sp) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t smem_base = smem_u32(smem);
    if (smem_base & 1023u) {                                   // (operand tiles need 1024-byte alignment; dynamic shared memory starts so)
        if (threadIdx.x == 0) atomicCAS(&g_enc_kv_status, 0, 40);
        return;
    }
    float* consts = reinterpret_cast<float*>(smem + KV_OFF_CONST);      // projection biases less their head's mean, K 64 | V 64
    const uint32_t bars = smem_base + KV_OFF_BAR;
    auto raw_full = [&](int s) { return bars + 8u * s; };              // [2]
    auto raw_empty = [&](int s) { return bars + 8u * (2 + s); };       // [2]
    auto a_full = [&](int s) { return bars + 8u * (4 + s); };          // [2]
    auto a_empty = [&](int s) { return bars + 8u * (6 + s); };         // [2]
    auto d_full = [&](int s) { return bars + 8u * (8 + s); };          // [2]
    auto d_empty = [&](int s) { return bars + 8u * (10 + s); };        // [2]
    auto t_full = [&](int q) { return bars + 8u * (12 + q); };         // [4] one per 32-row quarter of a tile
    auto t_empty = [&](int q) { return bars + 8u * (16 + q); };        // [4]
    const uint32_t acc_full = bars + 8u * 20, acc_free = bars + 8u * 21;
    auto w_full = [&](uint32_t s) { return bars + 8u * (22 + s); };    // [2]
    auto w_empty = [&](uint32_t s) { return bars + 8u * (24 + s); };   // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + KV_OFF_BAR + 224);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + KV_OFF_BAR + 232);

    const int tid = threadIdx.x, warp = (int)tc_uniform(tid >> 5), lane = tid & 31;
    const int pair = blockIdx.x & 1, cta = blockIdx.x >> 1;
    const int u_begin = sp.begin(cta), n_my = sp.begin(cta + 1) - u_begin;
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(raw_full(s), 64); mbar_init(raw_empty(s), 128); mbar_init(a_full(s), 128); mbar_init(a_empty(s), 1);
            mbar_init(d_full(s), 1); mbar_init(d_empty(s), 256); mbar_init(w_full(s), 1); mbar_init(w_empty(s), 1);
        }
        for (int q = 0; q < 4; ++q) { mbar_init(t_full(q), 64); mbar_init(t_empty(q), 5); }
        mbar_init(acc_full, 1); mbar_init(acc_free, 4);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 3) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (warp >= 4 && warp < 8) {                               // one head per warp
        const int c = pair * 64 + (warp & 1) * 32 + lane;
        const float* bias = warp < 6 ? bk : bv;
        const float v = bias ? __ldg(bias + c) : 0.0f;
        float m = v;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
        consts[(warp - 4) * 32 + lane] = v - m * (1.0f / 32.0f);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tc_uniform(*tmem_slot);
    pdl_wait();
    pdl_launch_next();
    // a chain of T products ends with the sample, with this block's last tile, or after KV_CHAIN tiles
    auto tile_of = [&](int i) { return (u_begin + i) % sp.tps; };
    auto chain_ends = [&](int i, int len) { return len == KV_CHAIN || i == n_my - 1 || tile_of(i) == sp.tps - 1; };

    if (warp < 2) {
        // ------------------------------------------ x loaders ------------------------------------------
        // thread t copies chunk (t & 7) of rows (t >> 3) + 8 k: rows eight apart lie 1024 bytes apart in the swizzled tile
        const uint32_t dst0 = smem_base + KV_OFF_RAW + tc_swz(tid >> 3, tid & 7);
        uint32_t sr = 0, ph = 0;
        bool alive = true;
        for (int i = 0; i < n_my && alive; ++i) {
            const int u = u_begin + i, b = u / sp.tps, row0 = (u - b * sp.tps) * EN_ROWS + (tid >> 3);
            const float* xb = x + ((int64_t)b * S + row0) * EN_D + (tid & 7) * 4;
            for (int kb = 0; kb < 4; ++kb) {
                if (!mbar_wait(raw_empty(sr), ph ^ 1, abort_flag, 41, &g_enc_kv_status)) { alive = false; break; }
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    const bool ok = row0 + 8 * k < S;
                    const float* p = ok ? xb + k * (8 * EN_D) + kb * TC_BK : x;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst0 + sr * KV_RAW + k * 1024), "l"(p), "r"(ok ? 16 : 0) : "memory");
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(raw_full(sr)) : "memory");
                if (++sr == KV_NR) { sr = 0; ph ^= 1u; }
            }
        }
        cp_async_wait_all();
    } else if (warp >= 4 && warp < 8) {
        // ------------------------------------------ x splitters ------------------------------------------
        const int q = warp & 3, r = q * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
        uint32_t roff[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) roff[c] = tc_swz(r, c);
        uint32_t s = 0, ph = 0;                                 // raw and A rings have the same depth
        for (int n = 0; n < 4 * n_my; ++n) {
            if (!mbar_wait(raw_full(s), ph, abort_flag, 42, &g_enc_kv_status)) break;
            // the raw stage is free for the next load as soon as its values are in registers
            const uint8_t* src = smem + KV_OFF_RAW + s * KV_RAW;
            float4 w[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) w[j] = *reinterpret_cast<const float4*>(src + roff[j]);
            mbar_arrive(raw_empty(s));
            uint32_t hi[32], lo[32];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                split_tf32(w[j].x, hi[4 * j], lo[4 * j]); split_tf32(w[j].y, hi[4 * j + 1], lo[4 * j + 1]);
                split_tf32(w[j].z, hi[4 * j + 2], lo[4 * j + 2]); split_tf32(w[j].w, hi[4 * j + 3], lo[4 * j + 3]);
            }
            if (!mbar_wait(a_empty(s), ph ^ 1, abort_flag, 43, &g_enc_kv_status)) break;
            tc_fence_after();
            const uint32_t a_hi = tmem_base + lane_addr + KV_A + s * 64;
            tc_st16(a_hi, reinterpret_cast<uint32_t(&)[16]>(hi[0]));
            tc_st16(a_hi + 16, reinterpret_cast<uint32_t(&)[16]>(hi[16]));
            tc_st16(a_hi + 32, reinterpret_cast<uint32_t(&)[16]>(lo[0]));
            tc_st16(a_hi + 48, reinterpret_cast<uint32_t(&)[16]>(lo[16]));
            tc_wait_st();
            tc_fence_before();
            mbar_arrive(a_full(s));
            if (++s == KV_NR) { s = 0; ph ^= 1u; }
        }
    } else if (warp == 2) {
        // ------------------------------------------ weight images ------------------------------------------
        if (lane == 0) {
            uint32_t s = 0, ph = 0;
            for (int n = 0; n < 4 * n_my; ++n) {
                if (!mbar_wait(w_empty(s), ph ^ 1, abort_flag, 44, &g_enc_kv_status)) break;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(w_full(s)), "r"(32768) : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(smem_base + s * 32768), "l"(wkv_img + (pair * 4 + (n & 3)) * 8192), "r"(32768), "r"(w_full(s)) : "memory");
                if (++s == 2) { s = 0; ph ^= 1u; }
            }
        }
        __syncwarp();
    } else if (warp == 3) {
        // ------------------------------------------ MMA issuer ------------------------------------------
        if (tc_elect()) {
            constexpr uint32_t idesc = tc_idesc(128);
            uint32_t s = 0, ph = 0;
            int chain = 0, nchain = 0;                          // tiles in the running T chain, chains begun
            bool alive = true;
            // T products of tile i
            auto t_products = [&](int i) {
                if (chain == 0 && nchain > 0 && !mbar_wait(acc_free, (uint32_t)((nchain - 1) & 1), abort_flag, 47, &g_enc_kv_status)) return false;
                for (int q = 0; q < 4; ++q) {
                    if (!mbar_wait(t_full(q), (uint32_t)(i & 1), abort_flag, 48, &g_enc_kv_status)) return false;
                    tc_fence_after();
                    const uint32_t blk = smem_base + KV_OFF_T + q * KV_BLOCK;
                    const uint64_t da = tc_smem_desc(blk), db = tc_smem_desc(blk + 16384);
#pragma unroll
                    for (int k8 = 0; k8 < 4; ++k8)
                        tc_mma_tf32_ss(tmem_base + KV_T, da + k8 * 2, db + k8 * 2, idesc, (chain > 0 || q > 0 || k8 > 0) ? 1u : 0u);
                    tc_commit(t_empty(q));
                }
                if (chain_ends(i, ++chain)) { tc_commit(acc_full); chain = 0; ++nchain; }
                return true;
            };
            for (int i = 0; i < n_my && alive; ++i) {
                const uint32_t buf = (uint32_t)(i & 1), dph = (uint32_t)((i >> 1) & 1);
                if (!mbar_wait(d_empty(buf), dph ^ 1, abort_flag, 45, &g_enc_kv_status)) { alive = false; break; }
                tc_fence_after();
                const uint32_t d = tmem_base + buf * 128;
                for (int kb = 0; kb < 4 && alive; ++kb) {
                    // (the A and W rings have the same depth)
                    if (!alive || !mbar_wait(w_full(s), ph, abort_flag, 54, &g_enc_kv_status) ||
                        !mbar_wait(a_full(s), ph, abort_flag, 46, &g_enc_kv_status)) { alive = false; break; }
                    tc_fence_after();
                    const uint64_t bh = tc_smem_desc(smem_base + s * 32768), bl = tc_smem_desc(smem_base + s * 32768 + 16384);
                    const uint32_t ah0 = tmem_base + KV_A + s * 64;
#pragma unroll
                    for (int k8 = 0; k8 < 4; ++k8) {
                        const uint32_t ah = ah0 + k8 * 8, al = ah + 32;
                        tc_mma_tf32_ts(d, al, bh + k8 * 2, idesc, (kb > 0 || k8 > 0) ? 1u : 0u);
                        tc_mma_tf32_ts(d, ah, bl + k8 * 2, idesc, 1u);
                        tc_mma_tf32_ts(d, ah, bh + k8 * 2, idesc, 1u);
                    }
                    tc_commit(a_empty(s));
                    tc_commit(w_empty(s));
                    if (++s == KV_NR) { s = 0; ph ^= 1u; }
                }
                if (!alive) break;
                tc_commit(d_full(buf));
                if (i > 0) alive = t_products(i - 1);
            }
            if (alive && n_my > 0) (void)t_products(n_my - 1);
        }
        __syncwarp();
    } else if (warp >= 8 && warp < 16) {
        // ------------------------------------------ normalisation ------------------------------------------
        const int q = warp & 3, isv = (warp - 8) >> 2;
        const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
        uint8_t* tile = smem + KV_OFF_T + q * KV_BLOCK + isv * 16384;
        uint32_t coff[8];                                       // this node's position inside a row with (row & 7) = j
#pragma unroll
        for (int j = 0; j < 8; ++j) coff[j] = (uint32_t)(j * 128 + (((lane >> 2) ^ j) << 4) + (lane & 3) * 4);
        const float4* c4 = reinterpret_cast<const float4*>(consts + isv * 64);
        for (int i = 0; i < n_my; ++i) {
            const uint32_t buf = (uint32_t)(i & 1), dph = (uint32_t)((i >> 1) & 1);
            const bool valid = tile_of(i) * EN_ROWS + q * 32 + lane < S;
            if (!mbar_wait(d_full(buf), dph, abort_flag, 49, &g_enc_kv_status)) break;
            tc_fence_after();
            bool ok = true;
#pragma unroll 1
            for (int hd = 0; hd < 2; ++hd) {                    // 32 channels each
                float v[32];
                tc_ld32(tmem_base + lane_addr + buf * 128 + isv * 64 + hd * 32, v);
                if (hd == 1) { tc_fence_before(); mbar_arrive(d_empty(buf)); }
                float2* v2 = reinterpret_cast<float2*>(v);
                float2 q0 = make_float2(0.f, 0.f), q1 = q0;
#pragma unroll
                for (int j4 = 0; j4 < 8; ++j4) {
                    const float4 bb = c4[hd * 8 + j4];
                    v2[2 * j4] = add2(v2[2 * j4], make_float2(bb.x, bb.y));
                    v2[2 * j4 + 1] = add2(v2[2 * j4 + 1], make_float2(bb.z, bb.w));
                    q0 = fma2(v2[2 * j4], v2[2 * j4], q0);
                    q1 = fma2(v2[2 * j4 + 1], v2[2 * j4 + 1], q1);
                }
                const float inv = valid ? 1.0f / sqrtf(((q0.x + q0.y) + (q1.x + q1.y)) * (1.0f / 32.0f) + eps) : 0.0f;
                // the operand tile of this quarter is free once the previous tile's MMAs and sums have read it
                if (hd == 0 && i > 0) ok = mbar_wait(t_empty(q), (uint32_t)((i - 1) & 1), abort_flag, 50, &g_enc_kv_status);
                if (!ok) break;
                uint8_t* rows = tile + hd * 8192;
                const float2 inv2 = make_float2(inv, inv), minus2 = make_float2(-1.0f, -1.0f);
#pragma unroll
                for (int j8 = 0; j8 < 32; j8 += 8) {            // (four independent pairs at a time)
                    float2 n[4], l[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e) n[e] = mul2(v2[j8 / 2 + e], inv2);
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        l[e] = fma2(make_float2(__uint_as_float(__float_as_uint(n[e].x) & 0xffffe000u), __uint_as_float(__float_as_uint(n[e].y) & 0xffffe000u)), minus2, n[e]);
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const int r = kv_tile_row(j8 + e, 0);
                        const float nv = (e & 1) ? n[e >> 1].y : n[e >> 1].x, lv = (e & 1) ? l[e >> 1].y : l[e >> 1].x;
                        *reinterpret_cast<float*>(rows + (r >> 3) * 1024 + coff[r & 7]) = nv;
                        // (half an ulp of tf32 added: the tensor core's truncation then rounds to nearest)
                        *reinterpret_cast<uint32_t*>(rows + ((r >> 3) + 2) * 1024 + coff[r & 7]) = __float_as_uint(lv) + 0x1000u;
                    }
                }
            }
            if (!ok) break;
            fence_proxy_async();
            mbar_arrive(t_full(q));
        }
    } else if (warp >= 16) {
        // ------------------------------------------ sums ------------------------------------------
        // T: this thread owns tensor-memory lane 32 q + lane = operand row of K channel 16 q + (lane & 15), hi (lane < 16) or lo.
        // Position sums: channel 32 (q & 1) + lane of K (q < 2) or V, from its fp32 row.
        const int q = warp & 3, hd = q >> 1, sch = (q & 1) * 32 + lane, srow = kv_tile_row(sch, 0);
        const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
        float* mypos = reinterpret_cast<float*>(smem + KV_OFF_POS) + q * 64;       // [2][32]
        uint32_t roff[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) roff[c] = (uint32_t)((q >> 1) * 16384) + tc_swz(srow, c);
        float acc[32], sum[3] = {0.f, 0.f, 0.f}, pp[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 32; ++j) acc[j] = 0.0f;
        float2 pcur[4], pnext[4];                               // position values of a tile's four nodes of this lane, fetched a tile ahead
        auto fetch_pos = [&](int i) {
            const int u = u_begin + (i < n_my ? i : 0), b = u / sp.tps, node0 = (u - b * sp.tps) * EN_ROWS + lane;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                pnext[k] = i < n_my && node0 + 32 * k < S ? __ldg(reinterpret_cast<const float2*>(pos) + (int64_t)b * S + node0 + 32 * k) : make_float2(0.f, 0.f);
        };
        fetch_pos(0);
        int chain = 0, nchain = 0;
        bool alive = true;
        for (int i = 0; i < n_my && alive; ++i) {
#pragma unroll
            for (int k = 0; k < 4; ++k) pcur[k] = pnext[k];
            fetch_pos(i + 1);
#pragma unroll
            for (int bq = 0; bq < 4; ++bq) {
                __syncwarp();
                const float2 pn = pcur[bq];
                mypos[lane] = pn.x; mypos[32 + lane] = pn.y;
                pp[0] += pn.x * pn.x; pp[1] += pn.x * pn.y; pp[2] += pn.y * pn.y; pp[3] += pn.x; pp[4] += pn.y;
                __syncwarp();
                if (!mbar_wait(t_full(bq), (uint32_t)(i & 1), abort_flag, 51, &g_enc_kv_status)) { alive = false; break; }
                const uint8_t* blk = smem + KV_OFF_T + bq * KV_BLOCK;
                float4 v[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) v[c] = *reinterpret_cast<const float4*>(blk + roff[c]);
                __syncwarp();
                if (lane == 0) mbar_arrive(t_empty(bq));
                float2 a0 = make_float2(0.f, 0.f), a1 = a0, a2 = a0;
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float4 px = reinterpret_cast<const float4*>(mypos)[c], py = reinterpret_cast<const float4*>(mypos)[8 + c];
                    const float2 va = make_float2(v[c].x, v[c].y), vb = make_float2(v[c].z, v[c].w);
                    a0 = fma2(va, make_float2(px.x, px.y), a0); a0 = fma2(vb, make_float2(px.z, px.w), a0);
                    a1 = fma2(va, make_float2(py.x, py.y), a1); a1 = fma2(vb, make_float2(py.z, py.w), a1);
                    a2 = add2(va, a2); a2 = add2(vb, a2);
                }
                sum[0] += a0.x + a0.y; sum[1] += a1.x + a1.y; sum[2] += a2.x + a2.y;
            }
            if (!alive) break;
            if (!chain_ends(i, ++chain)) continue;
            chain = 0;
            if (!mbar_wait(acc_full, (uint32_t)(nchain & 1), abort_flag, 52, &g_enc_kv_status)) break;
            ++nchain;
            tc_fence_after();
#pragma unroll
            for (int g = 0; g < 2; ++g) {                       // columns: 16 hi and 16 lo rows of V channels 16 g .. 16 g + 15 of this head
                float v[32];
                tc_ld32(tmem_base + lane_addr + KV_T + hd * 64 + g * 32, v);
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[16 * g + j] += v[j] + v[16 + j];
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_free);
            if (i < n_my - 1 && tile_of(i) != sp.tps - 1) continue;
            // the sample's (or this block's) last tile: hi + lo rows, then out
            const int b = (u_begin + i) / sp.tps;
            float* out = partial + ((int64_t)(b * EN_PAIRS + pair) * sp.max_parts + (cta - sp.owner(b * sp.tps))) * EN_P_FLOATS;
            const int ch = 16 * q + (lane & 15), half = lane >> 4;
            float full[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float lo_half = acc[j] + __shfl_xor_sync(0xffffffffu, acc[j], 16), hi_half = acc[16 + j] + __shfl_xor_sync(0xffffffffu, acc[16 + j], 16);
                full[j] = half ? hi_half : lo_half;
            }
            float4* dst = reinterpret_cast<float4*>(out + EN_P_CORE + ch * 32 + half * 16);
#pragma unroll
            for (int j = 0; j < 4; ++j) dst[j] = make_float4(full[4 * j], full[4 * j + 1], full[4 * j + 2], full[4 * j + 3]);
#pragma unroll
            for (int e = 0; e < 3; ++e) { out[(q < 2 ? EN_P_K : EN_P_V) + e * 64 + sch] = sum[e]; sum[e] = 0.0f; }
#pragma unroll
            for (int e = 0; e < 5; ++e) {
                float t = pp[e];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
                if (q == 0 && lane == 0) out[EN_P_POS + e] = t;
                pp[e] = 0.0f;
            }
#pragma unroll
            for (int j = 0; j < 32; ++j) acc[j] = 0.0f;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 3) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

int encoder_kv(const float* x, const void* wkv, const float* bk, const float* bv, float eps, const float* pos, float* partial, int S,
               const EncoderSplit& sp, cudaStream_t st) {
    static SmemOptIn configured;
    if (int e = smem_opt_in(encoder_kv_kernel, KV_SMEM, configured)) return e;
    return launch_chained(encoder_kv_kernel, EN_PAIRS * sp.per_pair, KV_THREADS, KV_SMEM, st, x, (const float*)wkv, bk, bv, eps, pos, partial, S, sp);
}

int encoder_kv_status(bool reset) {
    int v = 0;
    if (reset) return cudaMemcpyToSymbol(g_enc_kv_status, &v, sizeof(int)) == cudaSuccess ? SPGT_OK : SPGT_ERR_LAUNCH;
    return cudaMemcpyFromSymbol(&v, g_enc_kv_status, sizeof(int)) == cudaSuccess ? v : SPGT_ERR_LAUNCH;
}

}  // namespace spgt
