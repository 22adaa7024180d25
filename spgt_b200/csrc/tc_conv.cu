// 3x3 convolution, padding 1, NHWC, on tcgen05 with both operands in shared memory (3xTF32).
//
// A tile is 8 x 16 output pixels = the 128 rows of an MMA, row m at (m / 8, m % 8).  For 32 input channels at a time its 10 x 18
// input pixels are split ONCE into hi and lo and stored without swizzle as [4-channel chunk][pixel][16 bytes]: the
// eight rows of a core matrix are then eight neighbouring pixels, so the A operand of filter tap (dy, dx) is the same memory
// with the start address moved by dy * 10 + dx pixels.  (The implicit GEMM before this gathered and split every input value nine
// times; that, not the MMAs, set its pace: 275 cycles per 8 k-values and 128 pixels for 44 output channels.)
// The image rows of all samples are taken as one column of rows with one zero row after each sample, so only the last row of
// tiles of the whole batch is ragged.
//
// B = [W_hi | W_lo], one 32-channel block of one tap after the other through a ring of bulk copies.  Per 8 k-values one MMA
// A_hi x [W_hi | W_lo] (two partial accumulators) and one A_lo x W_hi; with A in shared memory an MMA takes
// max(N / 2, 32 + N / 4) cycles, 101 for 48 output channels and 194 for 128.  Two accumulator buffers: the epilogue of a
// tile overlaps the MMAs of the next.  Measured on their own, 32 x 106 x 106: 128 -> 128 channels 397 us, tensor pipe 93 % busy;
// 128 -> 44 237 us, 56 % (A is read from shared memory twice as long as the narrow MMA takes, 72 of 101 cycles).
//   warps 0-7 load and split, 8 weight loader, 9 MMA issuer, 10-13 epilogue.
// Every wait is a bounded mbarrier poll that records a code on expiry.
#include "tc_common.cuh"

namespace spgt {

__device__ int g_conv_status = 0;

constexpr int CV_TX = 8, CV_TY = 16, CV_HX = CV_TX + 2, CV_HY = CV_TY + 2, CV_PX = CV_HX * CV_HY;       // tile, halo, halo pixels
constexpr int CV_CH = 32;                                                 // channels of a stage
constexpr uint32_t CV_LBO = (CV_PX + 1) * 16;                             // odd number of 16-byte units: stores without bank conflicts
constexpr uint32_t CV_SBO = CV_HX * 16;
constexpr uint32_t CV_HALF = CV_CH / 4 * CV_LBO, CV_STAGE = 2 * CV_HALF;  // hi (or lo) part of a stage
constexpr int CV_NA = 2, CV_STAGERS = 256, CV_ITEMS = (CV_PX + CV_STAGERS / 8 - 1) / (CV_STAGERS / 8);
constexpr int CV_THREADS = CV_STAGERS + 64 + 128, CV_SLOT = 16 * 4 + 16;
template <int BN> struct CvCfg {
    // One bulk copy brings the taps of a filter row (the issuing thread needs about 400 cycles per copy and wait whatever the size,
    // as long as a tap's MMAs for 48 channels take), or one tap of 128 channels.
    static constexpr int TAPS = BN == 128 ? 1 : 3, W_TAP = 2 * BN * CV_CH * 4, W_BLOCK = TAPS * W_TAP, NW = BN == 128 ? 3 : 2, ACCW = 2 * BN;
    static constexpr int TMEM = 2 * ACCW <= 256 ? 256 : 512;
    static constexpr int OFF_A = NW * W_BLOCK, OFF_STG = OFF_A + CV_NA * CV_STAGE, OFF_BIAS = OFF_STG + 128 * CV_SLOT, OFF_BAR = OFF_BIAS + BN * 4;
    static constexpr size_t BYTES = OFF_BAR + 256;
    static_assert(BYTES <= 227 * 1024 && W_BLOCK % 1024 == 0, "shared memory budget");
};

struct ConvParams {
    const float *x, *wimg, *bias;
    float* y;
    int cin_pitch, cin, cout_pitch, cout, B, H, W, act, gx, n_tiles;
};

// K-major operand without swizzle: core matrices of 8 rows x 16 bytes, LBO apart along k, SBO along the rows.
__device__ __forceinline__ uint64_t cv_a_desc(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)(CV_LBO >> 4) << 16) | ((uint64_t)(CV_SBO >> 4) << 32) | (1ull << 46);
}

template <int BN>
__global__ void __launch_bounds__(CV_THREADS, 1) conv3x3_kernel(const ConvParams p) {
    using C = CvCfg<BN>;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t smem_base = smem_u32(smem);
    if (smem_base & 1023u) {
        if (threadIdx.x == 0) atomicCAS(&g_conv_status, 0, 80);
        return;
    }
    float* bias = reinterpret_cast<float*>(smem + C::OFF_BIAS);
    const uint32_t bars = smem_base + C::OFF_BAR;
    auto a_full = [&](uint32_t s) { return bars + 8u * s; };             // [2]
    auto a_empty = [&](uint32_t s) { return bars + 8u * (2 + s); };      // [2]
    auto acc_full = [&](uint32_t s) { return bars + 8u * (4 + s); };     // [2]
    auto acc_empty = [&](uint32_t s) { return bars + 8u * (6 + s); };    // [2]
    auto w_full = [&](uint32_t s) { return bars + 8u * (8 + s); };       // [NW]
    auto w_empty = [&](uint32_t s) { return bars + 8u * (8 + C::NW + s); };
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + C::OFF_BAR + 224);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + C::OFF_BAR + 232);

    const int tid = threadIdx.x, warp = (int)tc_uniform(tid >> 5), lane = tid & 31;
    const int n_my = ((int)blockIdx.x < p.n_tiles) ? (p.n_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
    const int chunks = (p.cin + CV_CH - 1) / CV_CH;
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) { mbar_init(a_full(s), CV_STAGERS); mbar_init(a_empty(s), 1); mbar_init(acc_full(s), 1); mbar_init(acc_empty(s), 128); }
        for (int s = 0; s < C::NW; ++s) { mbar_init(w_full(s), 1); mbar_init(w_empty(s), 1); }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(C::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i < BN; i += CV_THREADS) bias[i] = p.bias != nullptr && i < p.cout ? __ldg(p.bias + i) : 0.0f;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tc_uniform(*tmem_slot);
    pdl_wait();
    pdl_launch_next();

    if (warp < 8) {
        // ------------------------------------------ load and split ------------------------------------------
        // thread (pixel, 4 channels): eight threads read the 32 channels of a pixel
        const int c4 = tid & 7, p0 = tid >> 3;
        uint32_t s = 0, ph = 0;
        bool alive = true;
        const float* src[CV_ITEMS];
        float4 v[CV_ITEMS];
        auto locate = [&](int ti) {                              // source address of every item of a tile (nullptr: outside the image)
            const int tile = (int)blockIdx.x + ti * (int)gridDim.x, ty = tile / p.gx, tx = tile - ty * p.gx;
#pragma unroll
            for (int k = 0; k < CV_ITEMS; ++k) {
                const int px = p0 + k * (CV_STAGERS / 8), yy = px / CV_HX, xx = px - yy * CV_HX;
                const int g = ty * CV_TY - 1 + yy, x = tx * CV_TX - 1 + xx;
                src[k] = nullptr;
                if (px < CV_PX && g >= 0 && x >= 0 && x < p.W) {
                    const int b = g / (p.H + 1), y = g - b * (p.H + 1);
                    if (b < p.B && y < p.H) src[k] = p.x + ((int64_t)(b * p.H + y) * p.W + x) * p.cin_pitch + c4 * 4;
                }
            }
        };
        auto fetch = [&](int chunk) {
            const bool in = chunk * CV_CH + c4 * 4 < p.cin;
#pragma unroll
            for (int k = 0; k < CV_ITEMS; ++k)
                v[k] = in && src[k] != nullptr ? __ldca(reinterpret_cast<const float4*>(src[k] + chunk * CV_CH)) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        if (n_my > 0) { locate(0); fetch(0); }
        for (int ti = 0; ti < n_my && alive; ++ti)
            for (int chunk = 0; chunk < chunks; ++chunk) {
                if (!mbar_wait(a_empty(s), ph ^ 1u, abort_flag, 81, &g_conv_status)) { alive = false; break; }
                uint8_t* dst = smem + C::OFF_A + s * CV_STAGE + c4 * CV_LBO + p0 * 16;
#pragma unroll
                for (int k = 0; k < CV_ITEMS; ++k) {
                    if (p0 + k * (CV_STAGERS / 8) < CV_PX) {
                        uint4 h, l;
                        split_tf32(v[k].x, h.x, l.x); split_tf32(v[k].y, h.y, l.y); split_tf32(v[k].z, h.z, l.z); split_tf32(v[k].w, h.w, l.w);
                        *reinterpret_cast<uint4*>(dst + k * (CV_STAGERS / 8 * 16)) = h;
                        *reinterpret_cast<uint4*>(dst + CV_HALF + k * (CV_STAGERS / 8 * 16)) = l;
                    }
                }
                fence_proxy_async();
                mbar_arrive(a_full(s));
                if (++s == CV_NA) { s = 0; ph ^= 1u; }
                if (chunk + 1 < chunks) fetch(chunk + 1);        // lands while the MMAs work on the stage before
                else if (ti + 1 < n_my) { locate(ti + 1); fetch(0); }
            }
    } else if (warp == 8) {
        // ------------------------------------------ weight blocks ------------------------------------------
        if (lane == 0) {
            uint32_t s = 0, ph = 0;
            const int blocks = chunks * (9 / C::TAPS);
            bool alive = true;
            for (int ti = 0; ti < n_my && alive; ++ti)
                for (int k = 0; k < blocks; ++k) {
                    if (!mbar_wait(w_empty(s), ph ^ 1u, abort_flag, 82, &g_conv_status)) { alive = false; break; }
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(w_full(s)), "r"(C::W_BLOCK) : "memory");
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                 ::"r"(smem_base + s * C::W_BLOCK), "l"(p.wimg + (int64_t)k * (C::W_BLOCK / 4)), "r"(C::W_BLOCK), "r"(w_full(s)) : "memory");
                    if (++s == (uint32_t)C::NW) { s = 0; ph ^= 1u; }
                }
        }
        __syncwarp();
    } else if (warp == 9) {
        // ------------------------------------------ MMA issuer ------------------------------------------
        if (tc_elect()) {
            constexpr uint32_t idesc2 = tc_idesc(2 * BN), idesc1 = tc_idesc(BN);
            uint32_t s = 0, ph = 0, ws = 0, wph = 0;
            bool alive = true;
            for (int ti = 0; ti < n_my && alive; ++ti) {
                const uint32_t buf = (uint32_t)(ti & 1), d = tmem_base + buf * C::ACCW;
                if (!mbar_wait(acc_empty(buf), (uint32_t)((ti >> 1) & 1) ^ 1u, abort_flag, 83, &g_conv_status)) break;
                for (int chunk = 0; chunk < chunks && alive; ++chunk) {
                    if (!mbar_wait(a_full(s), ph, abort_flag, 84, &g_conv_status)) { alive = false; break; }
                    const uint32_t a0 = smem_base + C::OFF_A + s * CV_STAGE;
                    const int left = p.cin - chunk * CV_CH, nk8 = left >= CV_CH ? CV_CH / 8 : (left + 7) / 8;
                    for (int tap0 = 0; tap0 < 9; tap0 += C::TAPS) {
                        if (!mbar_wait(w_full(ws), wph, abort_flag, 85, &g_conv_status)) { alive = false; break; }
                        tc_fence_after();
#pragma unroll
                        for (int e = 0; e < C::TAPS; ++e) {
                            const int tap = tap0 + e, dy = tap / 3, dx = tap - dy * 3;
                            const uint64_t ah = cv_a_desc(a0 + (uint32_t)(dy * CV_HX + dx) * 16), al = cv_a_desc(a0 + CV_HALF + (uint32_t)(dy * CV_HX + dx) * 16);
                            const uint64_t db = tc_smem_desc(smem_base + ws * C::W_BLOCK + e * C::W_TAP);
                            constexpr uint64_t AK = 2 * CV_LBO >> 4;     // two 4-channel chunks per k-step
                            auto step = [&](int k8) {
                                tc_mma_tf32_ss(d, ah + k8 * AK, db + k8 * 2, idesc2, (chunk > 0 || tap > 0 || k8 > 0) ? 1u : 0u);
                                tc_mma_tf32_ss(d, al + k8 * AK, db + k8 * 2, idesc1, 1u);
                            };
                            if (nk8 == 4) {
#pragma unroll
                                for (int k8 = 0; k8 < 4; ++k8) step(k8);
                            } else {
                                for (int k8 = 0; k8 < nk8; ++k8) step(k8);
                            }
                        }
                        tc_commit(w_empty(ws));
                        if (++ws == (uint32_t)C::NW) { ws = 0; wph ^= 1u; }
                    }
                    if (!alive) break;
                    tc_commit(a_empty(s));
                    if (++s == CV_NA) { s = 0; ph ^= 1u; }
                }
                if (alive) tc_commit(acc_full(buf));
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------ epilogue ------------------------------------------
        // thread = one pixel: bias and activation on 16 channels into its staging row, then the warp stores its 32 pixels (four
        // image rows of eight) with four lanes per pixel
        const int q = warp & 3;
        float* slot = reinterpret_cast<float*>(smem + C::OFF_STG + (q * 32 + lane) * CV_SLOT);
        const uint8_t* stage = smem + C::OFF_STG + q * 32 * CV_SLOT;
        const int sl = (lane & 3) * 4, sr = lane >> 2;           // store phase: channel offset, pixel in the eight of an image row
        for (int ti = 0; ti < n_my; ++ti) {
            const uint32_t buf = (uint32_t)(ti & 1), taddr = tmem_base + ((uint32_t)(q * 32) << 16) + buf * C::ACCW;
            const int tile = (int)blockIdx.x + ti * (int)gridDim.x, ty = tile / p.gx, tx = tile - ty * p.gx;
            float* yp[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int g = ty * CV_TY + q * 4 + i, b = g / (p.H + 1), y = g - b * (p.H + 1), x = tx * CV_TX + sr;
                yp[i] = b < p.B && y < p.H && x < p.W ? p.y + ((int64_t)(b * p.H + y) * p.W + x) * p.cout_pitch + sl : nullptr;
            }
            if (!mbar_wait(acc_full(buf), (uint32_t)((ti >> 1) & 1), abort_flag, 86, &g_conv_status)) break;
            tc_fence_after();
#pragma unroll 1
            for (int c0 = 0; c0 < BN; c0 += 16) {
                float v[16];
                tc_ld16_sum(taddr + c0, BN, v);
                if (c0 + 16 >= BN) { tc_fence_before(); mbar_arrive(acc_empty(buf)); }
                auto finish = [&](auto actf) {
#pragma unroll
                    for (int j4 = 0; j4 < 4; ++j4) {
                        const float4 b = *reinterpret_cast<const float4*>(bias + c0 + 4 * j4);
                        *reinterpret_cast<float4*>(slot + 4 * j4) =
                            make_float4(actf(v[4 * j4] + b.x), actf(v[4 * j4 + 1] + b.y), actf(v[4 * j4 + 2] + b.z), actf(v[4 * j4 + 3] + b.w));
                    }
                };
                if (p.act == SPGT_ACT_SILU2) finish([](float t) { return silu_f(silu_f(t)); });
                else if (p.act == SPGT_ACT_RELU) finish([](float t) { return fmaxf(t, 0.0f); });
                else if (p.act == SPGT_ACT_SILU) finish([](float t) { return silu_f(t); });
                else finish([](float t) { return t; });
                __syncwarp();
                if (c0 + sl < p.cout) {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (yp[i] != nullptr)
                            *reinterpret_cast<float4*>(yp[i] + c0) = *reinterpret_cast<const float4*>(stage + (i * 8 + sr) * CV_SLOT + sl * 4);
                }
                __syncwarp();
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 9) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(C::TMEM) : "memory");
    }
}

// [9 * Cin][ldw] (k = tap * Cin + c) -> per (32 channels, tap) the B operand image [W_hi | W_lo] of BN rows, zero padded.
__global__ void conv_weight_prepare_kernel(const float* __restrict__ w, int ldw, int cin, int cout, int bn, float* __restrict__ img, int total) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int kk = i % CV_CH, n = (i / CV_CH) % bn, block = i / (CV_CH * bn), tap = block % 9, c = block / 9 * CV_CH + kk;
    const float v = n < cout && c < cin ? __ldg(w + (int64_t)(tap * cin + c) * ldw + n) : 0.0f;
    tc_img_store(img + (int64_t)block * (2 * bn * CV_CH), bn, n, kk, v);
}

// The same from torch's layout [cout][cin][3][3], and the bias zero padded to bout channels.
__global__ void conv_weight_prepare_oihw_kernel(const float* __restrict__ w, const float* __restrict__ bias, int cin, int cout, int bn,
                                                float* __restrict__ img, int total, float* __restrict__ bpad, int bout) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < bout) bpad[i] = i < cout ? __ldg(bias + i) : 0.0f;
    if (i >= total) return;
    const int kk = i % CV_CH, n = (i / CV_CH) % bn, block = i / (CV_CH * bn), tap = block % 9, c = block / 9 * CV_CH + kk;
    const float v = n < cout && c < cin ? __ldg(w + ((int64_t)n * cin + c) * 9 + tap) : 0.0f;
    tc_img_store(img + (int64_t)block * (2 * bn * CV_CH), bn, n, kk, v);
}

int conv_status(bool reset) {
    int v = 0;
    if (reset) return cudaMemcpyToSymbol(g_conv_status, &v, sizeof(int)) == cudaSuccess ? SPGT_OK : SPGT_ERR_LAUNCH;
    return cudaMemcpyFromSymbol(&v, g_conv_status, sizeof(int)) == cudaSuccess ? v : SPGT_ERR_LAUNCH;
}

// Output channels per block: the narrowest width that holds them all, because an MMA's time falls with its width.  16 x 106 x 106,
// 128 -> 52 channels: 124 us with 64, 182 with 128, 157 for the implicit GEMM's 64-wide tile; 64 -> 64: 68, 96 and 90.
static int conv_bn(int cout) { return cout <= 48 ? 48 : cout <= 64 ? 64 : 128; }

template <int BN> static int conv_launch(const ConvParams& p, cudaStream_t st) {
    static SmemOptIn configured;
    if (int e = smem_opt_in(conv3x3_kernel<BN>, CvCfg<BN>::BYTES, configured)) return e;
    const int grid = p.n_tiles < num_sms() ? p.n_tiles : num_sms();
    return launch_chained(conv3x3_kernel<BN>, grid, CV_THREADS, CvCfg<BN>::BYTES, st, p);
}

}  // namespace spgt

using namespace spgt;

extern "C" size_t spgt_conv3x3_weight_bytes(int Cin, int Cout) {
    if (Cin <= 0 || Cout <= 0 || Cout > 128) return 0;
    return (size_t)ceil_div(Cin, CV_CH) * 9 * 2 * conv_bn(Cout) * CV_CH * sizeof(float);
}

extern "C" int spgt_conv3x3_weight_prepare(const float* w_kn, int ldw, int Cin, int Cout, void* out, size_t out_bytes, spgt_stream_t stream) {
    if (!w_kn || !out) return SPGT_ERR_NULL;
    const size_t need = spgt_conv3x3_weight_bytes(Cin, Cout);
    if (need == 0 || ldw < Cout) return SPGT_ERR_SHAPE;
    if (out_bytes < need) return SPGT_ERR_WORKSPACE;
    if (!aligned16(out)) return SPGT_ERR_ALIGN;
    const int bn = conv_bn(Cout), total = ceil_div(Cin, CV_CH) * 9 * bn * CV_CH;
    conv_weight_prepare_kernel<<<ceil_div(total, 256), 256, 0, (cudaStream_t)stream>>>(w_kn, ldw, Cin, Cout, bn, (float*)out, total);
    return launch_status();
}

extern "C" int spgt_conv3x3_weight_prepare_oihw(const float* w, const float* bias, int cin, int cout, int Cin, int Cout, void* out, size_t out_bytes,
                                                float* bias_out, spgt_stream_t stream) {
    if (!w || !bias || !out || !bias_out) return SPGT_ERR_NULL;
    const size_t need = spgt_conv3x3_weight_bytes(Cin, Cout);
    if (need == 0 || cin <= 0 || cout <= 0 || cin > Cin || cout > Cout) return SPGT_ERR_SHAPE;
    if (out_bytes < need) return SPGT_ERR_WORKSPACE;
    if (!aligned16(out)) return SPGT_ERR_ALIGN;
    const int bn = conv_bn(Cout), total = ceil_div(Cin, CV_CH) * 9 * bn * CV_CH;
    conv_weight_prepare_oihw_kernel<<<ceil_div(total, 256), 256, 0, (cudaStream_t)stream>>>(w, bias, cin, cout, bn, (float*)out, total, bias_out, Cout);
    return launch_status();
}

extern "C" int spgt_conv3x3_nhwc_fwd(const float* x, int cin_pitch, int cin_off, int Cin, const void* wprep, const float* bias,
                                     float* y, int cout_pitch, int cout_off, int Cout, int B, int Hh, int Ww, int act,
                                     spgt_stream_t stream) {
    if (!x || !wprep || !y) return SPGT_ERR_NULL;
    if (B <= 0 || Hh <= 0 || Ww <= 0 || Cin <= 0 || Cout <= 0 || Cout > 128 || cin_off < 0 || cout_off < 0) return SPGT_ERR_SHAPE;
    if (cin_off + Cin > cin_pitch || cout_off + Cout > cout_pitch || act < 0 || act > 3) return SPGT_ERR_SHAPE;
    if ((Cin & 3) || (cin_off & 3) || (cin_pitch & 3) || (Cout & 3) || (cout_off & 3) || (cout_pitch & 3)) return SPGT_ERR_SHAPE;
    const int64_t rows = (int64_t)B * (Hh + 1), tiles = ceil_div(rows, (int64_t)CV_TY) * ceil_div(Ww, CV_TX);
    if (rows > 0x7fffffffLL - 64 || tiles > 0x7fffffffLL / 2) return SPGT_ERR_SHAPE;      // (rows and tiles are counted in 32 bits)
    if (!aligned16(x) || !aligned16(wprep) || !aligned16(y)) return SPGT_ERR_ALIGN;
    const ConvParams p{x + cin_off, (const float*)wprep, bias, y + cout_off, cin_pitch, Cin, cout_pitch, Cout, B, Hh, Ww, act, ceil_div(Ww, CV_TX), (int)tiles};
    switch (conv_bn(Cout)) {
        case 48: return conv_launch<48>(p, (cudaStream_t)stream);
        case 64: return conv_launch<64>(p, (cudaStream_t)stream);
        default: return conv_launch<128>(p, (cudaStream_t)stream);
    }
}
