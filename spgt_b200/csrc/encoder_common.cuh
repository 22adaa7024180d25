// Shared by the fused encoder kernels (encoder_kv.cu, encoder_fold.cu, encoder_out.cu): how the grid nodes of a batch are cut
// into row tiles, which thread block takes which tiles, and where its partial sums go.
//
// One encoder layer (network/sp_layer.py:94-104 of the reference, drop rates 0), per sample:
//   K, V = LayerNorm(x Wk + bk), LayerNorm(x Wv + bv) per head,  T_h = [pos K_h]^T [pos V_h] / S,
//   y    = x + concat_h([pos q_h] T_h) Wfc + bfc  with  q = x Wq + bq,          out = y + FFN(y).
// q is linear in x, so the attention output is too:  y = x + x M + pos P + c  with, per sample,
//   G_h = T_h Wfc_h (34 x 128),  M = Wq G' (G' = the channel rows of all G_h),  P = sum_h G_h[pos rows],  c = bq G' + bfc.
// Q is therefore never formed and neither are K and V in memory: encoder_kv_kernel reads x and leaves partial sums of T,
// encoder_fold_kernel turns them into M, P, c, encoder_out_kernel reads x again and writes the layer's output.
#pragma once
#include "tc_common.cuh"

namespace spgt {

constexpr int EN_D = 128, EN_DPOS = 2, EN_ROWS = 128;         // width, position values, rows of a tile
constexpr int EN_PAIRS = 2;                                    // head pairs: a block of encoder_kv_kernel works on two of the four heads

// The LayerNorm is applied in three places: the channel means are taken out of Wk, Wv and the biases beforehand, the kernel scales
// every node's 32 channels by 1 / sqrt(mean square + eps), and its weight w and bias b enter when T is put together, from
//   T[c][d] = wk_c wv_d sum k_c v_d + wk_c bv_d sum k_c + bk_c wv_d sum v_d + bk_c bv_d S      (k, v: the scaled values)
// Partial sums of one (sample, head pair, block): products [64 K channels of the pair][32 V channels of the same head]; K, then V
// channels against (pos 0, pos 1, 1) [3][64] each; position products xx, xy, yy and sums x, y.
constexpr int EN_P_CORE = 0, EN_P_K = 2048, EN_P_V = EN_P_K + 192, EN_P_POS = EN_P_V + 192, EN_P_FLOATS = EN_P_POS + 32;

// Work split of encoder_kv_kernel: U = B * tps row tiles per head pair, in order over `per_pair` blocks, the first `more` of which
// take one tile more than the `each` of the others.
struct EncoderSplit {
    int tps, units, per_pair, each, more, max_parts;
    __host__ __device__ int begin(int c) const { return c * each + (c < more ? c : more); }
    __host__ __device__ int owner(int u) const {               // the block that works on tile u
        const int head = more * (each + 1);
        return u < head ? u / (each + 1) : more + (u - head) / each;
    }
};
inline EncoderSplit encoder_split(int B, int S, int sms) {
    EncoderSplit s;
    s.tps = ceil_div(S, EN_ROWS);
    s.units = B * s.tps;
    s.per_pair = sms / EN_PAIRS < s.units ? sms / EN_PAIRS : s.units;
    if (s.per_pair < 1) s.per_pair = 1;
    s.each = s.units / s.per_pair;
    s.more = s.units - s.each * s.per_pair;
    s.max_parts = (s.tps - 1) / s.each + 2;                    // most blocks that can share the tiles of one sample
    if (s.max_parts > s.per_pair) s.max_parts = s.per_pair;
    return s;
}

}  // namespace spgt
