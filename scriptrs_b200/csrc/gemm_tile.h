// Which tile a product of gemm.cu takes.  Host arithmetic only (plain C++, no CUDA types), so that it can be swept over every
// form of a call without a GPU.
#pragma once
#include <stdint.h>

#include <algorithm>

namespace sb {

// kActGlu: the N accumulator columns are groups of 32 = 16 values followed by their 16 gates; the output has N / 2
// columns, out[16 g + i] = v[32 g + i] * sigmoid(v[32 g + 16 + i]) (bf16 output, N % 256 == 0).
enum GemmAct : int { kActNone = 0, kActSilu = 1, kActRelu = 2, kActGlu = 3 };
enum GemmOut : int {
    kOutBf16 = 0,      // out[M x N] bf16 = act(acc * scales + bias)
    kOutF32 = 1,       // out[M x N] f32  = act(acc * scales + bias) * alpha
    kOutResidual = 2,  // out[M x N] f32 += alpha * act(acc * scales + bias)
    kOutFp8 = 3,       // out[M x N] e4m3 = act(acc * scales + bias) / out_row_scale[m]   (N % 256 == 0)
};

// The epilogue's four warps per column half of a tile hand over slabs of so many accumulator columns (128 bytes per output
// row, 64 for a GLU tile whose half is 64 columns); a half is a whole number of slabs.
constexpr int gemm_halves(int bn) { return bn >= 128 ? 2 : 1; }
constexpr int gemm_slab_cols(int act, int out_mode, int half_cols) {
    if (out_mode == kOutFp8) return 128;
    if (act == kActGlu) return half_cols == 64 ? 64 : 128;
    return out_mode == kOutBf16 ? 64 : 32;
}

struct GemmTile {
    int bn;    // columns (128 rows per CTA)
    int ctas;  // 2: a pair of CTAs on 256 x 256
};

// The tile of an M x N x K product (N % 128 == 0; N % 256 == 0 for kOutFp8 and kActGlu).  pair_tiles: 0 never, 1 where it
// pays, 2 every product large enough.
inline GemmTile gemm_tile(int64_t M, int N, int K, bool fp8, int act, int out_mode, int sm_count, int pair_tiles) {
    const int64_t m_tiles = (M + 127) / 128;
    // Two CTAs per 256 x 256 tile when there is at least one such tile per pair of SMs.  Measured in the 8 h encoder
    // step against single-CTA tiles: residual-add products -15 % time (their fp32 epilogue leaves L2 little room
    // for operand traffic), K = 4096 products -9 %, QKV -6 %, the other K = 1024 products unchanged; the K = 256
    // sub-sampling products are 25 % slower (nothing to amortise), so short K stays on single-CTA tiles.
    const bool wide_ok = N % 256 == 0;
    const bool wide = wide_ok && (out_mode == kOutFp8 || act == kActGlu || m_tiles * (N / 256) >= sm_count);
    const int64_t pair_tiles_n = (M + 255) / 256 * (N / 256);
    const bool pair = pair_tiles && wide && pair_tiles_n >= sm_count / 2 && (pair_tiles == 2 || K >= 512);
    if (pair && pair_tiles == 2) return {256, 2};
    // e4m3 rows leave in slabs of 128 columns, which only the halves of a 256-column tile hold, whatever the operands
    if (fp8 || out_mode == kOutFp8) return pair ? GemmTile{256, 2} : GemmTile{wide ? 256 : 128, 1};
    // The tile with the least waves x cost of a 64-wide step of K.  The costs (in 0.01 us) are those of products of one wave,
    // where the ring's depth against the latency of the operands sets the pace: 0.15 us a step at 32 columns, 0.18 at 64,
    // 0.22 at 128, 0.39 at 256 (the tensor core alone: 0.09, 0.10, 0.14, 0.27), 0.37 for a pair's tile.  Measured, us, at 32 / 64 / 128 / 256 columns / pairs:
    // N = K = 1024, fp32 add: M = 188  5.2 / 6.2 / 7.2 / 11.1 / 11.7, M = 752  7.6 / 6.5 / 7.6 / 11.7 / 12.5, M = 4032  19 / 14 / 12.3 / 12.5 / 13.4;
    // N = 1024, K = 4096: M = 188  12.1 / 13.3 / 17.4 / 28.5 / 26.9, M = 1504  28.8 / 22.1 / 17.0 / 27.5 / 27.5, M = 4032  63 / 41 / 31 / 28.6 / 29.1;
    // N = 4096, K = 1024: M = 188  - / 6.7 / 7.8 / 11.4 / 12.1, M = 1504  - / 18.7 / 15.1 / 17.6 / 18.3, M = 52000  - / 544 / 409 / 353 / 312.
    // A bf16 row wants 64 columns for its slab.  Products with short K are bound by their epilogues: widest tile in one wave.
    auto waves = [&](int bn) { return (m_tiles * (N / bn) + sm_count - 1) / sm_count; };
    if (K < 512) {
        if (wide) return {256, 1};
        for (int bn : {64, 128})
            if (waves(bn) == 1) return {bn, 1};
        return {wide_ok ? 256 : 128, 1};
    }
    GemmTile best{0, 1};
    int64_t least = INT64_MAX;
    auto offer = [&](int bn, int ctas, int64_t cost) {
        if (cost < least) { least = cost; best = {bn, ctas}; }
    };
    if (pair) offer(256, 2, (pair_tiles_n + sm_count / 2 - 1) / (sm_count / 2) * 37);
    if (wide_ok) offer(256, 1, waves(256) * 39);
    offer(128, 1, waves(128) * 22);
    offer(64, 1, waves(64) * 18);
    if (out_mode != kOutBf16) offer(32, 1, waves(32) * 15);
    return best;
}

}  // namespace sb
