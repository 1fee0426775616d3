// TDT greedy decoding with the predictor and joint products on the tensor cores (sm_100a): one persistent cooperative kernel
// for a whole batch, of three: at most 16 sequences, some hundred, and more.
//
// The state machine is that of the fp32 kernel in decode.cu (ParakeetModel::greedy_decode and GreedyDecodeState,
// src/model.rs:64-214), and as in the reference the predictor runs only for sequences that emitted a token
// (src/model.rs:136-160): its output stays cached while a sequence walks over blanks.  One iteration:
//   A  W_hh0 h0 (+ the table W_ih0 emb(token) + b, one row per vocabulary entry) -> cell 0 -> h0', c0'
//      W_hh1 h1 -> partial gates of layer 1 (does not need h0', so it shares the phase)
//   B  W_ih1 h0' + partial -> cell 1 -> h1', c1'
//   C  W_pred h1' -> z = relu(enc_proj[frame] + pred)
//   D  W_out z -> logits
//   E  arg-max, confidence, record, commit, advance; lists of the sequences alive and of those that emitted
// with a grid-wide barrier between phases; A to C run over the sequences that emitted and are skipped when there are
// none.  Every product has K = 640.
//
// What bounds it: latency, and with hundreds of sequences the instructions around the products.  A batch of one does 6.0
// million multiply-adds per emitted token and 0.66 per blank, three times over (below), against 24 MB of weights in L2; a step
// is a chain of up to five dependent phases of about a microsecond and as many barriers.  Hence mma.sync and not tcgen05: the
// weight rows are the M side, 16 rows are a tile, and the 444 four-warp groups of the chip share the 40 to 320 tiles of a
// phase (a 128-row tensor-memory tile would leave most SMs idle and its set-up costs more than the product).  A
// group keeps its tile's fragments in registers (80 per thread), over all sequences of the phase and, when a phase
// repeats, over the iterations; the fragments of the phase to come are fetched before the barrier that starts it.
// Against host-stepped tensor-memory GEMMs over a tripled K (eight kernels an iteration, all sequences in every product), the
// loop alone, sequences of 186 frames, ms with blanks in most steps / with an emission in nearly every step: 1 sequence
// 9.4 -> 0.70 / 17.3 -> 2.2, 280 13.1 -> 5.0 / 35 -> 16, 1120 19.1 -> 10.3 / 56 -> 39, 2236 25.9 -> 18.2 / 73 -> 72.
//
// fp32 operands go to the bf16 tensor cores as split sums: x = hi + lo with hi = bf16(x), lo = bf16(x - hi), and
// x . w ~= hi.hi + hi.lo + lo.hi (the dropped term is below 2^-16 of |x||w|), each of the three in an fp32 accumulator of
// its own, K in four parts of 160, one per warp, added in a fixed order: a sequence's numbers do not depend on the batch.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "context.h"
#include "decode.h"
#include "gemm.h"
#include "tc_ptx.cuh"

namespace sb {

namespace {

constexpr int kH = kPredHidden;        // 640
static_assert(kH == 640 && kJointDim == 640, "every product of the loop has K = 640");
constexpr int kGates = 4 * kH;
constexpr int kKB = kH / 32;           // 20 blocks of 32 k values
constexpr int kQuadWarps = 4;          // warps that share a tile's K
constexpr int kWarpKB = kKB / kQuadWarps;
constexpr int kQuads = 3;              // four-warp groups per CTA
constexpr int kDecThreads = kQuads * kQuadWarps * 32;
constexpr int kTileU4 = kKB * 4 * 32;  // uint4 per packed 16-row tile
constexpr int kLstmTiles = kGates / 16, kPredTiles = kJointDim / 16, kOutTiles = (kJointOut + 15) / 16;
constexpr int kOutPad = kOutTiles * 16;  // 1040
constexpr int kPStride = 20;           // floats per column of a partial tile: conflict-free fragment stores

__device__ __forceinline__ void split2(float x, bf16& hi, bf16& lo) {
    hi = __float2bfloat16(x);
    lo = __float2bfloat16(x - __bfloat162float(hi));
}

// ---------------------------------------------------------------- preparation
// dst [rows x 3 cols] = [hi | hi | lo] of src [rows x cols] (activations of the encoder projection).
__global__ void __launch_bounds__(256)
split_act_kernel(const float* __restrict__ src, bf16* __restrict__ dst, int64_t rows, int cols) {
    const int64_t n = rows * cols;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        const int64_t r = i / cols;
        const int c = (int)(i - r * cols);
        bf16 hi, lo;
        split2(src[i], hi, lo);
        bf16* d = dst + r * 3 * cols;
        d[c] = hi;
        d[cols + c] = hi;
        d[2 * cols + c] = lo;
    }
}

// dst [rows x 3 cols] = [hi | lo | hi] of the rows of src (weights of the encoder projection).
__global__ void __launch_bounds__(256)
split_weight_kernel(const float* __restrict__ src, int cols, bf16* __restrict__ dst, int rows) {
    const int64_t n = (int64_t)rows * cols;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        const int r = (int)(i / cols), c = (int)(i % cols);
        bf16 hi, lo;
        split2(src[i], hi, lo);
        bf16* d = dst + (size_t)r * 3 * cols;
        d[c] = hi;
        d[cols + c] = lo;
        d[2 * cols + c] = hi;
    }
}

// Rows of W [rows x 640] in the order of mma.m16n8k16 A fragments: tile, block of 32 k, {hi, hi, lo, lo} of its two MMAs, lane,
// the four registers {row g: k, k + 1; row g + 8: the same; row g: k + 2, k + 3; row g + 8}, k = 8 q (+ 4 for the second MMA; g =
// lane / 4, q = lane % 4), which permutes k inside the block; the activations are read with the same permutation.  An MMA
// takes its four registers as one aligned group, so they are loaded as one: from any other order they are moved there, by
// hundreds of moves an item where the compiler does it at the use.
// LSTM rows are regrouped so that a tile holds the four gates of four units: row 4 unit + gate.
__global__ void __launch_bounds__(128)
pack_fragments_kernel(const float* __restrict__ w, int rows, bool lstm, uint4* __restrict__ dst) {
    const int tile = blockIdx.x, lane = threadIdx.x & 31, part = threadIdx.x >> 5;
    const int g = lane >> 2, q = lane & 3;
    for (int kb = 0; kb < kKB; ++kb) {
        __align__(16) bf16 v[8];
        for (int e = 0; e < 8; ++e) {
            const int r = tile * 16 + g + ((e & 2) ? 8 : 0), k = kb * 32 + 8 * q + 4 * (part & 1) + 2 * (e >> 2) + (e & 1);
            const int src = lstm ? (r & 3) * kH + (r >> 2) : r;
            bf16 hi, lo;
            split2(src < rows ? w[(size_t)src * kH + k] : 0.0f, hi, lo);
            v[e] = part < 2 ? hi : lo;
        }
        dst[(size_t)tile * kTileU4 + (kb * 4 + part) * 32 + lane] = *reinterpret_cast<const uint4*>(v);
    }
}

// table[token][4 unit + gate] = W_ih0 emb(token) + b0, summed in double: the embedding half of the first cell's gates is a
// function of the token alone.  grid (tokens, 10), 256 threads.
__global__ void __launch_bounds__(256)
token_gates_kernel(const float* __restrict__ embedding, const float* __restrict__ w_ih, const float* __restrict__ b,
                   float* __restrict__ table) {
    __shared__ float e[kH];
    const int token = blockIdx.x, row = blockIdx.y * 256 + threadIdx.x;  // row = gate * 640 + unit
    for (int i = threadIdx.x; i < kH; i += 256) e[i] = embedding[(size_t)token * kH + i];
    __syncthreads();
    double acc = (double)b[row];
    const float4* w4 = reinterpret_cast<const float4*>(w_ih + (size_t)row * kH);
    for (int i = 0; i < kH / 4; ++i) {
        const float4 v = w4[i];
        acc += (double)v.x * e[4 * i] + (double)v.y * e[4 * i + 1] + (double)v.z * e[4 * i + 2] + (double)v.w * e[4 * i + 3];
    }
    table[(size_t)token * kGates + 4 * (row % kH) + row / kH] = (float)acc;
}

// Bias of layer 1 in the regrouped order, and the joint output bias padded to whole tiles.
__global__ void bias_kernel(const float* __restrict__ b1, float* __restrict__ b1_out, const float* __restrict__ bo,
                            float* __restrict__ bo_out) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < kGates) b1_out[4 * (i % kH) + i / kH] = b1[i];
    if (i < kOutPad) bo_out[i] = i < kJointOut ? bo[i] : 0.0f;
}

// ---------------------------------------------------------------- the loop
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint4 a, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// Everything that the loop writes is read through L2 (ld.cg): the SMs' L1 caches do not see each other's stores.
struct LoopState {
    DecodeState s;          // outputs, offsets, frame / token / symbol counters; of its float arrays only pred
    DecodeTcWeights w;
    const float* b_pred;
    // Candidate and committed predictor states share two slots per sequence: slot `parity` is committed, the other one takes
    // what the predictor computes from it; emitting a token flips the parity.  [slot][layer][plane hi / lo][n_seq][640]
    bf16* h;
    float* c;               // [slot][layer][n_seq][640]
    bf16* z;                // [n_seq][1280] joint input
    float* part;            // [n_seq][2560] recurrent half of layer 1's gates
    // Every tile of 16 joint outputs leaves {largest token logit, its index, sum of exp(logit - largest)} per sequence; the
    // last tile also leaves its logits (the blank and the durations).  Two sets, used in turn.
    float4* stat;           // [2][n_seq][65]
    float* tail;            // [2][n_seq][16]
    // lists of the step (even / odd): sequences alive, sequences whose predictor must run
    uint32_t *live, *upd;   // [2][n_seq]
    int* counts;            // [3][2]: alive, must run; three sets used in turn
    unsigned* barrier;
    int* error;
};

constexpr uint32_t kSeqMask = 0x1FFFu, kTokenMask = 0x7FFu;  // a list entry: sequence | last token << 13 | parity << 30
constexpr int kTokenShift = 13;

enum { kPhaseA = 0, kPhaseB = 1, kPhaseC = 2, kPhaseD = 3 };

struct Fragments {
    uint4 a[kWarpKB][4];    // {hi, hi, lo, lo} of the two MMAs of this warp's five k blocks
    const uint4* tile;      // what they hold
};

__device__ __forceinline__ const uint4* tile_of(const DecodeTcWeights& w, int phase, int t) {
    if (phase == kPhaseA) return (t < kLstmTiles ? w.hh0 : w.hh1 - (size_t)kLstmTiles * kTileU4) + (size_t)t * kTileU4;
    const uint4* base = phase == kPhaseB ? w.ih1 : (phase == kPhaseC ? w.pred : w.out);
    return base + (size_t)t * kTileU4;
}
__device__ __forceinline__ void fetch_fragments(Fragments& f, const uint4* tile, int qwarp, int lane) {
    if (f.tile == tile) return;
    f.tile = tile;
    const uint4* src = tile + (size_t)qwarp * kWarpKB * 4 * 32 + lane;
#pragma unroll
    for (int kb = 0; kb < kWarpKB; ++kb)
#pragma unroll
        for (int p = 0; p < 4; ++p) f.a[kb][p] = __ldg(src + (kb * 4 + p) * 32);
}

// Activations (hidden vectors, joint inputs) lie in global memory in the order in which a lane needs them: for every block of
// 32 k and every q the eight hi values, then the eight lo values, 32 bytes that one load brings.  A warp's load then takes
// eight whole 128-byte lines; with hi and lo in planes of their own it took half of sixteen (2236 clips 44.1 -> 37.2 ms
// for the whole call, 280 clips 7.4 -> 6.4).
constexpr int kRowElems = 2 * kH;  // bf16 per row
__device__ __forceinline__ int elem_of(int k) { return (k >> 3) * 16 + (k & 7); }  // hi; the lo value is 8 further
struct Pair {
    uint4 hi, lo;
};
// Plain loads, which may hit in L1: the acquire of the grid barrier has discarded what L1 held before.
__device__ __forceinline__ Pair load_pair(const bf16* p) {
    Pair v;
    asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v.hi.x), "=r"(v.hi.y), "=r"(v.hi.z), "=r"(v.hi.w), "=r"(v.lo.x), "=r"(v.lo.y), "=r"(v.lo.z), "=r"(v.lo.w)
                 : "l"(p)
                 : "memory");
    return v;
}
__device__ __forceinline__ Pair load_pair_shared(uint32_t at) {
    Pair v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.hi.x), "=r"(v.hi.y), "=r"(v.hi.z), "=r"(v.hi.w) : "r"(at));
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.lo.x), "=r"(v.lo.y), "=r"(v.lo.z), "=r"(v.lo.w) : "r"(at + 16));
    return v;
}
constexpr int kBlockElems = 4 * 16;  // bf16 from one block of 32 k to the next
__device__ __forceinline__ void load_x(Pair (&x)[kWarpKB], const bf16* p) {
#pragma unroll
    for (int kb = 0; kb < kWarpKB; ++kb) x[kb] = load_pair(p + kb * kBlockElems);
}
// Products of a warp's five k blocks: hi.hi, hi.lo and lo.hi into accumulators of their own.
__device__ __forceinline__ void block_product(const uint4 (&a)[4], const Pair& x, float (&d)[3][4]) {
    mma_bf16(d[0], a[0], x.hi.x, x.hi.y);
    mma_bf16(d[1], a[0], x.lo.x, x.lo.y);
    mma_bf16(d[2], a[2], x.hi.x, x.hi.y);
    mma_bf16(d[0], a[1], x.hi.z, x.hi.w);
    mma_bf16(d[1], a[1], x.lo.z, x.lo.w);
    mma_bf16(d[2], a[3], x.hi.z, x.hi.w);
}
__device__ __forceinline__ void product(const Fragments& f, const Pair (&x)[kWarpKB], float (&v)[4]) {
    float d[3][4] = {};
#pragma unroll
    for (int kb = 0; kb < kWarpKB; ++kb) block_product(f.a[kb], x[kb], d);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = d[0][i] + (d[1][i] + d[2][i]);
}
// The same, refilling each block's registers with the next product's activations as soon as they have been used.
__device__ __forceinline__ void product_refill(const Fragments& f, Pair (&x)[kWarpKB], float (&v)[4], const bf16* next, bool refill) {
    float d[3][4] = {};
#pragma unroll
    for (int kb = 0; kb < kWarpKB; ++kb) {
        block_product(f.a[kb], x[kb], d);
        if (refill) x[kb] = load_pair(next + kb * kBlockElems);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = d[0][i] + (d[1][i] + d[2][i]);
}
// A warp's partial tile (16 rows x 8 columns from column 8 j) -> shared memory, [column][row].
__device__ __forceinline__ void store_partial(float* mine, int j, int lane, const float (&v)[4]) {
    float* o = mine + (8 * j + 2 * (lane & 3)) * kPStride + (lane >> 2);
    o[0] = v[0];
    o[kPStride] = v[1];
    o[8] = v[2];
    o[kPStride + 8] = v[3];
}
__device__ __forceinline__ void quad_barrier(int quad) {
    asm volatile("bar.sync %0, %1;" ::"r"(quad + 1), "r"(kQuadWarps * 32) : "memory");
}
template <int N>
__device__ __forceinline__ float sum_partials(const float (*P)[N], int at) { return (P[0][at] + P[1][at]) + (P[2][at] + P[3][at]); }

__device__ __forceinline__ float logistic(float x) { return 1.0f / (1.0f + expf(-x)); }

// One LSTM unit from its four gate pre-activations (i, f, g, o), in one thread: 64 of a group's 128 threads take the 4 units x
// 16 columns of a tile.  With a gate per lane, logistic function and hyperbolic tangent in neighbouring lanes, every warp went
// through both, and through the cell's own tangent four times over.
__device__ __forceinline__ void cell(float4 v, float c_old, float& cn, float& hn) {
    cn = fmaf(logistic(v.y), c_old, logistic(v.x) * tanhf(v.z));
    hn = logistic(v.w) * tanhf(cn);
}
template <int N>
__device__ __forceinline__ float4 sum_partials4(const float (*P)[N], int at) {
    const float4 a = *reinterpret_cast<const float4*>(&P[0][at]), b = *reinterpret_cast<const float4*>(&P[1][at]);
    const float4 c = *reinterpret_cast<const float4*>(&P[2][at]), d = *reinterpret_cast<const float4*>(&P[3][at]);
    return make_float4((a.x + b.x) + (c.x + d.x), (a.y + b.y) + (c.y + d.y), (a.z + b.z) + (c.z + d.z), (a.w + b.w) + (c.w + d.w));
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
// The same sixteen lanes that hold a column of a joint output tile reduce it (row = lane % 16 of the tile).
__device__ __forceinline__ void tile_stat(float v, int tile, int row, int lane, bool ok, float4* stat, float* tail) {
    float m = row < kVocab ? v : -INFINITY;
    int idx = row;
    const float own = m;
    if (!(m > -INFINITY)) { m = -INFINITY; idx = 0x7fffffff; }  // nothing to compare with (not a number counts in the sum only)
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, m, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > m || (ov == m && oi < idx)) { m = ov; idx = oi; }
    }
    float e = own == -INFINITY ? 0.0f : expf(own - m);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if (!ok) return;
    if ((lane & 15) == 0) __stcg(stat + tile, make_float4(m, __int_as_float(idx), e, 0.0f));
    if (tile == kOutTiles - 1) __stcg(tail + (lane & 15), v);
}

struct Decision {
    int token, dur;
    float conf;
};
// One warp: arg-max over the tiles (ties to the lowest index), confidence = largest softmax, arg-max of the durations.
__device__ __forceinline__ Decision decide_tokens(const float4* stat, const float* tail, int lane) {
    static_assert(kOutTiles == 65 && kVocab == 64 * 16 + 1, "the last tile holds the blank and the durations");
    float4 t[3];
    t[0] = __ldcg(stat + lane);
    t[1] = __ldcg(stat + 32 + lane);
    t[2] = lane == 0 ? __ldcg(stat + 64) : make_float4(-INFINITY, __int_as_float(0x7fffffff), 0.0f, 0.0f);
    float dl[kDurations];
#pragma unroll
    for (int i = 0; i < kDurations; ++i) dl[i] = __ldcg(tail + 1 + i);
    float best = t[0].x;
    int token = __float_as_int(t[0].y);
#pragma unroll
    for (int i = 1; i < 3; ++i)
        if (t[i].x > best) { best = t[i].x; token = __float_as_int(t[i].y); }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, token, o);
        if (ov > best || (ov == best && oi < token)) { best = ov; token = oi; }
    }
    if (token == 0x7fffffff) token = 0;  // not one comparable logit: the first entry, as a scan from entry 0 leaves it
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i)
        if (t[i].z != 0.0f) sum += t[i].z * expf(t[i].x - best);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    int dur = 0;
#pragma unroll
    for (int i = 1; i < kDurations; ++i)
        if (dl[i] > dl[0]) { dl[0] = dl[i]; dur = i; }
    return {token, dur, best > -INFINITY ? 1.0f / sum : NAN};
}
// Frame and symbol counter after a decision (src/model.rs:196-209).
__device__ __forceinline__ void advance(bool emit, int dur, int& frame, int& symbols) {
    symbols += emit ? 1 : 0;
    if (dur > 0) { frame += dur; symbols = 0; }
    else if (!emit || symbols >= kMaxSymbols) { frame += 1; symbols = 0; }
}
__device__ __forceinline__ void record(const DecodeState& s, uint32_t b, int n, const Decision& d, int frame) {
    if (n < s.max_tokens) {
        const size_t o = (size_t)b * s.max_tokens + n;
        s.out_tokens[o] = (uint32_t)d.token;
        s.out_frames[o] = frame;
        s.out_durs[o] = d.dur;
        s.out_conf[o] = d.conf;
    } else {
        atomicExch(s.overflow, 1);
    }
}

// ---------------------------------------------------------------- many sequences
// A phase's work is (tiles x groups of 16 sequences), tile-major; each four-warp group takes a contiguous share of it, so that
// it meets at most two or three tiles.  An item is a chain list entry -> activation rows -> products -> sum over the warps ->
// epilogue of some 4000 cycles; the list entries are read one item ahead and every activation register is refilled for the
// next product as soon as the current one has used it, so that the L2 latencies lie under the MMAs.  Sharing the rows of an
// item among the three groups of a CTA (cp.async or bulk copies into shared memory) takes a third of the L2 traffic but was
// slower, 5.9 and 7.6 ms against 5.0 for 280 clips: the groups then wait for one another.
constexpr int kMaxSeqs = 8192;     // thirteen bits of a list entry

__device__ __forceinline__ constexpr int tiles_of(int phase) {
    return phase == kPhaseA ? 2 * kLstmTiles : (phase == kPhaseB ? kLstmTiles : (phase == kPhaseC ? kPredTiles : kOutTiles));
}
struct Share {
    int begin, end, groups;
};
__device__ __forceinline__ Share share_of(int phase, int n, int quad) {
    const int groups = (n + 15) >> 4;
    const int64_t total = (int64_t)tiles_of(phase) * groups;
    const int shares = gridDim.x * kQuads, me = quad * gridDim.x + blockIdx.x;
    return {(int)(total * me / shares), (int)(total * (me + 1) / shares), groups};
}

// A cell's new state -> the candidate slot of sequence b.
__device__ __forceinline__ void put_cell(const LoopState& L, size_t b, int slot, int layer, int unit, float cn, float hn) {
    bf16 hi, lo;
    split2(hn, hi, lo);
    bf16* h = L.h + ((size_t)(slot * 2 + layer) * L.s.n_seq + b) * kRowElems + elem_of(unit);
    __stcg(L.c + ((size_t)(slot * 2 + layer) * L.s.n_seq + b) * kH + unit, cn);
    h[0] = hi;
    h[8] = lo;
}

template <int PHASE>
__device__ __forceinline__ void run_phase(const LoopState& L, Fragments& f, const uint32_t* list, int n, int quad, int qwarp, int lane,
                                          float (*sm)[kQuadWarps][16 * kPStride], size_t set = 0) {
    const DecodeState& s = L.s;
    const Share sh = share_of(PHASE, n, quad);
    if (sh.begin >= sh.end) return;
    const size_t BH = (size_t)s.n_seq * kH;
    const int g = lane >> 2, q = lane & 3, qt = qwarp * 32 + lane, r16 = qt & 15;
    // activation row of a list entry (this lane's part of it)
    auto row_of = [&](uint32_t e, int tile) -> const bf16* {
        const size_t b = e & kSeqMask;
        const bf16* r;
        if (PHASE == kPhaseD) {
            r = L.z + b * kRowElems;
        } else {
            const int slot = (int)(e >> 30) ^ (PHASE == kPhaseA ? 0 : 1);
            const int layer = PHASE == kPhaseA ? (tile >= kLstmTiles ? 1 : 0) : (PHASE == kPhaseB ? 0 : 1);
            r = L.h + ((size_t)(slot * 2 + layer) * s.n_seq + b) * kRowElems;
        }
        return r + qwarp * kWarpKB * kBlockElems + q * 16;
    };
    int tile = sh.begin / sh.groups, n0 = (sh.begin - tile * sh.groups) * 16;
    // a column beyond the list repeats the last one and is not stored
    uint32_t e0 = __ldcg(list + min(n0 + g, n - 1)), e1 = __ldcg(list + min(n0 + 8 + g, n - 1));
    fetch_fragments(f, tile_of(L.w, PHASE, tile), qwarp, lane);
    Pair x[kWarpKB];
    load_x(x, row_of(e0, tile));
    for (int item = sh.begin; item < sh.end; ++item) {
        const bool rec = PHASE == kPhaseA && tile >= kLstmTiles;  // the recurrent half of layer 1
        const bool two = n - n0 > 8, more = item + 1 < sh.end;
        const int row = tile * 16 + r16;
        int next_tile = tile, next_n0 = n0 + 16;
        if (next_n0 >= n) { next_n0 = 0; ++next_tile; }
        uint32_t f0 = 0, f1 = 0;
        if (more) {
            f0 = __ldcg(list + min(next_n0 + g, n - 1));
            f1 = __ldcg(list + min(next_n0 + 8 + g, n - 1));
        }
        // What the epilogue adds is fetched under the product.  Cells: threads of two of the four warps, by turns, finish unit
        // qt % 4 of column (qt / 4) % 16, which is the column of one of their own list entries; other phases: thread qt
        // finishes row qt % 16 of columns qt / 16 (+ 8).
        const bool cells = PHASE == kPhaseB || (PHASE == kPhaseA && !rec);
        const bool cell_warp = cells && (qwarp >> 1) == (item & 1);
        const uint32_t ec = (qwarp & 1) ? e1 : e0;
        const int unit = tile * 4 + (lane & 3);
        float4 gates = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float c_cell = 0.0f;
        if (cell_warp) {
            const size_t b = ec & kSeqMask;
            if (PHASE == kPhaseA) {
                gates = __ldg(reinterpret_cast<const float4*>(L.w.token_gates + (size_t)((ec >> kTokenShift) & kTokenMask) * kGates) + unit);
                c_cell = __ldcg(L.c + (size_t)((ec >> 30) * 2) * BH + b * kH + unit);
            } else {
                gates = add4(__ldcg(reinterpret_cast<const float4*>(L.part + b * kGates) + unit), __ldg(reinterpret_cast<const float4*>(L.w.b1) + unit));
                c_cell = __ldcg(L.c + (size_t)((ec >> 30) * 2 + 1) * BH + b * kH + unit);
            }
        }
        uint32_t e[2];
        float add[2], c_old[2];
        if (!cells) {
            e[0] = __shfl_sync(0xffffffffu, e0, 4 * (qt >> 4));
            e[1] = __shfl_sync(0xffffffffu, e1, 4 * (qt >> 4));
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const size_t b = e[j] & kSeqMask;
                add[j] = c_old[j] = 0.0f;
                if (PHASE == kPhaseC) {
                    add[j] = __ldg(L.b_pred + row);
                    c_old[j] = __ldg(s.enc_proj + (size_t)(s.enc_off[b] + __ldcg(s.frame_idx + b)) * kJointDim + row);
                } else if (PHASE == kPhaseD) {
                    add[j] = __ldg(L.w.b_out + row);
                }
            }
        }
        float v0[4], v1[4];
        product_refill(f, x, v0, row_of(e1, tile), two);
        if (two) product_refill(f, x, v1, row_of(f0, next_tile), more);
        else if (more) load_x(x, row_of(f0, next_tile));
        float (*P)[16 * kPStride] = sm[(item - sh.begin) & 1];
        store_partial(P[qwarp], 0, lane, v0);
        if (two) store_partial(P[qwarp], 1, lane, v1);
        if (more && next_tile != tile) fetch_fragments(f, tile_of(L.w, PHASE, next_tile), qwarp, lane);
        quad_barrier(quad);  // also: the other buffer's readers are done
        if (cells) {
            const int col = (qt >> 2) & 15;
            if (cell_warp && n0 + col < n) {
                constexpr int layer = PHASE == kPhaseB ? 1 : 0;
                float cn, hn;
                cell(add4(sum_partials4(P, col * kPStride + 4 * (lane & 3)), gates), c_cell, cn, hn);
                put_cell(L, ec & kSeqMask, (int)(ec >> 30) ^ 1, layer, unit, cn, hn);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (j && !two) break;
                const float val = sum_partials(P, ((qt >> 4) + 8 * j) * kPStride + r16) + add[j];
                const size_t b = e[j] & kSeqMask;
                const bool ok = n0 + (qt >> 4) + 8 * j < n;
                if (PHASE == kPhaseA) {
                    if (ok) __stcg(L.part + b * kGates + (row - kGates), val);
                } else if (PHASE == kPhaseC) {
                    if (ok) {
                        bf16 hi, lo;
                        split2(fmaxf(c_old[j] + val, 0.0f), hi, lo);
                        __stcg(s.pred + b * kJointDim + row, val);
                        L.z[b * kRowElems + elem_of(row)] = hi;
                        L.z[b * kRowElems + elem_of(row) + 8] = lo;
                    }
                } else {
                    tile_stat(val, tile, row, lane, ok, L.stat + (set * s.n_seq + b) * kOutTiles, L.tail + (set * s.n_seq + b) * 16);
                    if (ok && s.trace && row < kJointOut) {
                        const int nsteps = __ldcg(s.n_steps + b);
                        if (nsteps < s.trace_cap) s.trace[(b * s.trace_cap + nsteps) * kJointOut + row] = val;
                    }
                }
            }
        }
        e0 = f0;
        e1 = f1;
        tile = next_tile;
        n0 = next_n0;
    }
}

// One warp per sequence: arg-max, confidence, record, commit, advance (src/model.rs:79-90,180-209), the joint input of
// the next frame where the predictor output stays valid, and the lists of the next step.
__device__ __forceinline__ void decide(const LoopState& L, uint32_t entry, int lane, size_t set, uint32_t* next_live, uint32_t* next_upd,
                                       int* next_counts) {
    const DecodeState& s = L.s;
    const uint32_t b = entry & kSeqMask;
    const int frame = __ldcg(s.frame_idx + b), len = s.enc_len[b];
    const int nsteps = __ldcg(s.n_steps + b), n_tokens = __ldcg(s.n_tokens + b);
    int symbols = __ldcg(s.emitted + b);
    const Decision d = decide_tokens(L.stat + (set * s.n_seq + b) * kOutTiles, L.tail + (set * s.n_seq + b) * 16, lane);
    const bool emit = d.token != kVocab - 1;
    int nf = frame;
    advance(emit, d.dur, nf, symbols);
    if (!emit && nf < len) {
        // the cached predictor output stays valid: joint input of the new frame
        const float4* en = reinterpret_cast<const float4*>(s.enc_proj + (size_t)(s.enc_off[b] + nf) * kJointDim);
        const float4* pr = reinterpret_cast<const float4*>(s.pred + (size_t)b * kJointDim);
#pragma unroll
        for (int i = 0; i < kJointDim / 128; ++i) {
            const float4 x = __ldg(en + lane + 32 * i), p = __ldcg(pr + lane + 32 * i);
            const float zv[4] = {fmaxf(x.x + p.x, 0.0f), fmaxf(x.y + p.y, 0.0f), fmaxf(x.z + p.z, 0.0f), fmaxf(x.w + p.w, 0.0f)};
            __align__(8) bf16 hi[4], lo[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) split2(zv[e], hi[e], lo[e]);
            bf16* zo = L.z + (size_t)b * kRowElems + elem_of(4 * (lane + 32 * i));
            *reinterpret_cast<uint2*>(zo) = *reinterpret_cast<const uint2*>(hi);
            *reinterpret_cast<uint2*>(zo + 8) = *reinterpret_cast<const uint2*>(lo);
        }
    }
    if (lane == 0) {
        // committing the state that produced the token (src/model.rs:188-189) is the flip of the parity
        const uint32_t next = emit ? ((entry ^ (1u << 30)) & ~(kTokenMask << kTokenShift)) | ((uint32_t)d.token << kTokenShift) : entry;
        if (emit) {
            record(s, b, n_tokens, d, frame);
            s.n_tokens[b] = n_tokens + 1;
        }
        s.frame_idx[b] = nf;
        s.emitted[b] = symbols;
        s.n_steps[b] = nsteps + 1;
        if (nf < len) {
            // the order of a list does not matter: the columns of a product are independent
            next_live[atomicAdd(next_counts, 1)] = next;
            if (emit) next_upd[atomicAdd(next_counts + 1, 1)] = next;
        }
    }
}

// Grid-wide barrier over co-resident CTAs (cooperative launch).  The wait is bounded: when it runs out the kernel raises
// *error and leaves; the other CTAs then run out of time too.
struct GridBarrier {
    unsigned* counter;
    int* error;
    int* gave_up;  // shared memory
    unsigned target = 0;
    __device__ __forceinline__ GridBarrier(const LoopState& L, int* flag) : counter(L.barrier), error(L.error), gave_up(flag) {
        if (threadIdx.x == 0) *gave_up = 0;
    }
    // aborted (shared memory): set by a thread of this CTA whose wait ran out
    __device__ __forceinline__ bool sync(volatile int* aborted = nullptr) {
        target += gridDim.x;
        __syncthreads();
        if (threadIdx.x == 0 && aborted && *aborted) {
            atomicExch(error, 1);
            *gave_up = 1;
        } else if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
            unsigned seen;
            const long long t0 = clock64();
            while (true) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
                if (seen >= target) break;
                if (clock64() - t0 > 4000000000LL) {
                    atomicExch(error, 1);
                    *gave_up = 1;
                    break;
                }
            }
        }
        __syncthreads();
        return *gave_up == 0;
    }
};

__global__ void __launch_bounds__(kDecThreads, 1)
tdt_decode_tc_kernel(const __grid_constant__ LoopState L, int max_steps) {
    __shared__ __align__(16) float P[kQuads][2][kQuadWarps][16 * kPStride];
    __shared__ int gave_up;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, quad = warp / kQuadWarps, qwarp = warp % kQuadWarps;
    const int n_seq = L.s.n_seq;
    GridBarrier grid(L, &gave_up);
    Fragments f;
    f.tile = nullptr;
    auto fetch_ahead = [&](int phase, int n) {
        const Share sh = share_of(phase, n, quad);
        if (sh.begin < sh.end) fetch_fragments(f, tile_of(L.w, phase, sh.begin / sh.groups), qwarp, lane);
    };
    for (int step = 0; step < max_steps; ++step) {
        const uint32_t* live = L.live + (size_t)(step & 1) * n_seq;
        const uint32_t* upd = L.upd + (size_t)(step & 1) * n_seq;
        const int2 n = __ldcg(reinterpret_cast<const int2*>(L.counts) + step % 3);  // {alive, predictor must run}
        if (n.x == 0) break;
        if (n.y > 0) {
            run_phase<kPhaseA>(L, f, upd, n.y, quad, qwarp, lane, P[quad]);
            fetch_ahead(kPhaseB, n.y);
            if (!grid.sync()) return;
            run_phase<kPhaseB>(L, f, upd, n.y, quad, qwarp, lane, P[quad]);
            fetch_ahead(kPhaseC, n.y);
            if (!grid.sync()) return;
            run_phase<kPhaseC>(L, f, upd, n.y, quad, qwarp, lane, P[quad]);
            fetch_ahead(kPhaseD, n.x);
            if (!grid.sync()) return;
        }
        run_phase<kPhaseD>(L, f, live, n.x, quad, qwarp, lane, P[quad], step & 1);
        // the counters of the step after the next were last read when this step's predecessor began
        if (blockIdx.x == 0 && tid == 0) __stcg(reinterpret_cast<int2*>(L.counts) + (step + 2) % 3, make_int2(0, 0));
        if (!grid.sync()) return;
        uint32_t* next_live = L.live + (size_t)((step + 1) & 1) * n_seq;
        uint32_t* next_upd = L.upd + (size_t)((step + 1) & 1) * n_seq;
        int* next_counts = L.counts + 2 * ((step + 1) % 3);
        for (int i = warp * gridDim.x + blockIdx.x; i < n.x; i += gridDim.x * (kDecThreads / 32))
            decide(L, __ldcg(live + i), lane, step & 1, next_live, next_upd, next_counts);
        if (!grid.sync()) return;
    }
}

// ---------------------------------------------------------------- very many sequences
// Above, every group reads a phase's activations for its own tile, 585 times an iteration in all, and a warp does six MMAs for
// the 32 bytes a lane that it has loaded.  Here two groups of four warps have the registers for two tiles each: a CTA runs 64
// rows over the same columns, whose activations come once, by cp.async, into a ring of four places of 16 columns in shared memory,
// two to three items ahead; each read of it feeds twelve MMAs.  What bounds it: an item of 64 rows x 16 columns takes some 3400
// cycles where its MMAs alone take 2030 (8 cycles each and partition), because every other instruction on a partition costs
// its MMAs about two cycles; a second group for the epilogues changes nothing.  The loop alone against the kernel above, ms
// with blanks in most steps / with an emission in nearly every step: 280 sequences 5.2 / 16.3 against 5.0 / 16.1, 400 5.7 / 19.4
// against 5.9 / 20.1, 1120 10.3 / 39 against 11.5 / 44, 2236 18.2 / 72 against 20.4 / 81: the line lies between the first two.
// (At 2236, all with an emission in nearly every step: weights of 64 rows in shared memory and activations in registers 76; this
// layout with the copies and epilogues in the product groups 101; four such groups of one tile each 105.)  The sums are those of the other kernels, term by term: a sequence's numbers do not depend on the
// kernel that its batch took.
constexpr int kWideSeqs = 384;  // the smallest batch of this kernel
constexpr int kWideQuads = 2, kWideThreads = (kWideQuads + 1) * kQuadWarps * 32;
constexpr int kWideTiles = 2 * kWideQuads;       // tiles of a CTA's block
constexpr int kRing = 4;                         // places of 16 columns
constexpr int kRowBytes = 2 * kRowElems;
constexpr int kRowPitch = kRowBytes + 16;        // a quarter-warp's reads (two columns x four pieces) on distinct banks
constexpr int kSlotBytes = 16 * kRowPitch;
constexpr int kWidePart = 2 * 16 * kPStride;     // floats of partial sums per warp
constexpr size_t kWideSmem = (size_t)kRing * kSlotBytes + sizeof(float) * 2 * kWideQuads * kQuadWarps * kWidePart;
static_assert(kLstmTiles % kWideTiles == 0, "a block of phase A belongs to one layer");
static_assert(kSlotBytes % 128 == 0, "places begin on whole lines");

// The CTA's share of a phase: items (block of tiles x group of 16 columns), block-major.  With two CTAs or more for every block a
// share stays inside one, whose weights are then loaded once; the block of the first item depends on the phase alone.
struct WideShare {
    int begin, end, groups;
};
__device__ __forceinline__ int wide_blocks(int phase) { return (tiles_of(phase) + kWideTiles - 1) / kWideTiles; }
__device__ __forceinline__ int wide_first_block(int phase) { return wide_blocks(phase) * blockIdx.x / gridDim.x; }
__device__ __forceinline__ WideShare wide_share(int phase, int n) {
    const int groups = (n + 15) >> 4, blocks = wide_blocks(phase), grid = gridDim.x, cta = blockIdx.x;
    if (2 * blocks > grid) return {blocks * groups * cta / grid, blocks * groups * (cta + 1) / grid, groups};
    const int block = wide_first_block(phase);
    const int first = (block * grid + blocks - 1) / blocks, count = ((block + 1) * grid + blocks - 1) / blocks - first;
    return {block * groups + groups * (cta - first) / count, block * groups + groups * (cta - first + 1) / count, groups};
}

// What tile_stat makes of a tile's column (lane % 16), by two lanes: lane / 16 takes the rows of that parity.  The same
// comparisons, and the sum in the order of tile_stat's exchanges, whose last one is between the parities.
template <int N>
__device__ __forceinline__ void column_stat(const LoopState& L, const float (*P)[N], int at, int tile, int lane, bool ok, size_t b, size_t set) {
    const DecodeState& s = L.s;
    const int odd = lane >> 4, rows = kVocab - tile * 16;  // tokens of this tile, if fewer than 16
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = sum_partials(P, at + 2 * q + odd) + __ldg(L.w.b_out + tile * 16 + 2 * q + odd);
    float m = -INFINITY;
    int idx = 0x7fffffff;
#pragma unroll
    for (int q = 0; q < 8; ++q)
        if (2 * q + odd < rows && v[q] > m) { m = v[q]; idx = tile * 16 + 2 * q + odd; }
    const float om = __shfl_xor_sync(0xffffffffu, m, 16);
    const int oi = __shfl_xor_sync(0xffffffffu, idx, 16);
    if (om > m || (om == m && oi < idx)) { m = om; idx = oi; }
    float e[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) e[q] = 2 * q + odd >= rows || v[q] == -INFINITY ? 0.0f : expf(v[q] - m);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < o; ++q) e[q] += e[q + o];
    e[0] += __shfl_xor_sync(0xffffffffu, e[0], 16);
    if (!ok) return;
    if (!odd) __stcg(L.stat + (set * s.n_seq + b) * kOutTiles + tile, make_float4(m, __int_as_float(idx), e[0], 0.0f));
    if (tile == kOutTiles - 1) {
#pragma unroll
        for (int q = 0; q < 8; ++q) __stcg(L.tail + (set * s.n_seq + b) * 16 + 2 * q + odd, v[q]);
    }
    const int nsteps = s.trace ? __ldcg(s.n_steps + b) : 0;
    if (s.trace && nsteps < s.trace_cap) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (tile * 16 + 2 * q + odd < kJointOut) s.trace[(b * s.trace_cap + nsteps) * kJointOut + tile * 16 + 2 * q + odd] = v[q];
    }
}

// Roles: two groups of four warps form products and do nothing else, so that the tensor cores do not wait for list entries, gates
// and cells; a third group copies the activations in and finishes what the first two have summed, one item behind them.
constexpr int kProductRegs = 208, kFinishRegs = 88;
static_assert(128 * (2 * kProductRegs + kFinishRegs) <= kWideThreads * 168, "the block is launched with 168 registers a thread");

struct WideState {
    unsigned taken;                    // items that have gone through since the kernel began
    uint32_t ring, full, done, freed;  // shared-memory addresses: places; barriers: place filled, sums stored, sums read
    float (*parts)[kWidePart];         // [2][kWideQuads][kQuadWarps] partial sums
    volatile int* abort_flag;
};
struct WideWeights {
    uint4 a[2][kWarpKB][4];  // a warp's quarter of K of its group's two tiles
    int holds;               // phase and block that they belong to
};

__device__ __forceinline__ void wide_weights(WideWeights& W, const DecodeTcWeights& w, int phase, int block, int quad, int qwarp, int lane) {
    if (W.holds == (phase << 16 | block)) return;
    W.holds = phase << 16 | block;
#pragma unroll
    for (int t = 0; t < 2; ++t) {
        // a tile beyond the last repeats it; nothing reads its products
        const uint4* src = tile_of(w, phase, min(block * kWideTiles + 2 * quad + t, tiles_of(phase) - 1)) + (size_t)qwarp * kWarpKB * 4 * 32 + lane;
#pragma unroll
        for (int i = 0; i < kWarpKB * 4; ++i) W.a[t][i / 4][i % 4] = __ldg(src + i * 32);
    }
}

// Products of the CTA's items of a phase.  A wait that ran out is passed over like one that ended: the sums are garbage, every
// further wait ends at once, and the barrier behind the phase ends the kernel.
__device__ __forceinline__ void wide_products(const LoopState& L, WideState& S, WideWeights& W, int phase, int n, int quad, int qwarp, int lane) {
    const WideShare sh = wide_share(phase, n);
    const int items = sh.end - sh.begin;
    if (items <= 0) return;
    int block = sh.begin / sh.groups, group = sh.begin - block * sh.groups;
    const uint32_t at = S.ring + (lane >> 2) * kRowPitch + qwarp * kWarpKB * 128 + (lane & 3) * 32;
    for (int k = 0; k < items; ++k) {
        wide_weights(W, L.w, phase, block, quad, qwarp, lane);
        const unsigned use = S.taken + k;
        ptx::mbar_wait(S.full + 8 * (use % kRing), (use / kRing) & 1, S.abort_flag);
        const uint32_t row = at + use % kRing * kSlotBytes;
        float* mine = S.parts[((use & 1) * kWideQuads + quad) * kQuadWarps + qwarp];
        Pair x = load_pair_shared(row);
        float d[2][3][4];
#pragma unroll
        for (int i = 0; i < 2 * kWarpKB; ++i) {
            const int j = i / kWarpKB, kb = i % kWarpKB;
            Pair y;
            if (i + 1 < 2 * kWarpKB) y = load_pair_shared(row + (i + 1) / kWarpKB * 8 * kRowPitch + (i + 1) % kWarpKB * 128);
            if (kb == 0) {
#pragma unroll
                for (int q = 0; q < 24; ++q) d[q / 12][q / 4 % 3][q % 4] = 0.0f;
            }
            block_product(W.a[0][kb], x, d[0]);
            block_product(W.a[1][kb], x, d[1]);
            if (i + 1 < 2 * kWarpKB) x = y;
            if (kb == kWarpKB - 1) {
                if (j == 0 && use >= 2) ptx::mbar_wait(S.freed + 8 * (use & 1), (use / 2 + 1) & 1, S.abort_flag);
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    float v[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) v[q] = d[t][0][q] + (d[t][1][q] + d[t][2][q]);
                    store_partial(mine + t * 16 * kPStride, j, lane, v);
                }
            }
        }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(S.done + 8 * (use & 1));
        if (++group == sh.groups) { group = 0; ++block; }
    }
    S.taken += items;
}

// The rest of a phase, by 128 threads: copies and epilogues.
template <int PHASE>
__device__ __forceinline__ void wide_finish(const LoopState& L, WideState& S, const uint32_t* list, int n, int qt, size_t set) {
    const DecodeState& s = L.s;
    const WideShare sh = wide_share(PHASE, n);
    const int items = sh.end - sh.begin;
    if (items <= 0) return;
    const size_t BH = (size_t)s.n_seq * kH;
    const int lane = qt & 31, warp = qt >> 5, r16 = qt & 15;
    auto is_rec = [&](int block) { return PHASE == kPhaseA && block * kWideTiles >= kLstmTiles; };  // the recurrent half of layer 1
    // ---- the copies: eight threads per column.  Place of item k: (taken + k) % kRing; it is free when item k - kRing has been
    // multiplied, which this group has seen one item earlier.
    int ci = 0, cblock = sh.begin / sh.groups, cgroup = sh.begin - cblock * sh.groups;  // the item to copy next
    uint32_t ce = 0;                                                                    // its list entry of this thread's column
    auto copy_entry = [&]() { ce = ci < items ? __ldcg(list + min(cgroup * 16 + (qt >> 3), n - 1)) : 0; };
    auto copy = [&]() {
        if (ci >= items) return;
        const uint32_t place = (S.taken + ci) % kRing;
        const size_t b = ce & kSeqMask;
        const bf16* src;
        if (PHASE == kPhaseD) {
            src = L.z + b * kRowElems;
        } else {
            const int slot = (int)(ce >> 30) ^ (PHASE == kPhaseA ? 0 : 1);
            const int layer = PHASE == kPhaseA ? (is_rec(cblock) ? 1 : 0) : (PHASE == kPhaseB ? 0 : 1);
            src = L.h + ((size_t)(slot * 2 + layer) * s.n_seq + b) * kRowElems;
        }
        src += (qt & 7) * 8;
        const uint32_t dst = S.ring + place * kSlotBytes + (qt >> 3) * kRowPitch + (qt & 7) * 16;
#pragma unroll
        for (int i = 0; i < kRowBytes / 128; ++i)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 128 * i), "l"(src + 64 * i) : "memory");
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(S.full + 8 * place) : "memory");
        ++ci;
        if (++cgroup == sh.groups) { cgroup = 0; ++cblock; }
        copy_entry();
    };
    copy_entry();
    for (int i = 0; i < kRing - 1; ++i) copy();
    // ---- the epilogues.  Cells: two units of column (qt / 4) % 16; logits: a tile's column; else row qt % 16 of columns qt / 16
    // (+ 8) of all tiles.
    int block = sh.begin / sh.groups, group = sh.begin - block * sh.groups;
    auto entry = [&](int blk, int grp, int j) {
        const bool cells = PHASE == kPhaseB || (PHASE == kPhaseA && !is_rec(blk));
        const int col = cells ? (qt >> 2) & 15 : (PHASE == kPhaseD ? lane & 15 : (qt >> 4) + 8 * j);
        return __ldcg(list + min(grp * 16 + col, n - 1));
    };
    // what an item's sums are added to is fetched one item ahead, its list entries two
    struct Ahead {
        float4 gates[2];
        float c[2];
        int enc_row[2];
    };
    auto ahead = [&](Ahead& to, int blk, const uint32_t (&en)[2]) {
        if (PHASE == kPhaseB || (PHASE == kPhaseA && !is_rec(blk))) {
            const size_t b = en[0] & kSeqMask;
            constexpr int layer = PHASE == kPhaseB ? 1 : 0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int unit = (blk * kWideTiles + 2 * h + (qt >> 6)) * 4 + (qt & 3);
                if (PHASE == kPhaseA)
                    to.gates[h] = __ldg(reinterpret_cast<const float4*>(L.w.token_gates + (size_t)((en[0] >> kTokenShift) & kTokenMask) * kGates) + unit);
                else
                    to.gates[h] = __ldcg(reinterpret_cast<const float4*>(L.part + b * kGates) + unit);
                to.c[h] = __ldcg(L.c + (size_t)((en[0] >> 30) * 2 + layer) * BH + b * kH + unit);
            }
        } else if (PHASE == kPhaseC) {
#pragma unroll
            for (int j = 0; j < 2; ++j) to.enc_row[j] = s.enc_off[en[j] & kSeqMask] + __ldcg(s.frame_idx + (en[j] & kSeqMask));
        }
    };
    uint32_t e[2] = {entry(block, group, 0), entry(block, group, 1)}, f[2] = {0, 0};
    int next_block = block, next_group = group;
    auto next = [&]() {
        if (++next_group == sh.groups) { next_group = 0; ++next_block; }
    };
    next();
    if (items > 1) {
        f[0] = entry(next_block, next_group, 0);
        f[1] = entry(next_block, next_group, 1);
    }
    Ahead now, later;
    ahead(now, block, e);
    for (int k = 0; k < items; ++k) {
        const bool cells = PHASE == kPhaseB || (PHASE == kPhaseA && !is_rec(block));
        const int tile0 = block * kWideTiles, n0 = group * 16;
        copy();
        block = next_block;
        group = next_group;
        if (k + 1 < items) ahead(later, next_block, f);
        next();
        uint32_t after[2] = {0, 0};
        if (k + 2 < items) {
            after[0] = entry(next_block, next_group, 0);
            after[1] = entry(next_block, next_group, 1);
        }
        const unsigned use = S.taken + k;
        const uint32_t done = S.done + 8 * (use & 1);
        const uint32_t done_phase = (use / 2) & 1;
        float (*P)[kWidePart] = S.parts + (use & 1) * kWideQuads * kQuadWarps;
        const size_t b0 = e[0] & kSeqMask;
        if (cells) {
            const int from = (int)(e[0] >> 30), col = (qt >> 2) & 15;
            constexpr int layer = PHASE == kPhaseB ? 1 : 0;
            ptx::mbar_wait(done, done_phase, S.abort_flag);
            float4 g[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) g[h] = sum_partials4(P + h * kQuadWarps, ((qt >> 6) * 16 + col) * kPStride + 4 * (qt & 3));
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(S.freed + 8 * (use & 1));
            if (n0 + col < n) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int unit = (tile0 + 2 * h + (qt >> 6)) * 4 + (qt & 3);
                    if (PHASE == kPhaseB) now.gates[h] = add4(now.gates[h], __ldg(reinterpret_cast<const float4*>(L.w.b1) + unit));
                    float cn, hn;
                    cell(add4(g[h], now.gates[h]), now.c[h], cn, hn);
                    put_cell(L, b0, from ^ 1, layer, unit, cn, hn);
                }
            }
        } else if (PHASE == kPhaseD) {
            ptx::mbar_wait(done, done_phase, S.abort_flag);
            if (tile0 + warp < kOutTiles)
                column_stat(L, P + (warp >> 1) * kQuadWarps, ((warp & 1) * 16 + (lane & 15)) * kPStride, tile0 + warp, lane, n0 + (lane & 15) < n, b0, set);
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(S.freed + 8 * (use & 1));
        } else {
            float enc[2][kWideTiles];
            if (PHASE == kPhaseC) {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const float* er = s.enc_proj + (size_t)now.enc_row[j] * kJointDim + tile0 * 16 + r16;
#pragma unroll
                    for (int t = 0; t < kWideTiles; ++t) enc[j][t] = __ldg(er + 16 * t);
                }
            }
            ptx::mbar_wait(done, done_phase, S.abort_flag);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int col = (qt >> 4) + 8 * j;
                const size_t b = e[j] & kSeqMask;
                if (n0 + col >= n) continue;
#pragma unroll
                for (int t = 0; t < kWideTiles; ++t) {
                    const int r = (tile0 + t) * 16 + r16;
                    float val = sum_partials(P + (t >> 1) * kQuadWarps, ((t & 1) * 16 + col) * kPStride + r16);
                    if (PHASE == kPhaseA) {
                        __stcg(L.part + b * kGates + (r - kGates), val);
                    } else {
                        val += __ldg(L.b_pred + r);
                        bf16 hi, lo;
                        split2(fmaxf(enc[j][t] + val, 0.0f), hi, lo);
                        __stcg(s.pred + b * kJointDim + r, val);
                        L.z[b * kRowElems + elem_of(r)] = hi;
                        L.z[b * kRowElems + elem_of(r) + 8] = lo;
                    }
                }
            }
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(S.freed + 8 * (use & 1));
        }
        e[0] = f[0];
        e[1] = f[1];
        f[0] = after[0];
        f[1] = after[1];
        now = later;
    }
    S.taken += items;
}

__global__ void __launch_bounds__(kWideThreads, 1)
tdt_decode_wide_kernel(const __grid_constant__ LoopState L, int max_steps) {
    extern __shared__ __align__(128) unsigned char wide_dyn[];
    __shared__ __align__(8) uint64_t bars[kRing + 4];
    __shared__ int gave_up, abort_flag;
    const int tid = threadIdx.x, lane = tid & 31, warp = ptx::warp_index(), quad = warp / kQuadWarps, qwarp = warp % kQuadWarps;
    WideState S;
    S.taken = 0;
    S.ring = ptx::smem_u32(wide_dyn);
    S.full = ptx::smem_u32(bars);
    S.done = S.full + 8 * kRing;
    S.freed = S.done + 16;
    S.parts = reinterpret_cast<float (*)[kWidePart]>(wide_dyn + kRing * kSlotBytes);
    S.abort_flag = &abort_flag;
    if (tid == 0) {
        abort_flag = 0;
        for (int i = 0; i < kRing; ++i) ptx::mbar_init(S.full + 8 * i, 128);
        for (int i = 0; i < 2; ++i) {
            ptx::mbar_init(S.done + 8 * i, kWideQuads * kQuadWarps);
            ptx::mbar_init(S.freed + 8 * i, kQuadWarps);
        }
    }
    GridBarrier grid(L, &gave_up);
    auto sync = [&]() { return grid.sync(&abort_flag); };
    auto counts = [&](int step) { return __ldcg(reinterpret_cast<const int2*>(L.counts) + step % 3); };  // {alive, predictor must run}
    __syncthreads();
    if (quad < kWideQuads) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kProductRegs));
        WideWeights W;
        W.holds = -1;
        auto weights = [&](int phase) { wide_weights(W, L.w, phase, wide_first_block(phase), quad, qwarp, lane); };
        for (int step = 0; step < max_steps; ++step) {
            const int2 n = counts(step);
            if (n.x == 0) break;
            const int phases = n.y > 0 ? 4 : 1;
            bool ok = true;
            for (int p = 4 - phases; p < 4 && ok; ++p) {
                wide_products(L, S, W, p, p == kPhaseD ? n.x : n.y, quad, qwarp, lane);
                if (p != kPhaseD || n.y > 0) weights((p + 1) & 3);
                ok = sync();
            }
            if (!ok || !sync()) break;
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kFinishRegs));
        const int qt = tid - kWideQuads * kQuadWarps * 32, n_seq = L.s.n_seq;
        for (int step = 0; step < max_steps; ++step) {
            const uint32_t* live = L.live + (size_t)(step & 1) * n_seq;
            const uint32_t* upd = L.upd + (size_t)(step & 1) * n_seq;
            const int2 n = counts(step);
            if (n.x == 0) break;
            if (n.y > 0) {
                wide_finish<kPhaseA>(L, S, upd, n.y, qt, 0);
                if (!sync()) break;
                wide_finish<kPhaseB>(L, S, upd, n.y, qt, 0);
                if (!sync()) break;
                wide_finish<kPhaseC>(L, S, upd, n.y, qt, 0);
                if (!sync()) break;
            }
            wide_finish<kPhaseD>(L, S, live, n.x, qt, step & 1);
            // the counters of the step after the next were last read when this step's predecessor began
            if (blockIdx.x == 0 && qt == 0) __stcg(reinterpret_cast<int2*>(L.counts) + (step + 2) % 3, make_int2(0, 0));
            if (!sync()) break;
            uint32_t* next_live = L.live + (size_t)((step + 1) & 1) * n_seq;
            uint32_t* next_upd = L.upd + (size_t)((step + 1) & 1) * n_seq;
            int* next_counts = L.counts + 2 * ((step + 1) % 3);
            for (int i = qwarp * gridDim.x + blockIdx.x; i < n.x; i += gridDim.x * kQuadWarps)
                decide(L, __ldcg(live + i), lane, step & 1, next_live, next_upd, next_counts);
            if (!sync()) break;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");  // copies still under way land before the CTA's shared memory goes
    }
}

// ---------------------------------------------------------------- few sequences
// At most sixteen sequences: column b of every product is sequence b, every tile belongs to one four-warp group for the
// whole call, and every CTA takes the decisions itself (from the tiles' statistics, a kilobyte per sequence), so that a
// step over a blank has one grid barrier and one that follows an emission has four.  Groups 0..319 keep the fragments of
// phase A (the first 160 swap to phase B's and back while others work), 320..384 those of phase D, 385..424 phase C's.
// The cells' states stay in the registers of the groups that own the units.  Whole call, 188 frames, this kernel / the
// general one: 1 clip 0.80 / 1.37 ms; 16 clips here 2.20 ms, 17 clips there 2.59; the sixteen columns of two MMAs are the line.
constexpr int kSmallSeqs = 16;
constexpr int kSmallGroups = 2 * kLstmTiles + kOutTiles + kPredTiles;  // 425
constexpr int kZStride = kH + 32;  // bf16 per joint input row in shared memory: eight rows on distinct banks
constexpr size_t kSmallSmem = sizeof(bf16) * 2 * kSmallSeqs * kZStride;

__global__ void __launch_bounds__(kDecThreads, 1)
tdt_decode_small_kernel(const __grid_constant__ LoopState L, int max_steps) {
    extern __shared__ __align__(16) bf16 zs[];  // [plane][sequence][kZStride]
    __shared__ __align__(16) float P[kQuads][kQuadWarps][16 * kPStride];
    __shared__ int gave_up;
    __shared__ int sh_frame[kSmallSeqs], sh_symbols[kSmallSeqs], sh_token[kSmallSeqs], sh_tokens[kSmallSeqs], sh_steps[kSmallSeqs],
        sh_len[kSmallSeqs], sh_row[kSmallSeqs];
    __shared__ Decision sh_dec[kSmallSeqs];
    __shared__ unsigned sh_live, sh_upd, sh_par;
    const DecodeState& s = L.s;
    const int tid = threadIdx.x, warp = tid >> 5, quad = warp / kQuadWarps, n = s.n_seq;
    int lane = tid & 31, qwarp = warp % kQuadWarps;
    const bool two = n > 8;
    int me = quad * gridDim.x + blockIdx.x;
    const bool does_a = me < 2 * kLstmTiles, does_b = me < kLstmTiles;
    const bool does_d = !does_a && me < 2 * kLstmTiles + kOutTiles;
    const bool does_c = !does_a && !does_d && me < kSmallGroups;
    bool fills_z = false;  // some group of this CTA does phase D
    for (int k = 0; k < kQuads; ++k) {
        const int m = k * gridDim.x + blockIdx.x;
        fills_z |= m >= 2 * kLstmTiles && m < 2 * kLstmTiles + kOutTiles;
    }
    GridBarrier grid(L, &gave_up);
    const uint4* tile_a = does_a ? tile_of(L.w, kPhaseA, me) : nullptr;
    const uint4* tile_b = does_b ? tile_of(L.w, kPhaseB, me) : nullptr;
    Fragments f;
    f.tile = nullptr;
    if (does_a) fetch_fragments(f, tile_a, qwarp, lane);
    if (does_d) fetch_fragments(f, tile_of(L.w, kPhaseD, me - 2 * kLstmTiles), qwarp, lane);
    if (does_c) fetch_fragments(f, tile_of(L.w, kPhaseC, me - 2 * kLstmTiles - kOutTiles), qwarp, lane);
    if (warp == 0) {
        const int len = lane < n ? s.enc_len[lane] : 0;
        if (lane < n) {
            sh_len[lane] = len;
            sh_row[lane] = s.enc_off[lane];
            sh_frame[lane] = sh_symbols[lane] = sh_tokens[lane] = sh_steps[lane] = 0;
            sh_token[lane] = kVocab - 1;  // the blank (src/model.rs:123)
        }
        const unsigned live = __ballot_sync(0xffffffffu, len > 0);
        if (lane == 0) { sh_live = sh_upd = live; sh_par = 0; }
    }
    __syncthreads();
    float c0 = 0.0f, c0_new = 0.0f, c1 = 0.0f, c1_new = 0.0f;  // the state of this thread's cell

    for (int step = 0; step < max_steps; ++step) {
        const unsigned live = sh_live, upd = sh_upd, par = sh_par;
        if (live == 0) break;
        const size_t set = step & 1;
        // what follows from these is formed anew in every step: kept for all of them, it takes more registers than there are
        asm volatile("" : "+r"(lane), "+r"(qwarp), "+r"(me));
        const int g = lane >> 2, q = lane & 3, qt = qwarp * 32 + lane, r16 = qt & 15;
        const int colx[2] = {min(g, n - 1), min(8 + g, n - 1)};              // columns of this lane's operands
        const int col[2] = {min(qt >> 4, n - 1), min(8 + (qt >> 4), n - 1)};  // columns this thread finishes
        const bool mine[2] = {(qt >> 4) < n, 8 + (qt >> 4) < n};
        const int ccol = min(qt >> 2, n - 1), cunit = qt & 3;  // the cell of threads 0 .. 4 n - 1 of a group: column, unit of the tile
        const bool has_cell = qt < 4 * n;

        // product of this group's tile with the hidden vectors of `layer` (new: the candidates) -> P, summed by the caller
        auto hidden_product = [&](int layer, bool fresh, unsigned par) {
            float v[4];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (j && !two) break;
                const int slot = ((par >> colx[j]) & 1) ^ (fresh ? 1 : 0);
                Pair x[kWarpKB];
                load_x(x, L.h + ((size_t)(slot * 2 + layer) * n + colx[j]) * kRowElems + qwarp * kWarpKB * kBlockElems + q * 16);
                product(f, x, v);
                store_partial(P[quad][qwarp], j, lane, v);
            }
            quad_barrier(quad);
        };
        auto put_hidden = [&](int layer, unsigned par, int unit, float hn) {
            const int slot = ((par >> ccol) & 1) ^ 1;
            bf16 hi, lo;
            split2(hn, hi, lo);
            bf16* ho = L.h + ((size_t)(slot * 2 + layer) * n + ccol) * kRowElems + elem_of(unit);
            ho[0] = hi;
            ho[8] = lo;
        };
        if (upd) {
            // ---- A
            if (does_a) {
                const bool rec = me >= kLstmTiles;
                const int row = me * 16 + r16, unit = me * 4 + cunit;
                float4 gates = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (!rec && has_cell) gates = __ldg(reinterpret_cast<const float4*>(L.w.token_gates + (size_t)sh_token[ccol] * kGates) + unit);
                hidden_product(rec ? 1 : 0, false, par);
                if (rec) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        if (j && !two) break;
                        const float v = sum_partials(P[quad], ((qt >> 4) + 8 * j) * kPStride + r16);
                        if (mine[j] && ((upd >> col[j]) & 1)) __stcg(L.part + (size_t)col[j] * kGates + (row - kGates), v);
                    }
                } else if (has_cell && ((upd >> ccol) & 1)) {
                    float hn;
                    cell(add4(sum_partials4(P[quad], ccol * kPStride + 4 * cunit), gates), c0, c0_new, hn);
                    put_hidden(0, par, unit, hn);
                }
                if (does_b) fetch_fragments(f, tile_b, qwarp, lane);
            }
            if (!grid.sync()) return;
            // ---- B
            if (does_b) {
                const int unit = me * 4 + cunit;
                float4 gates = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (has_cell)
                    gates = add4(__ldcg(reinterpret_cast<const float4*>(L.part + (size_t)ccol * kGates) + unit), __ldg(reinterpret_cast<const float4*>(L.w.b1) + unit));
                hidden_product(0, true, par);
                if (has_cell && ((upd >> ccol) & 1)) {
                    float hn;
                    cell(add4(sum_partials4(P[quad], ccol * kPStride + 4 * cunit), gates), c1, c1_new, hn);
                    put_hidden(1, par, unit, hn);
                }
                fetch_fragments(f, tile_a, qwarp, lane);
            }
            if (!grid.sync()) return;
            // ---- C
            if (does_c) {
                const int row = (me - 2 * kLstmTiles - kOutTiles) * 16 + r16;
                const float bias = __ldg(L.b_pred + row);
                hidden_product(1, true, par);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (j && !two) break;
                    const float v = sum_partials(P[quad], ((qt >> 4) + 8 * j) * kPStride + r16) + bias;
                    if (mine[j] && ((upd >> col[j]) & 1)) __stcg(s.pred + (size_t)col[j] * kJointDim + row, v);
                }
            }
            if (!grid.sync()) return;
        }
        // ---- D: joint input of every live sequence into shared memory, then the product
        if (fills_z) {
            for (int i = tid; i < n * (kJointDim / 4); i += kDecThreads) {
                const int b = i / (kJointDim / 4), c4 = i % (kJointDim / 4);
                if (!((live >> b) & 1)) continue;
                const float4 x = __ldg(reinterpret_cast<const float4*>(s.enc_proj + (size_t)(sh_row[b] + sh_frame[b]) * kJointDim) + c4);
                const float4 p = __ldcg(reinterpret_cast<const float4*>(s.pred + (size_t)b * kJointDim) + c4);
                const float zv[4] = {fmaxf(x.x + p.x, 0.0f), fmaxf(x.y + p.y, 0.0f), fmaxf(x.z + p.z, 0.0f), fmaxf(x.w + p.w, 0.0f)};
                __align__(8) bf16 hi[4], lo[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) split2(zv[e], hi[e], lo[e]);
                *reinterpret_cast<uint2*>(zs + (size_t)b * kZStride + 4 * c4) = *reinterpret_cast<const uint2*>(hi);
                *reinterpret_cast<uint2*>(zs + (size_t)(kSmallSeqs + b) * kZStride + 4 * c4) = *reinterpret_cast<const uint2*>(lo);
            }
            __syncthreads();
            if (does_d) {
                const int tile = me - 2 * kLstmTiles, row = tile * 16 + r16;
                const float bias = __ldg(L.w.b_out + row);
                float v[4];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (j && !two) break;
                    const uint4* z = reinterpret_cast<const uint4*>(zs + (size_t)colx[j] * kZStride) + qwarp * kWarpKB * 4 + q;
                    Pair x[kWarpKB];
#pragma unroll
                    for (int kb = 0; kb < kWarpKB; ++kb) x[kb] = {z[kb * 4], z[kSmallSeqs * kZStride / 8 + kb * 4]};
                    product(f, x, v);
                    store_partial(P[quad][qwarp], j, lane, v);
                }
                quad_barrier(quad);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (j && !two) break;
                    const float lv = sum_partials(P[quad], ((qt >> 4) + 8 * j) * kPStride + r16) + bias;
                    const bool ok = mine[j] && ((live >> col[j]) & 1);
                    const size_t b = col[j];
                    tile_stat(lv, tile, row, lane, ok, L.stat + (set * n + b) * kOutTiles, L.tail + (set * n + b) * 16);
                    if (ok && s.trace && row < kJointOut && sh_steps[b] < s.trace_cap)
                        s.trace[(b * s.trace_cap + sh_steps[b]) * kJointOut + row] = lv;
                }
            }
        }
        if (!grid.sync()) return;
        // ---- E, in every CTA
        for (int b = warp; b < n; b += kDecThreads / 32) {
            if (!((live >> b) & 1)) continue;
            const Decision d = decide_tokens(L.stat + (set * n + b) * kOutTiles, L.tail + (set * n + b) * 16, lane);
            if (lane == 0) sh_dec[b] = d;
        }
        __syncthreads();
        if (warp == 0) {
            bool alive = false, emit = false;
            if (lane < n && ((live >> lane) & 1)) {
                const Decision d = sh_dec[lane];
                emit = d.token != kVocab - 1;
                if (emit) {
                    if (blockIdx.x == lane) record(s, lane, sh_tokens[lane], d, sh_frame[lane]);
                    sh_tokens[lane] += 1;
                    sh_token[lane] = d.token;
                }
                int frame = sh_frame[lane], symbols = sh_symbols[lane];
                advance(emit, d.dur, frame, symbols);
                sh_frame[lane] = frame;
                sh_symbols[lane] = symbols;
                sh_steps[lane] += 1;
                alive = frame < sh_len[lane];
            }
            const unsigned la = __ballot_sync(0xffffffffu, alive), em = __ballot_sync(0xffffffffu, emit);
            if (lane == 0) {
                sh_live = la;
                sh_upd = la & em;
                sh_par = par ^ em;  // committing the state that produced the token (src/model.rs:188-189)
            }
        }
        __syncthreads();
        const unsigned emitted = par ^ sh_par;
        if ((emitted >> ccol) & 1) {
            c0 = c0_new;
            c1 = c1_new;
        }
    }
    if (blockIdx.x == 0 && tid < n) {
        s.n_tokens[tid] = sh_tokens[tid];
        s.n_steps[tid] = sh_steps[tid];
    }
}

// Lists of the first step: every sequence with frames is alive and its predictor must run (blank, zero state).
__global__ void dec_init_kernel(LoopState L) {
    for (int b = blockIdx.x * 256 + threadIdx.x; b < L.s.n_seq; b += gridDim.x * 256)
        if (L.s.enc_len[b] > 0) {
            const uint32_t entry = b | (uint32_t)(kVocab - 1) << kTokenShift;  // the blank comes first (src/model.rs:123)
            L.live[atomicAdd(L.counts, 1)] = entry;
            L.upd[atomicAdd(L.counts + 1, 1)] = entry;
        }
}

constexpr size_t align256(size_t n) { return (n + 255) / 256 * 256; }

struct ScratchLayout {
    size_t h, c, z, part, stat, tail, live, upd, counts, barrier, total;
    explicit ScratchLayout(int n_seq) {
        const size_t B = (size_t)n_seq;
        size_t at = 0;
        auto take = [&](size_t bytes) { const size_t o = at; at += align256(bytes); return o; };
        // zeroed at the start: states, counters, barrier
        h = take(8 * B * kH * sizeof(bf16));
        c = take(4 * B * kH * sizeof(float));
        counts = take(6 * sizeof(int));
        barrier = take(sizeof(unsigned));
        z = take(2 * B * kH * sizeof(bf16));
        part = take(B * kGates * sizeof(float));
        stat = take(2 * B * kOutTiles * sizeof(float4));
        tail = take(2 * B * 16 * sizeof(float));
        live = take(2 * B * sizeof(uint32_t));
        upd = take(2 * B * sizeof(uint32_t));
        total = at;
    }
};

}  // namespace

constexpr size_t kPackedTiles = 3 * kLstmTiles + kPredTiles + kOutTiles;

size_t decode_tc_weight_bytes() {
    return sizeof(uint4) * kPackedTiles * kTileU4 + sizeof(float) * ((size_t)kVocab * kGates + kGates + kOutPad) +
           sizeof(bf16) * 3 * (size_t)kJointDim * kDModel;
}

cudaError_t decode_tc_prepare(const DecodeWeights& w, const float* w_enc, DecodeTcWeights* t, void* storage,
                              cudaStream_t st) {
    uint4* p = reinterpret_cast<uint4*>(storage);
    const size_t G = (size_t)kGates * kH;
    auto pack = [&](const float* src, int rows, int tiles, bool lstm) -> const uint4* {
        uint4* dst = p;
        pack_fragments_kernel<<<tiles, 128, 0, st>>>(src, rows, lstm, dst);
        p += (size_t)tiles * kTileU4;
        return dst;
    };
    t->hh0 = pack(w.w_hh, kGates, kLstmTiles, true);
    t->ih1 = pack(w.w_ih + G, kGates, kLstmTiles, true);
    t->hh1 = pack(w.w_hh + G, kGates, kLstmTiles, true);
    t->pred = pack(w.w_pred, kJointDim, kPredTiles, false);
    t->out = pack(w.w_out, kJointOut, kOutTiles, false);
    float* q = reinterpret_cast<float*>(p);
    t->token_gates = q;
    token_gates_kernel<<<dim3(kVocab, kGates / 256), 256, 0, st>>>(w.embedding, w.w_ih, w.b_gates, q);
    q += (size_t)kVocab * kGates;
    t->b1 = q;
    t->b_out = q + kGates;
    bias_kernel<<<(kGates + 255) / 256, 256, 0, st>>>(w.b_gates + kGates, q, w.b_out, q + kGates);
    q += kGates + kOutPad;
    t->wenc = reinterpret_cast<bf16*>(q);
    split_weight_kernel<<<512, 256, 0, st>>>(w_enc, kDModel, t->wenc, kJointDim);
    return cudaGetLastError();
}

size_t decode_tc_scratch_bytes(int64_t enc_rows, int n_seq) {
    return align256(sizeof(bf16) * (size_t)enc_rows * 3 * kDModel) + ScratchLayout(n_seq).total;
}

// enc_proj [rows x 640] = enc [rows x 1024] W_enc^T + b_enc through the split product.
cudaError_t decode_tc_enc_projection(const DecodeTcWeights& t, const float* d_enc, const float* b_enc, float* d_proj,
                                     int64_t rows, void* scratch, int sm_count, int* d_error, int64_t* launches,
                                     cudaStream_t st) {
    if (rows <= 0) return cudaSuccess;
    bf16* a = reinterpret_cast<bf16*>(scratch);
    split_act_kernel<<<2048, 256, 0, st>>>(d_enc, a, rows, kDModel);
    GemmArgs g{};
    g.a = a;
    g.w = t.wenc;
    g.bias = b_enc;
    g.out = d_proj;
    g.M = (int)rows;
    g.N = kJointDim;
    g.K = 3 * kDModel;
    g.ldo = kJointDim;
    g.act = kActNone;
    g.out_mode = kOutF32;
    g.alpha = 1.0f;
    g.fp8 = false;
    g.w_resident = true;
    const cudaError_t e = gemm_launch(g, sm_count, d_error, st);
    *launches += 2;
    return e != cudaSuccess ? e : cudaGetLastError();
}

// Runs the greedy loop for s.n_seq sequences (the integer state is set up by the caller).
cudaError_t decode_tc_run(const DecodeWeights& w, const DecodeTcWeights& t, const DecodeState& s, int max_steps,
                          int64_t enc_rows, void* scratch, int sm_count, int* d_error, int64_t* launches, cudaStream_t st) {
    if (s.n_seq > kMaxSeqs) return cudaErrorInvalidValue;
    char* base = static_cast<char*>(scratch) + align256(sizeof(bf16) * (size_t)enc_rows * 3 * kDModel);
    const ScratchLayout lay(s.n_seq);
    LoopState L{};
    L.s = s;
    L.w = t;
    L.b_pred = w.b_pred;
    L.h = reinterpret_cast<bf16*>(base + lay.h);
    L.c = reinterpret_cast<float*>(base + lay.c);
    L.z = reinterpret_cast<bf16*>(base + lay.z);
    L.part = reinterpret_cast<float*>(base + lay.part);
    L.stat = reinterpret_cast<float4*>(base + lay.stat);
    L.tail = reinterpret_cast<float*>(base + lay.tail);
    L.live = reinterpret_cast<uint32_t*>(base + lay.live);
    L.upd = reinterpret_cast<uint32_t*>(base + lay.upd);
    L.counts = reinterpret_cast<int*>(base + lay.counts);
    L.barrier = reinterpret_cast<unsigned*>(base + lay.barrier);
    L.error = d_error;
    cudaError_t e = cudaMemsetAsync(base, 0, lay.z, st);
    if (e != cudaSuccess) return e;
    void* args[] = {&L, &max_steps};
    if (s.n_seq <= kSmallSeqs && sm_count * kQuads >= kSmallGroups) {
        e = cudaFuncSetAttribute(tdt_decode_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallSmem);
        if (e != cudaSuccess) return e;
        e = cudaLaunchCooperativeKernel((const void*)tdt_decode_small_kernel, dim3(sm_count), dim3(kDecThreads), args, kSmallSmem, st);
        *launches += 1;
        return e != cudaSuccess ? e : cudaGetLastError();
    }
    dec_init_kernel<<<std::min(32, (s.n_seq + 255) / 256), 256, 0, st>>>(L);
    if (s.n_seq >= kWideSeqs) {
        e = cudaFuncSetAttribute(tdt_decode_wide_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kWideSmem);
        if (e != cudaSuccess) return e;
        e = cudaLaunchCooperativeKernel((const void*)tdt_decode_wide_kernel, dim3(sm_count), dim3(kWideThreads), args, kWideSmem, st);
    } else {
        e = cudaLaunchCooperativeKernel((const void*)tdt_decode_tc_kernel, dim3(sm_count), dim3(kDecThreads), args, 0, st);
    }
    *launches += 2;
    return e != cudaSuccess ? e : cudaGetLastError();
}

}  // namespace sb
