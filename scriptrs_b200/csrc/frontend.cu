// Log-mel frontend for sm_100a: PCM (f32 or 16-bit) -> normalised log-mel [T x 128] per clip, one kernel.
//
// Replaces the reference's CPU feature extractor (src/frontend.rs:104-241):
// pre-emphasis 0.97, 256-sample zero padding on both sides, Hann window of 400
// left-aligned in a 512-point real FFT, power spectrum, 128-bin Slaney mel
// filterbank, ln(x + 2^-24), per-feature mean / variance normalisation over
// all frames of the clip.
//
// frontend_clip_kernel: one CTA (8 warps) per clip, two CTAs per SM.  A batch with too few clips to fill the chip has
// its clips' rows spread over CTAs (the same kernel, a few steps each) and the statistics and normalisation done by
// frontend_norm_kernel, column block by column block: the same arithmetic in the same order, bit for bit.
//   rows      The clip is walked 16 frames at a time.  The raw samples of the next 16 frames arrive by cp.async
//             (16-byte pieces where the clip's placement allows it) while the current ones are transformed; one
//             pass turns them into pre-emphasised, zero-padded samples (16-bit input is converted here).  Each
//             warp then transforms two frames, sixteen lanes per frame (frontend_core.cuh: two register radix-16
//             passes around one shared-memory transpose, untangling + power, sparse mel filterbank, ln), and leaves
//             the two log-mel rows in a 16-row stage in shared memory.  At the top of the next step the stage is
//             written out with 16-byte stores, and threads 0..127 add its rows to their column sums.
//   statistics The reference sums every column strictly left to right in f32 (frontend.rs:225-236); for a constant
//             column (an all-zero clip) the result consists of the rounding residue of exactly that order, so the
//             order is kept: thread c owns column c.  The first sum comes from the stage (no re-read); the second
//             pass (squared deviations) streams the clip's rows back through a cp.async ring per warp.
//   normalise (v - mean) / std over the clip's rows, 16-byte loads and stores, all threads.
// While one CTA of an SM is in its two bandwidth-bound tail passes the other one keeps the SM's issue slots busy
// with transforms, so the passes cost little wall time although they re-read the clip's rows.  The kernel is bound by
// shared-memory wavefronts and issue slots, not by DRAM: the filterbank taps and as much state as fits live in
// registers (128 per thread, two CTAs per SM), and buffers are laid out so that the two frames of a warp use
// different banks.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "frontend.h"
#include "frontend_core.cuh"

namespace sb {

namespace {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr int kStepFrames = 2 * kWarps;                           // 16 frames per step
constexpr int kRawElems = 2816;  // the step's samples + the one before them + up to 7 of alignment shift, in 16-byte pieces
constexpr int kRingRows = 16;    // rows per ring slot of the second statistics pass
constexpr int kRingSlots = 4;

constexpr int kStageStride = kMels + 16;  // floats per stage row: the two frames of a warp write different banks

struct __align__(16) SmemLayout {
    float2 scratch[kWarps][2][fe::kFrameScratch];  // per frame: transpose buffer, then Z, then the power bins; the
                                                   // statistics ring after the last step
    float raw[kRawElems];                          // raw samples of the next step (16-bit input: first half)
    float ys[kRawElems + 8];                       // pre-emphasised samples of this step, indexed like raw (+ ys_off)
    float stage[kStepFrames][kStageStride];        // log-mel rows of one step
    float window[kWin];
    float2 tw_post[132];
    float2 twid[256];
    float mean[kMels];
    float stdv[kMels];
    int16_t mel_start[kMels];
};
static_assert(sizeof(float2) * kWarps * 2 * fe::kFrameScratch >= sizeof(float) * 4 * kRingSlots * kRingRows * 32,
              "the statistics ring must fit in the transform scratch");

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(uint32_t dst, const void* src, int src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

template <typename TIn>
struct Sample;
template <>
struct Sample<float> {
    static constexpr int kPerPiece = 4;  // samples per 16 bytes
    static __device__ __forceinline__ float get(const void* raw, int j) { return static_cast<const float*>(raw)[j]; }
};
template <>
struct Sample<int16_t> {
    static constexpr int kPerPiece = 8;
    static __device__ __forceinline__ float get(const void* raw, int j) {
        return fe::pcm16_to_f32(static_cast<const int16_t*>(raw)[j]);
    }
};

// (v - mean) / std with the IEEE quotient (frontend.rs:237-239), four columns at a time.  For a divisor in the range
// below the quotient is formed from the correctly rounded reciprocal and one exact-remainder correction, three
// instructions, which gives the correctly rounded result (Markstein's correction step; checked against the
// hardware division on 4e8 operand pairs, all-ones significands included); any other divisor takes __fdiv_rn.
struct Normaliser {
    float4 mu, sd, rc;
    bool fast;
    static __device__ __forceinline__ bool plain(float d) {
        const uint32_t b = __float_as_uint(d);
        return d >= 7.62939453125e-06f && d < 128.0f && (b & 0x7FFFFFu) != 0x7FFFFFu;  // 2^-17 <= d < 2^7
    }
    static __device__ __forceinline__ float quot(float x, float d, float r) {
        const float q = __fmul_rn(x, r);
        return fmaf(fmaf(-q, d, x), r, q);
    }
    __device__ __forceinline__ Normaliser(float4 mean, float4 std) : mu(mean), sd(std) {
        fast = plain(sd.x) && plain(sd.y) && plain(sd.z) && plain(sd.w);
        rc = make_float4(__frcp_rn(sd.x), __frcp_rn(sd.y), __frcp_rn(sd.z), __frcp_rn(sd.w));
    }
    __device__ __forceinline__ float4 apply(float4 v) const {
        const float a = __fsub_rn(v.x, mu.x), b = __fsub_rn(v.y, mu.y);
        const float c = __fsub_rn(v.z, mu.z), d = __fsub_rn(v.w, mu.w);
        if (fast) return make_float4(quot(a, sd.x, rc.x), quot(b, sd.y, rc.y), quot(c, sd.z, rc.z), quot(d, sd.w, rc.w));
        return make_float4(__fdiv_rn(a, sd.x), __fdiv_rn(b, sd.y), __fdiv_rn(c, sd.z), __fdiv_rn(d, sd.w));
    }
};

// SPLIT: the CTA computes only the log-mel rows of `chunk` steps of its clip (grid: chunks x clips); the statistics
// and the normalisation are frontend_norm_kernel's.
template <typename TIn, bool SPLIT>
__global__ void __launch_bounds__(kThreads, 2)
frontend_clip_kernel(const TIn* __restrict__ pcm, const int64_t* __restrict__ clip_start,
                     const int64_t* __restrict__ clip_len, const int64_t* __restrict__ frame_off,
                     float* __restrict__ out, float preemph, const FrontendTables* __restrict__ tables, int normalize,
                     int chunk) {
    if constexpr (SPLIT) asm volatile("griddepcontrol.launch_dependents;");  // frontend_norm_kernel waits for this grid itself
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmemLayout& sm = *reinterpret_cast<SmemLayout*>(smem_raw);
    constexpr int PP = Sample<TIn>::kPerPiece;

    const int clip = SPLIT ? blockIdx.y : blockIdx.x;
    const int64_t c0 = clip_start[clip];
    const int64_t n = clip_len[clip];
    const int64_t fo = frame_off[clip];
    const int T = (int)(frame_off[clip + 1] - fo);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const TIn* x = pcm + c0;
    // Placement of the clip in memory: shared-memory index j of a step's buffers holds clip sample gbase + j, with
    // gbase chosen so that index 0 sits on a 16-byte boundary of the PCM buffer.  `shift` (0 .. PP-1) is how far the
    // sample before the step lies above that boundary; it is the same for every step (a step is 2560 samples).
    const int64_t elem0 = (int64_t)(reinterpret_cast<uintptr_t>(pcm) / sizeof(TIn)) + c0;   // absolute element index
    const int shift = (int)(((elem0 - kPad - 1) % PP + PP) % PP);
    // A frame's first sample sits at index shift + 1 + 160 fl of the pre-emphasised buffer; the transform reads sample
    // pairs with 8-byte loads, so an odd shift + 1 (a clip that starts on an odd sample of the PCM buffer) moves the
    // whole buffer up by one element.
    const int ys_off = (shift + 1) & 1;
    const int first_step = SPLIT ? (int)blockIdx.x * chunk : 0;
    const int all_steps = (T + kStepFrames - 1) / kStepFrames;
    const int n_steps = SPLIT ? min(all_steps, first_step + chunk) : all_steps;
    if (SPLIT && first_step >= n_steps) return;

    // Raw samples of a step -> shared memory, asynchronously; zero outside the clip (frontend.rs:59-65).
    auto fetch = [&](int step) {
        const int64_t gbase = (int64_t)step * kStepFrames * kHop - kPad - 1 - shift;
        TIn* dst = reinterpret_cast<TIn*>(sm.raw);
        if (gbase >= 0 && gbase + kRawElems <= n) {  // the whole step lies inside the clip
            const TIn* src = x + gbase;
            for (int q = tid; q < kRawElems / PP; q += kThreads) cp_async16(smem_addr(dst + q * PP), src + q * PP, 16);
        } else {
            for (int q = tid; q < kRawElems / PP; q += kThreads) {
                const int64_t g = gbase + (int64_t)q * PP;
                const uint32_t d = smem_addr(dst + q * PP);
                if (g >= 0 && g + PP <= n) {
                    cp_async16(d, x + g, 16);
                } else if (g + PP <= 0 || g >= n) {
                    *reinterpret_cast<uint4*>(dst + q * PP) = make_uint4(0u, 0u, 0u, 0u);
                } else if constexpr (sizeof(TIn) == 4) {
#pragma unroll
                    for (int e = 0; e < PP; ++e) {
                        const bool in = g + e >= 0 && g + e < n;
                        cp_async4(d + 4 * e, x + (in ? g + e : 0), in ? 4 : 0);
                    }
                } else {
                    // 16-bit samples at a clip edge: plain loads (cp.async moves at least four bytes)
#pragma unroll
                    for (int e = 0; e < PP; ++e) {
                        const bool in = g + e >= 0 && g + e < n;
                        dst[q * PP + e] = in ? x[g + e] : TIn(0);
                    }
                }
            }
        }
        cp_async_commit();
    };
    fetch(first_step);

    // Tables -> shared memory.
    for (int i = tid; i < kWin; i += kThreads) sm.window[i] = tables->window[i];
    for (int i = tid; i < 132; i += kThreads) sm.tw_post[i] = tables->tw_post[i];
    for (int i = tid; i < 256; i += kThreads) sm.twid[i] = tables->twid[i];
    for (int i = tid; i < kMels; i += kThreads) sm.mel_start[i] = tables->mel_start[i];
    const float log_floor = tables->log_floor;

    float sum = 0.0f;  // threads 0..127: running sum of column tid, frontend.rs:230
    // Rows of a finished step: out to memory (16-byte stores), and into the column sums in frame order.
    auto flush = [&](int step) {
        const int f0 = step * kStepFrames;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int idx = tid + kThreads * k, row = idx >> 5, c4 = idx & 31;
            if (f0 + row < T)
                reinterpret_cast<float4*>(out + (fo + f0 + row) * kMels)[c4] = reinterpret_cast<const float4*>(sm.stage[row])[c4];
        }
        if (!SPLIT && tid < kMels) {
            const int rows = min(kStepFrames, T - f0);
            if (rows == kStepFrames) {
#pragma unroll
                for (int r = 0; r < kStepFrames; ++r) sum = __fadd_rn(sum, sm.stage[r][tid]);
            } else {
                for (int r = 0; r < rows; ++r) sum = __fadd_rn(sum, sm.stage[r][tid]);
            }
        }
    };

    const int half = lane >> 4, p = lane & 15;
    float taps[kMelTapRows];  // this lane's filterbank taps (rows 16 g + p)
    fe::load_mel_taps(p, tables->melw, taps);
    for (int step = first_step; step < n_steps; ++step) {
        cp_async_wait<0>();
        __syncthreads();  // this step's raw samples are in; the previous step's rows are all in the stage
        if (step > first_step) flush(step - 1);
        // Pre-emphasis (frontend.rs:150-159): y[0] = x[0]; y[i] = x[i] - c * x[i-1], product rounded first; zero outside
        // the clip (the padding is added after the pre-emphasis, frontend.rs:59-65).
        {
            const int64_t gbase = (int64_t)step * kStepFrames * kHop - kPad - 1 - shift;
            const void* raw = sm.raw;
            const bool inside = gbase >= 0 && gbase + kRawElems <= n;
            for (int q = tid; q < kRawElems / 4; q += kThreads) {
                const int j = 4 * q;
                float xs[5];
                xs[0] = j > 0 ? Sample<TIn>::get(raw, j - 1) : 0.0f;
#pragma unroll
                for (int e = 0; e < 4; ++e) xs[e + 1] = Sample<TIn>::get(raw, j + e);
                float4 y;
                float* yv = reinterpret_cast<float*>(&y);
                const int64_t g = gbase + j;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float v = __fsub_rn(xs[e + 1], __fmul_rn(preemph, xs[e]));
                    yv[e] = (inside || (g + e >= 0 && g + e < n)) ? v : 0.0f;
                }
                if (ys_off == 0) {
                    *reinterpret_cast<float4*>(sm.ys + j) = y;
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) sm.ys[j + 1 + e] = yv[e];
                }
            }
        }
        __syncthreads();  // samples ready; the stage and the raw buffer are free again
        if (step + 1 < n_steps) fetch(step + 1);  // lands while this step is transformed
        {
            const int fl = 2 * warp + half;                                // frame of the step this half-warp transforms
            const float* ysf = sm.ys + shift + 1 + ys_off + fl * kHop;     // its 400 samples
            float2* B = sm.scratch[warp][half];
            fe::pass1(p, ysf, sm.window, sm.twid, B);
            __syncwarp();
            {
                float2 z[16];
                fe::pass2(p, B, z);
                __syncwarp();
                fe::store_z(p, z, B);
            }
            __syncwarp();
            float* pwf = reinterpret_cast<float*>(B);  // the power bins take Z's place once every lane holds its Z values
            {
                float2 zk[8], zc[8], z0;
                fe::untangle_load(p, B, zk, zc, z0);
                __syncwarp();
                fe::untangle_store(p, zk, zc, z0, sm.tw_post, pwf);
            }
            __syncwarp();
            fe::mel_rows(p, pwf, taps, sm.mel_start, log_floor, sm.stage[fl]);
        }
    }
    __syncthreads();
    flush(n_steps - 1);
    if (SPLIT || !normalize) return;

    // ---- statistics, frontend.rs:225-236.  Thread c (< 128) owns column c; warp w streams rows of columns
    // 32 w .. 32 w + 31 through its own ring of kRingSlots x kRingRows rows.
    __syncthreads();  // every row of the clip has been stored by this CTA
    const float* rows = out + fo * kMels;
    if (warp < kMels / 32) {
        const float mean = __fdiv_rn(sum, (float)T);
        float* ring = reinterpret_cast<float*>(&sm.scratch[0][0][0]) + warp * (kRingSlots * kRingRows * 32);
        const int n_blk = (T + kRingRows - 1) / kRingRows;
        auto issue = [&](int blk) {
            if (blk < n_blk) {
                float* slot = ring + (blk % kRingSlots) * (kRingRows * 32);
#pragma unroll
                for (int k = 0; k < kRingRows * 8 / 32; ++k) {
                    const int q = lane + 32 * k, r = q >> 3, ch = q & 7;
                    const int row = blk * kRingRows + r;
                    const bool in = row < T;
                    cp_async16(smem_addr(slot + r * 32 + 4 * ch), rows + (int64_t)(in ? row : 0) * kMels + 32 * warp + 4 * ch,
                               in ? 16 : 0);
                }
            }
            cp_async_commit();
        };
#pragma unroll
        for (int s = 0; s < kRingSlots - 1; ++s) issue(s);
        float acc = 0.0f;
        for (int blk = 0; blk < n_blk; ++blk) {
            issue(blk + kRingSlots - 1);  // refills the slot that was read one iteration ago
            cp_async_wait<kRingSlots - 1>();
            __syncwarp();
            const float* slot = ring + (blk % kRingSlots) * (kRingRows * 32);
            const int nr = min(kRingRows, T - blk * kRingRows);
            if (nr == kRingRows) {
#pragma unroll
                for (int r = 0; r < kRingRows; ++r) {
                    const float d = __fsub_rn(slot[r * 32 + lane], mean);
                    acc = __fadd_rn(acc, __fmul_rn(d, d));
                }
            } else {
                for (int r = 0; r < nr; ++r) {
                    const float d = __fsub_rn(slot[r * 32 + lane], mean);
                    acc = __fadd_rn(acc, __fmul_rn(d, d));
                }
            }
            __syncwarp();  // all lanes are done with the slot before the next issue overwrites it
        }
        cp_async_wait<0>();
        // variance / (T - 1); T == 1 divides 0 by 0 and yields NaN exactly as the reference does.
        const float variance = __fdiv_rn(acc, __fsub_rn((float)T, 1.0f));
        sm.mean[tid] = mean;
        sm.stdv[tid] = __fadd_rn(__fsqrt_rn(variance), 1e-5f);
    }
    __syncthreads();
    // ---- normalise, frontend.rs:237-239
    {
        const int c4 = tid & 31;
        const Normaliser norm(reinterpret_cast<const float4*>(sm.mean)[c4], reinterpret_cast<const float4*>(sm.stdv)[c4]);
        float4* rows4 = reinterpret_cast<float4*>(out + fo * kMels);
        constexpr int U = 8;
        for (int r0 = tid >> 5; r0 < T; r0 += 8 * U) {
            float4 v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int r = r0 + 8 * u;
                if (r < T) v[u] = __ldcg(rows4 + (int64_t)r * 32 + c4);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int r = r0 + 8 * u;
                if (r < T) rows4[(int64_t)r * 32 + c4] = norm.apply(v[u]);
            }
        }
    }
}

// Statistics and normalisation of a clip whose log-mel rows lie in `out`, COLS columns per CTA (grid: column groups x
// clips).  The T x COLS block of the clip is fetched once into shared memory (cp.async, kNormGroups commit groups, so
// that the column sums start on the first rows while the others are under way); one warp then walks its columns in
// frame order, a lane per column, exactly as the one-CTA-per-clip kernel does (frontend.rs:225-236: the order of the
// sums is part of the result), and all warps normalise.  Bound by the two serial chains of T dependent additions.
constexpr int kNormGroups = 8;
template <int COLS>
__global__ void __launch_bounds__(kThreads)
frontend_norm_kernel(const int64_t* __restrict__ frame_off, float* __restrict__ out) {
    extern __shared__ __align__(16) float block[];  // [T][COLS]
    __shared__ __align__(16) float s_mean[COLS], s_std[COLS];
    constexpr int PC = COLS / 4;  // 16-byte pieces per row
    const int clip = blockIdx.y;
    const int64_t fo = frame_off[clip];
    const int T = (int)(frame_off[clip + 1] - fo);
    float* rows = out + fo * kMels + blockIdx.x * COLS;
    const int tid = threadIdx.x, lane = tid & 31;
    const int group_rows = (T + kNormGroups - 1) / kNormGroups;
    asm volatile("griddepcontrol.wait;" ::: "memory");  // the rows of this clip are complete and visible
#pragma unroll 1
    for (int g = 0; g < kNormGroups; ++g) {
        const int r0 = g * group_rows, n = max(0, min(T, r0 + group_rows) - r0) * PC;
        for (int i = tid; i < n; i += kThreads) {
            const int r = r0 + i / PC, c = 4 * (i % PC);
            cp_async16(smem_addr(block + r * COLS + c), rows + (int64_t)r * kMels + c, 16);
        }
        cp_async_commit();
    }
    float sum = 0.0f;
    const float* col = block + (lane % COLS);
    auto add_group = [&](int g) {
        if (tid >= 32) return;
        const int r1 = min(T, (g + 1) * group_rows);
#pragma unroll 16
        for (int r = g * group_rows; r < r1; ++r) sum = __fadd_rn(sum, col[r * COLS]);
    };
    static_assert(kNormGroups == 8, "one wait per group below");
    cp_async_wait<7>(); __syncthreads(); add_group(0);
    cp_async_wait<6>(); __syncthreads(); add_group(1);
    cp_async_wait<5>(); __syncthreads(); add_group(2);
    cp_async_wait<4>(); __syncthreads(); add_group(3);
    cp_async_wait<3>(); __syncthreads(); add_group(4);
    cp_async_wait<2>(); __syncthreads(); add_group(5);
    cp_async_wait<1>(); __syncthreads(); add_group(6);
    cp_async_wait<0>(); __syncthreads(); add_group(7);
    if (tid < 32) {
        const float mean = __fdiv_rn(sum, (float)T);
        float acc = 0.0f;
#pragma unroll 16
        for (int r = 0; r < T; ++r) {
            const float d = __fsub_rn(col[r * COLS], mean);
            acc = __fadd_rn(acc, __fmul_rn(d, d));
        }
        // variance / (T - 1); T == 1 divides 0 by 0 and yields NaN exactly as the reference does.
        const float variance = __fdiv_rn(acc, __fsub_rn((float)T, 1.0f));
        if (lane < COLS) {
            s_mean[lane] = mean;
            s_std[lane] = __fadd_rn(__fsqrt_rn(variance), 1e-5f);
        }
    }
    __syncthreads();
    static_assert(kThreads % PC == 0, "a thread keeps its columns");
    const int c4 = tid % PC;
    const Normaliser norm(reinterpret_cast<const float4*>(s_mean)[c4], reinterpret_cast<const float4*>(s_std)[c4]);
#pragma unroll 4
    for (int r = tid / PC; r < T; r += kThreads / PC)
        *reinterpret_cast<float4*>(rows + (int64_t)r * kMels + 4 * c4) =
            norm.apply(*reinterpret_cast<const float4*>(block + r * COLS + 4 * c4));
}

constexpr int kNormMaxSmem = 225 * 1024;
constexpr int kSplitMaxFrames = kNormMaxSmem / (16 * (int)sizeof(float));  // 3600 (36 s): 16 columns per CTA; half of it: 32

template <int COLS>
cudaError_t norm_launch(const int64_t* d_frame_off, int n_clips, int max_frames, float* feats, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kMels / COLS, n_clips);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)max_frames * COLS * sizeof(float);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, frontend_norm_kernel<COLS>, d_frame_off, feats);
}

template <typename TIn>
cudaError_t launch_format(const TIn* pcm, const int64_t* d_clip_start, const int64_t* d_clip_len, const int64_t* d_frame_off,
                          int n_clips, int64_t total_frames, int max_frames, float preemph, const FrontendTables* d_tables,
                          float* feats, bool normalize, int sm_count, cudaStream_t stream, int64_t* launches) {
    *launches += 1;
    // One CTA per clip, or the clip's steps and columns spread over the chip.  The one-CTA kernel takes 0.205 us per frame of
    // the longest clip until the SMs are full; the split 1.35 ns per frame in all on 148 SMs, 5 us for its second
    // launch, and 4.5 us for every further wave of that launch's CTAs, whose shared memory is sized for the longest clip: a long
    // clip among thousands of short ones makes them many.  Measured (one-CTA kernel / split, us): 1 clip of 1501 frames
    // 304 / 31, 97 ragged ones 307 / 153, 127 330 / 276, 96 clips of 64 frames 21.5 / 23.9, of 101 frames 31 / 30, of 401 93 /
    // 62; one clip of 3594 frames with 2000 of 51 757 / 609, with 4000 of 101 838 / 1650, with 40000 of 11 frames 960 / 7100.
    // From 148 clips of one length the two lie within 12 % of one another, on either side (1501 frames: 148 clips 335 /
    // 296, 200 clips 453 / 424, 296 clips 489 / 576; 3001 frames: 148 clips 663 / 676): the rule leaves them on one launch.
    // A clip of one or two steps has nothing to split, and the column blocks of a longer one than kSplitMaxFrames do
    // not fit.
    const int cols = max_frames <= kSplitMaxFrames / 2 ? 32 : 16;
    const int64_t norm_smem = (int64_t)max_frames * cols * (int)sizeof(float);
    const int64_t slots = sm_count * std::max<int64_t>(1, std::min<int64_t>(8, 227 * 1024 / (norm_smem + 1024)));
    const int64_t waves = normalize ? ((int64_t)(kMels / cols) * n_clips + slots - 1) / slots : 1;
    const bool split = max_frames > 2 * kStepFrames && max_frames <= kSplitMaxFrames && n_clips <= 65535 &&
                       5.0 + 1.35e-3 * 148.0 / sm_count * total_frames + 4.5 * (waves - 1) < 0.205 * max_frames;
    if (!split) {
        frontend_clip_kernel<TIn, false><<<n_clips, kThreads, sizeof(SmemLayout), stream>>>(
            pcm, d_clip_start, d_clip_len, d_frame_off, feats, preemph, d_tables, normalize ? 1 : 0, 0);
        return cudaGetLastError();
    }
    const int max_steps = (max_frames + kStepFrames - 1) / kStepFrames;
    // steps per CTA: four CTAs for each of an SM's two places if the batch gives as many (the tables are loaded once per
    // CTA; one step per CTA is 15 % slower on 97 clips), and a bounded number of CTAs that find their clip already over
    const int64_t steps = total_frames / kStepFrames + n_clips;
    const int chunk = (int)std::max(std::min<int64_t>(16, std::max<int64_t>(1, steps / (8 * sm_count))), (max_steps * (int64_t)n_clips + 16383) / 16384);
    frontend_clip_kernel<TIn, true><<<dim3((max_steps + chunk - 1) / chunk, n_clips), kThreads, sizeof(SmemLayout), stream>>>(
        pcm, d_clip_start, d_clip_len, d_frame_off, feats, preemph, d_tables, 0, chunk);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess || !normalize) return e;
    *launches += 1;
    return cols == 32 ? norm_launch<32>(d_frame_off, n_clips, max_frames, feats, stream)
                      : norm_launch<16>(d_frame_off, n_clips, max_frames, feats, stream);
}

}  // namespace

size_t frontend_smem_bytes() { return sizeof(SmemLayout); }

cudaError_t frontend_configure() {
    auto opt_in = [](const void* kernel, size_t bytes) {
        return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    for (const void* k : {(const void*)frontend_clip_kernel<float, false>, (const void*)frontend_clip_kernel<float, true>,
                          (const void*)frontend_clip_kernel<int16_t, false>, (const void*)frontend_clip_kernel<int16_t, true>}) {
        const cudaError_t e = opt_in(k, sizeof(SmemLayout));
        if (e != cudaSuccess) return e;
    }
    const cudaError_t e = opt_in((const void*)frontend_norm_kernel<32>, kNormMaxSmem);
    return e != cudaSuccess ? e : opt_in((const void*)frontend_norm_kernel<16>, kNormMaxSmem);
}

cudaError_t frontend_launch(const void* pcm, SampleFormat fmt, const int64_t* d_clip_start, const int64_t* d_clip_len,
                            const int64_t* d_frame_off, int n_clips, int64_t total_frames, int max_frames, float preemph,
                            const FrontendTables* d_tables, float* feats, bool normalize, int sm_count, cudaStream_t stream,
                            int64_t* launches) {
    int64_t ignored;
    if (!launches) launches = &ignored;
    if (n_clips <= 0) return cudaSuccess;
    // 16-byte row accesses of the feature matrix and 4- / 2-byte aligned samples
    if ((reinterpret_cast<uintptr_t>(feats) & 15) || (reinterpret_cast<uintptr_t>(pcm) & (fmt == kSampleI16 ? 1 : 3)))
        return cudaErrorMisalignedAddress;
    if (fmt == kSampleI16)
        return launch_format(static_cast<const int16_t*>(pcm), d_clip_start, d_clip_len, d_frame_off, n_clips, total_frames,
                             max_frames, preemph, d_tables, feats, normalize, sm_count, stream, launches);
    return launch_format(static_cast<const float*>(pcm), d_clip_start, d_clip_len, d_frame_off, n_clips, total_frames,
                         max_frames, preemph, d_tables, feats, normalize, sm_count, stream, launches);
}

}  // namespace sb
