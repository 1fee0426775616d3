// First two stages of the dw-striding sub-sampling on sm_100a, in one kernel:
//   conv2d(1 -> 256, k3, s2, p1) + ReLU          as a product [positions x 16] x [16 x 256] on the tensor cores
//   depthwise conv2d(256, k3, s2, p1) + bias     on packed fp16 pairs
// Part of the encoder that the reference runs as a CoreML blob (src/model.rs:327-342, contract src/coreml.rs:75-135).
//   feats f32 [sum T x 128]  ->  out bf16 [sum T2 x 32 x 256]   (channels last; T1 = (T-1)/2+1, T2 = (T1-1)/2+1)
// The [T1 x 64 x 256] map between the two stages never reaches memory.
//
// grid (shares of the time rows, clips), 256 threads.  A CTA walks its share two output time rows at a time: it stages the
// 11 mel rows they depend on (cp.async, the next ones under the arithmetic of the current ones), gathers the 3 x 3 input
// patches of the 5 x 64 first-stage positions into an im2col tile of fp16
// (9 taps, a constant 1 that carries the bias, 6 zeros: K = 16), and then walks the channels in four blocks of 64:
//   product   mma.m16n8k16 (fp16 in, fp32 accumulate): each warp takes first-stage position tiles of 16 and all
//             8 channel tiles of the block, whose columns are dealt so that a lane ends up with 16 neighbouring channels of
//             a position; ReLU, rows outside the clip forced to zero (they are the second stage's
//             padding), 16-byte stores into a [5 rows x 65 columns x 64 channels] tile (column slot 0 = padding)
//   depthwise each thread owns four channels and two output frequencies and slides a 5 x 5 window over
//             the tile; fp16 multiply-adds (the result is rounded to bf16 anyway), 8-byte bf16 stores
// Bound by shared-memory wavefronts (the first-stage tile is written and read once per row and block: 3900 a step; 560 clips
// of 1497 frames 3.03 -> 2.70 ms against 4-byte stores, two channels a thread and no prefetch,
// which took 15.6 k warp instructions a step instead of 11.8 k).
// fp16 keeps 11 significant bits of the normalised features and of the weights; the accumulation of the first stage
// is fp32.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "subsample.h"

namespace sb {

namespace {

constexpr int kTO = 2;                // output time rows per CTA
constexpr int kNY = 2 * kTO + 1;      // first-stage rows per CTA
constexpr int kNX = 4 * kTO + 3;      // mel rows per CTA
constexpr int kXS = kMelBins + 8;     // floats per staged mel row; mel column f sits at index f + 4
constexpr int kPos = kNY * 64;        // first-stage positions per CTA
constexpr int kY0Stride = 72;         // halfs per (row, column slot) of the first-stage tile: 64 channels + 8 (36 words: eight
                                      // positions x 16 bytes of a quarter-warp's store fall into different banks)
constexpr int kImStride = 24;         // halfs per im2col position: 16 + 8 (12 words: conflict-free fragment loads)

struct __align__(16) SmemLayout {
    float xs[2][kNX][kXS];
    __half im2col[kPos][kImStride];
    __half y0[kNY][65][kY0Stride];
};

__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint2 b) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y));
}

__device__ __forceinline__ uint32_t relu_pack(float a, float b) {
    const __half2 h = __hmax2(__floats2half2_rn(a, b), __float2half2_rn(0.0f));
    return *reinterpret_cast<const uint32_t*>(&h);
}

// BYTES: size of one cp.async of the mel rows; 16 where the rows lie on 16-byte boundaries, else 4 (a caller's feature
// buffer need only be aligned to its floats).
template <int BYTES>
__global__ void __launch_bounds__(256, 3)
sub_conv0_dw1_tc_kernel(const float* __restrict__ feats, const int64_t* __restrict__ t0_off, const int* __restrict__ t1_off,
                        const int* __restrict__ t2_off, const uint2* __restrict__ w0_frag, const __half2* __restrict__ w1h,
                        __nv_bfloat16* __restrict__ out, int steps) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmemLayout& sm = *reinterpret_cast<SmemLayout*>(smem_raw);
    const int clip = blockIdx.y, first = blockIdx.x * steps * kTO;
    const int out_base = t2_off[clip];
    const int T2 = t2_off[clip + 1] - out_base;
    if (first >= T2) return;
    const int end = min(T2, first + steps * kTO);
    const int64_t base = t0_off[clip];
    const int T = (int)(t0_off[clip + 1] - base);
    const int T1 = t1_off[clip + 1] - t1_off[clip];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // mel rows 4 to0 - 3 .. 4 to0 + 4 TO - 1, zero outside the clip; the columns beside the 128 are zeroed once
    auto fetch = [&](int to0, int buf) {
        constexpr int PF = BYTES / 4, PR = kMelBins / PF;  // floats per piece, pieces per row
        for (int i = tid; i < kNX * PR; i += 256) {
            const int row = i / PR, c = PF * (i % PR);
            const int r = 4 * to0 - 3 + row;
            const bool in = r >= 0 && r < T;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&sm.xs[buf][row][4 + c]);
            const float* src = feats + (base + (in ? r : 0)) * kMelBins + c;
            if constexpr (BYTES == 16)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
            else
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(in ? 4 : 0) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(first, 0);
    for (int i = tid; i < 2 * kNX * 8; i += 256) {
        const int c = i & 7;
        sm.xs[i / (kNX * 8)][(i >> 3) % kNX][c < 4 ? c : kMelBins + c] = 0.0f;
    }
    // column slot 0 of the first-stage tile is the zero padding left of frequency 0
    for (int i = tid; i < kNY * kY0Stride; i += 256) sm.y0[i / kY0Stride][0][i % kY0Stride] = __float2half(0.0f);

    const int g = lane >> 2, t = lane & 3;
    const uint32_t* im = reinterpret_cast<const uint32_t*>(&sm.im2col[0][0]);  // kImStride / 2 words per position
    const int quad = tid & 15, fg = tid >> 4;  // depthwise stage: four channels of the block, two output frequencies

    for (int to0 = first, buf = 0; to0 < end; to0 += kTO, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // the mel rows are in
        // im2col: position (first-stage row ry, frequency f) <- its 3 x 3 patch, then 1 (bias), then zeros
        for (int pos = tid; pos < kPos; pos += 256) {
            const int ry = pos >> 6, f = pos & 63;
            __align__(16) __half h[16];
#pragma unroll
            for (int dt = 0; dt < 3; ++dt)
#pragma unroll
                for (int df = 0; df < 3; ++df) h[3 * dt + df] = __float2half_rn(sm.xs[buf][2 * ry + dt][2 * f + df + 3]);
            h[9] = __float2half(1.0f);
#pragma unroll
            for (int k = 10; k < 16; ++k) h[k] = __float2half(0.0f);
            uint4* dst = reinterpret_cast<uint4*>(sm.im2col[pos]);
            dst[0] = *reinterpret_cast<const uint4*>(&h[0]);
            dst[1] = *reinterpret_cast<const uint4*>(&h[8]);
        }
        if (to0 + kTO < end) fetch(to0 + kTO, buf ^ 1);  // that buffer's readers are behind the barrier above
        __syncthreads();

        for (int zb = 0; zb < 4; ++zb) {
            // ---- first stage for channels 64 zb .. 64 zb + 63
            uint2 bfrag[8];
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) bfrag[nt] = __ldg(w0_frag + (zb * 8 + nt) * 32 + lane);
            for (int mt = warp; mt < kNY * 4; mt += 8) {
                const int ry = mt >> 2, f0 = (mt & 3) * 16;
                const int r = 2 * to0 - 1 + ry;
                uint4* dst0 = reinterpret_cast<uint4*>(&sm.y0[ry][f0 + g + 1][16 * t]);
                uint4* dst1 = reinterpret_cast<uint4*>(&sm.y0[ry][f0 + g + 9][16 * t]);
                if (r < 0 || r >= T1) {  // rows outside the first-stage map are the second stage's padding
                    dst0[0] = dst0[1] = dst1[0] = dst1[1] = make_uint4(0u, 0u, 0u, 0u);
                    continue;
                }
                const int p0 = ry * 64 + f0 + g;
                uint32_t a[4];
                a[0] = im[p0 * (kImStride / 2) + t];
                a[1] = im[(p0 + 8) * (kImStride / 2) + t];
                a[2] = im[p0 * (kImStride / 2) + 4 + t];
                a[3] = im[(p0 + 8) * (kImStride / 2) + 4 + t];
                uint32_t lo[8], hi[8];
#pragma unroll
                for (int nt = 0; nt < 8; ++nt) {
                    float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                    mma_f16(c, a, bfrag[nt]);
                    lo[nt] = relu_pack(c[0], c[1]);
                    hi[nt] = relu_pack(c[2], c[3]);
                }
                dst0[0] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                dst0[1] = make_uint4(lo[4], lo[5], lo[6], lo[7]);
                dst1[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                dst1[1] = make_uint4(hi[4], hi[5], hi[6], hi[7]);
            }
            __syncthreads();
            // ---- depthwise stage for the same channels
            {
                __half2 w[9][2], acc[kTO][2][2];
                auto pair_of = [&](int k) {
                    const uint2 v = __ldg(reinterpret_cast<const uint2*>(w1h + k * (kSubChannels / 2) + zb * 32) + quad);
                    return v;
                };
#pragma unroll
                for (int k = 0; k < 9; ++k) {
                    const uint2 v = pair_of(k);
                    w[k][0] = *reinterpret_cast<const __half2*>(&v.x);
                    w[k][1] = *reinterpret_cast<const __half2*>(&v.y);
                }
                const uint2 bv = pair_of(9);
#pragma unroll
                for (int j = 0; j < kTO; ++j)
#pragma unroll
                    for (int o = 0; o < 2; ++o) {
                        acc[j][o][0] = *reinterpret_cast<const __half2*>(&bv.x);
                        acc[j][o][1] = *reinterpret_cast<const __half2*>(&bv.y);
                    }
#pragma unroll
                for (int ry = 0; ry < kNY; ++ry) {
                    __half2 v[5][2];
#pragma unroll
                    for (int s = 0; s < 5; ++s) {
                        const uint2 x = *reinterpret_cast<const uint2*>(&sm.y0[ry][4 * fg + s][4 * quad]);
                        v[s][0] = *reinterpret_cast<const __half2*>(&x.x);
                        v[s][1] = *reinterpret_cast<const __half2*>(&x.y);
                    }
#pragma unroll
                    for (int j = 0; j < kTO; ++j) {
                        const int dt = ry - 2 * j;
                        if (dt < 0 || dt > 2) continue;
#pragma unroll
                        for (int o = 0; o < 2; ++o)
#pragma unroll
                            for (int df = 0; df < 3; ++df)
#pragma unroll
                                for (int e = 0; e < 2; ++e) acc[j][o][e] = __hfma2(w[3 * dt + df][e], v[2 * o + df][e], acc[j][o][e]);
                    }
                }
#pragma unroll
                for (int j = 0; j < kTO; ++j) {
                    if (to0 + j >= end) break;
                    __nv_bfloat16* orow = out + ((size_t)(out_base + to0 + j) * 32 + 2 * fg) * kSubChannels + zb * 64 + 4 * quad;
#pragma unroll
                    for (int o = 0; o < 2; ++o) {
                        const float2 f = __half22float2(acc[j][o][0]), h = __half22float2(acc[j][o][1]);
                        __align__(8) __nv_bfloat162 pk[2] = {__floats2bfloat162_rn(f.x, f.y), __floats2bfloat162_rn(h.x, h.y)};
                        *reinterpret_cast<uint2*>(orow + (size_t)o * kSubChannels) = *reinterpret_cast<const uint2*>(pk);
                    }
                }
            }
            __syncthreads();  // the tile is overwritten by the next channel block
        }
    }
}

}  // namespace

size_t subsample_frag_count() { return (size_t)4 * 8 * 32; }

// w0 [256 x 9] (channel-major, taps 3 dt + df), b0 [256] -> B fragments of mma.m16n8k16 for every channel tile:
// lane (g = lane >> 2, t = lane & 3) of tile (zb, nt) holds {k = 2t, 2t+1} and {k = 2t+8, 2t+9} of channel
// 64 zb + 16 (g / 2) + 2 nt + g % 2 (the kernel's lanes then hold neighbouring channels), with k < 9 the taps, k = 9 the bias (the im2col tile holds a 1 there) and zeros above.
void subsample_build_frags(const float* w0, const float* b0, uint2* frags) {
    for (int zb = 0; zb < 4; ++zb)
        for (int nt = 0; nt < 8; ++nt)
            for (int lane = 0; lane < 32; ++lane) {
                const int g = lane >> 2, t = lane & 3, ch = 64 * zb + 16 * (g >> 1) + 2 * nt + (g & 1);
                auto tap = [&](int k) { return k < 9 ? w0[ch * 9 + k] : (k == 9 ? b0[ch] : 0.0f); };
                const __half2 lo = __floats2half2_rn(tap(2 * t), tap(2 * t + 1));
                const __half2 hi = __floats2half2_rn(tap(2 * t + 8), tap(2 * t + 9));
                uint2 v;
                v.x = *reinterpret_cast<const uint32_t*>(&lo);
                v.y = *reinterpret_cast<const uint32_t*>(&hi);
                frags[(zb * 8 + nt) * 32 + lane] = v;
            }
}

// w1 tap-major [9 x 256] f32 and b1 [256] -> [10 x 128] fp16 pairs (row 9 = bias)
void subsample_build_dw(const float* w1_tap_major, const float* b1, uint32_t* out_pairs) {
    for (int k = 0; k < 10; ++k)
        for (int c2 = 0; c2 < kSubChannels / 2; ++c2) {
            const float a = k < 9 ? w1_tap_major[k * kSubChannels + 2 * c2] : b1[2 * c2];
            const float b = k < 9 ? w1_tap_major[k * kSubChannels + 2 * c2 + 1] : b1[2 * c2 + 1];
            const __half2 h = __floats2half2_rn(a, b);
            out_pairs[k * (kSubChannels / 2) + c2] = *reinterpret_cast<const uint32_t*>(&h);
        }
}

cudaError_t subsample_configure() {
    const cudaError_t e = cudaFuncSetAttribute(sub_conv0_dw1_tc_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemLayout));
    return e != cudaSuccess ? e
                            : cudaFuncSetAttribute(sub_conv0_dw1_tc_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemLayout));
}

cudaError_t subsample_conv0_dw1_launch(const float* feats, const int64_t* d_t0, const int* d_t1, const int* d_t2, int n_clips,
                                       int max_t2, const void* w0_frag, const void* w1_pairs, void* out, int sm_count, cudaStream_t st) {
    if (n_clips <= 0 || max_t2 <= 0) return cudaSuccess;
    // four steps of two rows per CTA while that leaves four CTAs for each of the three places on an SM
    const int pairs = (max_t2 + kTO - 1) / kTO;
    const int steps = (int64_t)pairs * n_clips >= (int64_t)4 * 12 * sm_count ? 4 : 1;
    const dim3 grid((pairs + steps - 1) / steps, n_clips);
    if (reinterpret_cast<uintptr_t>(feats) & 3) return cudaErrorMisalignedAddress;
    auto* kernel = reinterpret_cast<uintptr_t>(feats) & 15 ? sub_conv0_dw1_tc_kernel<4> : sub_conv0_dw1_tc_kernel<16>;
    kernel<<<grid, 256, sizeof(SmemLayout), st>>>(feats, d_t0, d_t1, d_t2, static_cast<const uint2*>(w0_frag),
                                                  static_cast<const __half2*>(w1_pairs), static_cast<__nv_bfloat16*>(out), steps);
    return cudaGetLastError();
}

}  // namespace sb
