// Tensor-core GEMM for the encoder / joint projections (see gemm.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "gemm_tile.h"

namespace sb {

struct GemmArgs {
    const void* a;           // [M x K] row-major, bf16 (or e4m3 when fp8)
    const void* w;           // [N x K] row-major (nn.Linear layout), same type
    const float* bias;       // [N] or null
    const float* row_scale;  // fp8 only: per-row activation scale [M], or null
    const float* col_scale;  // fp8 only: per-output-channel weight scale [N], or null
    const float* out_row_scale;  // kOutFp8: per-row scale of the e4m3 output [M]
    void* out;
    int M, N, K;
    int ldo;                 // leading dimension of out in elements
    int act;
    int out_mode;
    float alpha;
    bool fp8;
    bool w_resident;         // w was complete before the kernel ahead of this one in the stream was launched (model weights):
                             // it may be read before that kernel ends
};

// Process-wide switch for two-CTA 256 x 256 tiles: 0 never, 1 for the products that gain from them (default),
// 2 for every product with at least one such tile per pair of SMs.
void gemm_set_pair_tiles(int mode);
// One-time set-up (driver entry point for tensor maps, shared-memory opt-in).
cudaError_t gemm_configure(const char** why);
// Launches the tcgen05 GEMM on `stream`.  `d_error` is a device int that the kernel
// sets non-zero if a bounded wait ran out.  Returns cudaErrorInvalidValue for shapes
// the kernel does not cover (N % 128 != 0, K % 64 (bf16) / 128 (fp8) != 0).
cudaError_t gemm_launch(const GemmArgs& g, int sm_count, int* d_error, cudaStream_t stream);

}  // namespace sb
