// Host-side launch interface of the few-token linear kernels on packed weights (qgemv.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace oab {

constexpr int kQGemvMaxTokens = 8;

// True when launch_qgemv takes the shape: NVFP4, NF4 (block size `group`) or int8, columns
// in whole vectors of 16, 1..8 tokens.
bool qgemv_supported(int format, int64_t rows, int64_t cols, int64_t tokens, int group);

// y (tokens, rows) = x (tokens, cols) W^T + bias, all bf16 and contiguous, sums in fp32.
// `packed` / `scales` / `global_scale` as the format stores them (quant.h); int8 scales are
// bf16.  x 32-byte aligned, packed 8-byte (int8: 16-byte) aligned.  bias may be null.
constexpr uintptr_t qgemv_packed_align(int format) { return format == 4 ? 16 : 8; }  // int8, others
cudaError_t launch_qgemv(int format, const void* packed, const void* scales, const float* global_scale, int group,
                         const void* x, int64_t tokens, const void* bias, void* y, int64_t rows, int64_t cols,
                         cudaStream_t st);

}  // namespace oab
