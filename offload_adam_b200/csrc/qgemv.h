// Host-side launch interface of the few-token linear kernels on packed weights (qgemv.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace oab {

constexpr int kQGemvMaxTokens = 4;

// True when launch_qgemv takes the shape: NVFP4, NF4 (block size `group`) or int8 with
// columns in whole vectors of 16, 1..kQGemvMaxTokens tokens; int4 (group size `group`) with
// columns in units of 128, at least 1024 rows, 1..2 tokens.  Inside these limits the kernel
// beats the dense route on a B200 (microseconds, 14336 x 4096 / 4096 x 4096 / 256 x 14336; the
// dense route takes 53 / 29 / 25):
//            1 token        2 tokens       4 tokens       5..8 tokens
//   NF4      26 / 15 / 12   30 / 16 / 12   48 / 27 / 12   78 / 43 / 34, not taken
//   NVFP4    19 / 10 / 10   27 / 16 / 10   43 / 25 / 12   78 / 43 / 34, not taken
//   int8     19 / 11 / 10   28 / 16 / 10   41 / 25 / 12   76 / 43 / 34, not taken
//   int4     27 / 12 / 26   32 / 14 / 32   59 / 24 / 66, not taken
bool qgemv_supported(int format, int64_t rows, int64_t cols, int64_t tokens, int group);

// y (tokens, rows) = x (tokens, cols) W^T + bias, all bf16 and contiguous, sums in fp32.
// `packed` / `scales` / `global_scale` as the format stores them (quant.h); int4 and int8
// scales are bf16.  x 32-byte aligned, packed aligned to qgemv_packed_align.  bias may be null.
constexpr uintptr_t qgemv_packed_align(int format) {
  return format == 4 ? 16 : (format == 3 ? 4 : 8);  // int8, int4, others
}
cudaError_t launch_qgemv(int format, const void* packed, const void* scales, const float* global_scale, int group,
                         const void* x, int64_t tokens, const void* bias, void* y, int64_t rows, int64_t cols,
                         cudaStream_t st);

}  // namespace oab
