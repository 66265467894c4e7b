// Host-side launch interface of the few-token linear kernels on packed weights (qgemv.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace oab {

constexpr int kQGemvMaxTokens = 4;

// True when launch_qgemv takes the shape: NVFP4, NF4 (block size `group`) or int8 with
// columns in whole vectors of 16, 1..kQGemvMaxTokens tokens; int4 (group size `group`) with
// columns in units of 128, at least 1024 rows, 1..2 tokens.  Inside these limits the kernel
// beats the dense route (de-quantization and a library product).  Microseconds of GPU time on a
// B200, replayed from a graph over weights of 0.4 GB, 14336 x 4096 / 4096 x 4096 / 256 x 14336;
// in the last column two launches of the most tokens a launch takes, then the dense route
// (the same for 5 and for 8 tokens):
//            1 token        2 tokens       4 tokens       twice as many, in two launches
//   NF4      19 /  8 /  6   24 / 12 /  6   39 / 21 /  7   77 / 40 / 12   dense 43 / 20 / 16
//   NVFP4    14 /  6 /  6   22 / 10 /  6   36 / 19 /  7   71 / 37 / 12   dense 44 / 20 / 16
//   int8     14 /  6 /  6   23 / 11 /  6   33 / 19 /  7   66 / 36 / 12   dense 48 / 20 / 16
//   int4     21 /  8 / -    25 /  9 / -                   50 / 17 / -    dense 47 / 20 / 16
// (NF4, 4 tokens, 4096 x 4096: even in a graph, called from Python 23 and 25.)
// Below 1024 rows int4 leaves SMs idle (a CTA takes 32 rows): 256 x 14336 took 26 us a call from
// Python, the dense route 25.
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
