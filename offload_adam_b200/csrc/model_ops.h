// Host-side launch interface of the elementwise model kernels (model_ops.cu): bf16 in and
// out, fp32 inside, one rounding per result.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace oab {

// y = silu(g) * u
cudaError_t launch_swiglu(const void* g, const void* u, void* y, int64_t n, cudaStream_t st);
// gg = gy * u * silu'(g), gu = gy * silu(g)
cudaError_t launch_swiglu_grad(const void* gy, const void* g, const void* u, void* gg, void* gu, int64_t n,
                               cudaStream_t st);

// A (batch, seq, heads, dim) tensor of bf16 with unit stride along dim; strides in elements.
struct RopeTensor {
  const void* in = nullptr;
  void* out = nullptr;  // contiguous
  int64_t sb = 0, ss = 0, sh = 0;
  int heads = 0;
};
// Rotates the heads of q and k (either may have 0 heads) by the tables cos / sin
// (seq, dim): out[i] = x[i] cos[i] - x[i + d/2] sin[i] for the first half of dim,
// out[i] = x[i] cos[i] + x[i - d/2] sin[i] for the second; the transpose of that when
// `transposed`.  dim % 16 == 0; bases and strides 16-byte aligned.
cudaError_t launch_rope(const RopeTensor& q, const RopeTensor& k, const void* cos, const void* sin, int64_t batch,
                        int64_t seq, int dim, bool transposed, cudaStream_t st);

// RMSNorm of rows of `cols` bf16 values (cols % 8 == 0, cols <= kNormMaxCols, 16-byte aligned):
// sum = bf16(x + r) when r is given (else the row is x itself and `sum` is not written),
// out = bf16(row * rstd * w) with rstd[i] = 1 / sqrt(mean(row^2) + eps).
constexpr int kNormMaxCols = 16384;
cudaError_t launch_rms_norm(const void* x, const void* r, const void* w, void* sum, void* out, float* rstd,
                            int64_t rows, int cols, float eps, cudaStream_t st);

// Gradients: dx = bf16(rstd (g w - xhat mean(g w xhat)) + gsum), xhat = x rstd; gsum (the
// gradient of `sum`) may be null.  dw = bf16(sum over rows of g xhat) through `partials`,
// rms_norm_partials(rows, cols) * cols floats; dw may be null.  Fixed summation order.
cudaError_t launch_rms_norm_grad(const void* g, const void* gsum, const void* x, const void* w, const float* rstd,
                                 void* dx, void* dw, float* partials, int64_t rows, int cols, cudaStream_t st);
int rms_norm_partials(int64_t rows, int cols);

// Gradient of an embedding table: dw (vocab, cols) = for every row the sum of the rows of
// g (n, cols) whose ids name it, zero for the others.  cols % 8 == 0, n <= kEmbedMaxTokens,
// vocab < 2^31; ids outside the table are ignored.  `work`: embed_work_ints(n, vocab) ints.
// Sums in fp32, in a fixed order.
constexpr int64_t kEmbedMaxTokens = 24576;
// Whether this beats PyTorch's gradient (fill, sort, partial sums, scatter).  Finding the
// tokens of a row compares every token with every other; what it saves is passes over the
// table.  Microseconds on a B200, ids uniform / skewed towards few rows, then
// PyTorch's for the skewed ones:
//   table           4096 tokens        12288               16384               24576
//   1024 x 256      55 /  56, 139      114 / 138, 144      148 / 177, 150      294 / 347, 164
//   8192 x 1024     49 /  48, 175      110 / 135, 223      141 / 174, 234      291 / 341, 268
//   128256 x 1024   83 /  96, 255      163 / 207, 350      196 / 251, 401      355 / 439, 501
//   32000 x 4096   108 / 134, 391      212 / 262, 762      252 / 316, 935      405 / 511, 1257
inline bool embed_kernel_wins(int64_t n, int64_t vocab, int64_t cols) {
  const int64_t table = vocab * cols;
  return n <= 12288 || (n <= 16384 && table >= 8000000) || (n <= kEmbedMaxTokens && table >= 100000000);
}
int64_t embed_work_ints(int64_t n, int64_t vocab);
cudaError_t launch_embed_grad(const void* g, const int64_t* ids, int64_t n, void* dw, int64_t vocab, int cols, int* work,
                              cudaStream_t st);

}  // namespace oab
