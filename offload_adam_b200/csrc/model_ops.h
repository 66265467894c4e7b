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
constexpr int64_t kEmbedMaxTokens = 32768;
int64_t embed_work_ints(int64_t n, int64_t vocab);
cudaError_t launch_embed_grad(const void* g, const int64_t* ids, int64_t n, void* dw, int64_t vocab, int cols, int* work,
                              cudaStream_t st);

}  // namespace oab
