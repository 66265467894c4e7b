// Host-side launch interface of the cross-entropy kernels (loss_ops.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace oab {

// Row pitch, in elements, of a logits buffer: rows start 32-byte aligned.
constexpr int kCePitchAlign = 16;

// Per row of bf16 `logits` (n rows of V values, `pitch` elements apart, base 32-byte
// aligned, pitch % 16 == 0): stats[i] = max, stats[n + i] = 1 / sum exp(x - max),
// stats[2n + i] = loss of the row against labels[i] (0 for labels[i] == -100; negative
// labels otherwise count as class 0).  A label >= V gives NaN and is written to *bad_label
// (memory that the host reads), which is otherwise left alone.
cudaError_t launch_ce_stats(const void* logits, int64_t pitch, const int64_t* labels, int64_t n, int64_t V,
                            float* stats, int64_t* bad_label, cudaStream_t st);

// inv[0] = 1 / max(1, number of labels != -100); loss[0] = inv * sum(row_loss[0..n)) when
// row_loss is given, else only inv is written.  Fixed summation order.
cudaError_t launch_ce_finish(const float* row_loss, const int64_t* labels, int64_t n, float* loss, float* inv,
                             cudaStream_t st);

// grad[i, j] = bf16((softmax(logits[i])[j] - [j == labels[i]]) * inv * g), rows with label
// -100 times 0.  `grad` has the pitch of `logits` and may be the same buffer.  `g` may be
// null (1).
cudaError_t launch_ce_grad(const void* logits, int64_t pitch, const int64_t* labels, int64_t n, int64_t V,
                           const float* row_max, const float* row_inv_sum, const float* inv, const float* g,
                           void* grad, cudaStream_t st);

// Sum of bf16 tensors in fp32, one after another: value = acc + g with acc bf16
// (acc_is_f32 false) or fp32; written to out_f32 (may be acc) or, rounded, to out_bf16.
// All 32-byte aligned.
cudaError_t launch_sum_bf16(const void* acc, bool acc_is_f32, const void* g, float* out_f32, void* out_bf16, int64_t n,
                            cudaStream_t st);

}  // namespace oab
