// Cross-entropy over bf16 logits: row statistics, loss, and the gradient of the logits.
//
// All arithmetic is fp32 on the bf16 values that the head's matrix product left.  What
// bounds these kernels is reading the logits: 1.05 GB for 4096 rows of a 128256-word
// vocabulary, once for the statistics (275 us on a B200, 3.8 TB/s) and
// once, plus a write, for the gradient (344 us, 6.1 TB/s).  The statistics are bound by their
// exponentials: as ex2.approx of a rounded product they took 223 us, but off by up to 5e-6
// of their value where fp32 exp is off by 1e-7, and zero below 1.2e-38.  The PyTorch operations that
// they replace (fp32 copies of the logits, log-sum-exp, softmax, scatter, scaling, casts and
// an fp32 gradient of the head) took 11 ms for the same rows: a training step of two layers
// of the 8B shape went from 38.9 to 27.9 ms, one of four layers and eight micro-batches with
// offloaded state from 487 to 395 ms.
#include "common.cuh"
#include "loss_ops.h"

namespace oab {
namespace {

constexpr int64_t kIgnore = -100;

__device__ __forceinline__ void unpack16(const V8& r, float (&x)[16]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    x[2 * i] = __uint_as_float(r.w[i] << 16);
    x[2 * i + 1] = __uint_as_float(r.w[i] & 0xffff0000u);
  }
}
// what is subtracted from the row before exp: a row of only -inf has no finite maximum
__device__ __forceinline__ float shift_of(float m) { return m == -INFINITY ? 0.f : m; }

// (m, s) of a set of values: m = max, s = sum exp(x - m).  Joins two disjoint sets.
__device__ __forceinline__ void join(float& m, float& s, float m2, float s2) {
  const float mn = fmaxf(m, m2), sh = shift_of(mn);
  s = __fadd_rn(__fmul_rn(s, expf(__fsub_rn(m, sh))), __fmul_rn(s2, expf(__fsub_rn(m2, sh))));
  m = mn;
}

// One CTA per row, one pass over it: every thread keeps the maximum and the rescaled sum
// of what it has seen and rescales once per 32 values.
template <int THREADS>
__global__ void __launch_bounds__(THREADS)
ce_stats_kernel(const uint16_t* __restrict__ logits, int64_t pitch, const int64_t* __restrict__ labels, int64_t n,
                int64_t V, float* __restrict__ stats, volatile int64_t* bad_label) {
  __shared__ float sm_m[THREADS / 32], sm_s[THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t nvec = (V + 15) >> 4;
  for (int64_t row = blockIdx.x; row < n; row += gridDim.x) {
    const uint16_t* x = logits + row * pitch;
    float m = -INFINITY, s = 0.f;
    for (int64_t v = threadIdx.x; v < nvec; v += 2 * THREADS) {
      float e[2][16];
      const bool second = v + THREADS < nvec;
      {
        const V8 a = ld32(x + v * 16);
        V8 b = a;
        if (second) b = ld32(x + (v + THREADS) * 16);
        unpack16(a, e[0]);
        unpack16(b, e[1]);
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int64_t left = V - (v + k * THREADS) * 16;  // values of the vector inside the row
        if (left < 16) {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (i >= left) e[k][i] = -INFINITY;
        }
      }
      float mn = m;
#pragma unroll
      for (int i = 0; i < 16; ++i) mn = fmaxf(mn, fmaxf(e[0][i], e[1][i]));
      const float sh = shift_of(mn);
      s = __fmul_rn(s, expf(__fsub_rn(m, sh)));
      float t0 = 0.f, t1 = 0.f;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        t0 = __fadd_rn(t0, expf(__fsub_rn(e[0][i], sh)));
        t1 = __fadd_rn(t1, expf(__fsub_rn(e[1][i], sh)));
      }
      s = __fadd_rn(s, __fadd_rn(t0, second ? t1 : 0.f));
      m = mn;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
      join(m, s, m2, s2);
    }
    if (lane == 0) { sm_m[warp] = m; sm_s[warp] = s; }
    __syncthreads();
    if (warp == 0) {
      m = lane < THREADS / 32 ? sm_m[lane] : -INFINITY;
      s = lane < THREADS / 32 ? sm_s[lane] : 0.f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
        join(m, s, m2, s2);
      }
      if (lane == 0) {
        const int64_t lab = labels[row];
        const int64_t at = lab < 0 ? 0 : lab;
        // an infinite maximum is the log-sum-exp itself
        const float lse = isinf(m) ? m : __fadd_rn(m, logf(s));
        const float picked = at < V ? bf16_bits_to_f32(x[at]) : NAN;
        if (at >= V) *bad_label = at;
        stats[row] = m;
        stats[n + row] = at < V ? __fdiv_rn(1.0f, s) : NAN;
        stats[2 * n + row] = __fmul_rn(__fsub_rn(lse, picked), lab == kIgnore ? 0.f : 1.f);
      }
    }
    __syncthreads();  // sm_m / sm_s are rewritten for the next row
  }
}

__global__ void __launch_bounds__(1024)
ce_finish_kernel(const float* __restrict__ row_loss, const int64_t* __restrict__ labels, int64_t n, float* loss,
                 float* inv) {
  __shared__ float red[32];
  __shared__ int red_n[32];
  float s = 0.f;
  int c = 0;
  for (int64_t i = threadIdx.x; i < n; i += 1024) {
    c += labels[i] != kIgnore;
    if (row_loss != nullptr) s = __fadd_rn(s, row_loss[i]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) red_n[threadIdx.x >> 5] = c;
  s = block_sum<1024>(s, red);  // its barriers also publish red_n
  if (threadIdx.x == 0) {
    int total = 0;
    for (int w = 0; w < 32; ++w) total += red_n[w];
    const float r = __fdiv_rn(1.0f, (float)(total < 1 ? 1 : total));
    *inv = r;
    if (row_loss != nullptr) *loss = __fmul_rn(s, r);
  }
}

// Streaming pass: one 16-value vector per thread and iteration, grid.y CTAs share a row.
constexpr int kGradThreads = 256;
__global__ void __launch_bounds__(kGradThreads)
ce_grad_kernel(const uint16_t* logits, int64_t pitch, const int64_t* __restrict__ labels, int64_t n, int64_t V,
               const float* __restrict__ row_max, const float* __restrict__ row_inv_sum,
               const float* __restrict__ inv, const float* __restrict__ g, uint16_t* grad) {
  const int64_t nvec = (V + 15) >> 4;
  const float scale_all = g != nullptr ? __fmul_rn(*inv, *g) : *inv;
  for (int64_t row = blockIdx.x; row < n; row += gridDim.x) {
    const int64_t lab = labels[row];
    const float scale = lab == kIgnore ? 0.f : scale_all;
    const int64_t at = lab < 0 ? 0 : lab;
    const float sh = shift_of(row_max[row]), is = row_inv_sum[row];
    const uint16_t* x = logits + row * pitch;
    uint16_t* d = grad + row * pitch;
    for (int64_t v = (int64_t)blockIdx.y * kGradThreads + threadIdx.x; v < nvec; v += (int64_t)gridDim.y * kGradThreads) {
      float e[16];
      unpack16(ld32_stream(x + v * 16), e);
      const int64_t hit = at - v * 16;
      V8 o;
#pragma unroll
      for (int i = 0; i < 16; ++i) e[i] = __fmul_rn(expf(__fsub_rn(e[i], sh)), is);
      if (hit >= 0 && hit < 16) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
          if (i == hit) e[i] = __fsub_rn(e[i], 1.0f);
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) o.w[i] = f32x2_to_bf16x2_rne(__fmul_rn(e[2 * i], scale), __fmul_rn(e[2 * i + 1], scale));
      st32(d + v * 16, o);  // the pitch covers the last vector
    }
  }
}

// The gradient of the head over several groups of rows.  A mixed-type PyTorch add took 1.8 ms
// for the 525 M weights of a 128256 x 4096 head, next to a fill and a cast; this reads and
// writes each operand once in 256-bit accesses.  Loss and gradients of 16384 tokens: 46.9 ms
// with the adds, 41.3 ms now; 8192 tokens, which now are one group, 24.0 and 19.0 ms.
template <bool ACC32, bool OUT32>
__global__ void __launch_bounds__(kGradThreads)
sum_bf16_kernel(const void* acc, const uint16_t* g, float* out32, uint16_t* out16, int64_t n) {
  const int64_t i = ((int64_t)blockIdx.x * kGradThreads + threadIdx.x) * 16;
  if (i >= n) return;
  if (i + 16 > n) {
    for (int64_t j = i; j < n; ++j) {
      const float a = ACC32 ? reinterpret_cast<const float*>(acc)[j] : bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(acc)[j]);
      const float v = __fadd_rn(a, bf16_bits_to_f32(g[j]));
      if (OUT32) out32[j] = v;
      else out16[j] = (uint16_t)f32_to_bf16_rne_bits(v);
    }
    return;
  }
  float a[16], b[16];
  unpack16(ld32_stream(g + i), b);
  if (ACC32) {
    const float* p = reinterpret_cast<const float*>(acc) + i;
    const V8 lo = ld32_stream(p), hi = ld32_stream(p + 8);
#pragma unroll
    for (int k = 0; k < 8; ++k) { a[k] = __uint_as_float(lo.w[k]); a[8 + k] = __uint_as_float(hi.w[k]); }
  } else {
    unpack16(ld32_stream(reinterpret_cast<const uint16_t*>(acc) + i), a);
  }
#pragma unroll
  for (int k = 0; k < 16; ++k) a[k] = __fadd_rn(a[k], b[k]);
  V8 lo, hi;
  if (OUT32) {
#pragma unroll
    for (int k = 0; k < 8; ++k) { lo.w[k] = __float_as_uint(a[k]); hi.w[k] = __float_as_uint(a[8 + k]); }
    st32(out32 + i, lo);
    st32(out32 + i + 8, hi);
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) lo.w[k] = f32x2_to_bf16x2_rne(a[2 * k], a[2 * k + 1]);
    st32(out16 + i, lo);
  }
}

bool ce_args_ok(const void* logits, int64_t pitch, int64_t V) {
  return (reinterpret_cast<uintptr_t>(logits) & 31u) == 0 && pitch % kCePitchAlign == 0 && pitch >= V;
}

}  // namespace

cudaError_t launch_ce_stats(const void* logits, int64_t pitch, const int64_t* labels, int64_t n, int64_t V,
                            float* stats, int64_t* bad_label, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (bad_label == nullptr || V <= 0 || !ce_args_ok(logits, pitch, V)) return cudaErrorInvalidValue;
  const unsigned grid = (unsigned)(n < (int64_t(1) << 30) ? n : (int64_t(1) << 30));
  count_launch();
  // a thread should have at least one pair of vectors: short rows take small CTAs
  if (V <= 128 * 64)
    ce_stats_kernel<128><<<grid, 128, 0, st>>>((const uint16_t*)logits, pitch, labels, n, V, stats, bad_label);
  else
    ce_stats_kernel<512><<<grid, 512, 0, st>>>((const uint16_t*)logits, pitch, labels, n, V, stats, bad_label);
  return cudaGetLastError();
}

cudaError_t launch_ce_finish(const float* row_loss, const int64_t* labels, int64_t n, float* loss, float* inv,
                             cudaStream_t st) {
  if (n > (int64_t(1) << 30)) return cudaErrorInvalidValue;
  count_launch();
  ce_finish_kernel<<<1, 1024, 0, st>>>(row_loss, labels, n, loss, inv);
  return cudaGetLastError();
}

cudaError_t launch_ce_grad(const void* logits, int64_t pitch, const int64_t* labels, int64_t n, int64_t V,
                           const float* row_max, const float* row_inv_sum, const float* inv, const float* g,
                           void* grad, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  if (V <= 0 || !ce_args_ok(logits, pitch, V) || !ce_args_ok(grad, pitch, V)) return cudaErrorInvalidValue;
  const int64_t nvec = (V + 15) / 16;
  // up to four vectors per thread and CTA: short-lived CTAs keep every SM busy to the end
  int64_t gy = (nvec + kGradThreads * 4 - 1) / (kGradThreads * 4);
  if (gy > 65535) gy = 65535;
  dim3 grid((unsigned)(n < (int64_t(1) << 30) ? n : (int64_t(1) << 30)), (unsigned)gy);
  count_launch();
  ce_grad_kernel<<<grid, kGradThreads, 0, st>>>((const uint16_t*)logits, pitch, labels, n, V, row_max, row_inv_sum, inv,
                                               g, (uint16_t*)grad);
  return cudaGetLastError();
}

cudaError_t launch_sum_bf16(const void* acc, bool acc_is_f32, const void* g, float* out_f32, void* out_bf16, int64_t n,
                            cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const uintptr_t all = reinterpret_cast<uintptr_t>(acc) | reinterpret_cast<uintptr_t>(g) |
                        reinterpret_cast<uintptr_t>(out_f32) | reinterpret_cast<uintptr_t>(out_bf16);
  const int64_t grid = (n + kGradThreads * 16 - 1) / (kGradThreads * 16);
  if ((all & 31u) || grid >= (int64_t(1) << 31) || (out_f32 == nullptr) == (out_bf16 == nullptr)) return cudaErrorInvalidValue;
  const uint16_t* gp = (const uint16_t*)g;
  uint16_t* o16 = (uint16_t*)out_bf16;
  count_launch();
  if (acc_is_f32 && out_f32) sum_bf16_kernel<true, true><<<(unsigned)grid, kGradThreads, 0, st>>>(acc, gp, out_f32, o16, n);
  else if (acc_is_f32) sum_bf16_kernel<true, false><<<(unsigned)grid, kGradThreads, 0, st>>>(acc, gp, out_f32, o16, n);
  else if (out_f32) sum_bf16_kernel<false, true><<<(unsigned)grid, kGradThreads, 0, st>>>(acc, gp, out_f32, o16, n);
  else sum_bf16_kernel<false, false><<<(unsigned)grid, kGradThreads, 0, st>>>(acc, gp, out_f32, o16, n);
  return cudaGetLastError();
}

}  // namespace oab
