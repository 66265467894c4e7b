// Elementwise parts of the decoder for sm_100a: SwiGLU and rotary embeddings, forward and
// backward.  Memory bound: each reads its inputs and writes its results once.
//
// Measured on a B200 for 4096 tokens of the 8B shape: SwiGLU 52 us forward (6.8 TB/s) and
// 85 us backward (6.9 TB/s), RoPE of 32 + 8 heads 19.5 us (4.3 TB/s) either way.  As PyTorch
// operations with their intermediate tensors they took 96 and 177 us, and about 170 us each
// way (negate, concatenate, two products and a sum for q and for k).
#include "common.cuh"
#include "model_ops.h"

namespace oab {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float lo_f32(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_f32(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// 1 / (1 + exp(-x)) with the approximate exponential and reciprocal (a few fp32 ulp; the
// results are rounded to bf16).  The non-ftz reciprocal keeps tiny values.
__device__ __forceinline__ float sigmoid(float x) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(__fadd_rn(1.0f, __expf(-x))));
  return r;
}
// x * sigmoid(x); for x = -inf this is -inf * 0 = NaN, as in x / (1 + exp(-x))
__device__ __forceinline__ float silu(float x) { return __fmul_rn(x, sigmoid(x)); }

__device__ __forceinline__ void silu_pair_grad(float gy, float g, float u, float& gg, float& gu) {
  const float s = sigmoid(g);
  gu = __fmul_rn(gy, __fmul_rn(g, s));
  gg = __fmul_rn(__fmul_rn(gy, u), __fmul_rn(s, __fmaf_rn(g, __fsub_rn(1.0f, s), 1.0f)));
}

// One 16-value vector per thread: nothing is reused, so short-lived CTAs (8 per SM) hide
// the latency and leave no long last wave.
__global__ void __launch_bounds__(kThreads)
swiglu_kernel(const uint16_t* __restrict__ g, const uint16_t* __restrict__ u, uint16_t* __restrict__ y, int64_t n,
              int vector_ok) {
  const int64_t i = ((int64_t)blockIdx.x * kThreads + threadIdx.x) * 16;
  if (vector_ok && i + 16 <= n) {
    const V8 a = ld32_stream(g + i), b = ld32_stream(u + i);
    V8 o;
#pragma unroll
    for (int w = 0; w < 8; ++w)
      o.w[w] = f32x2_to_bf16x2_rne(__fmul_rn(silu(lo_f32(a.w[w])), lo_f32(b.w[w])),
                                   __fmul_rn(silu(hi_f32(a.w[w])), hi_f32(b.w[w])));
    st32(y + i, o);
    return;
  }
  for (int64_t j = i; j < i + 16 && j < n; ++j)
    y[j] = (uint16_t)f32_to_bf16_rne_bits(__fmul_rn(silu(bf16_bits_to_f32(g[j])), bf16_bits_to_f32(u[j])));
}

__global__ void __launch_bounds__(kThreads)
swiglu_grad_kernel(const uint16_t* __restrict__ gy, const uint16_t* __restrict__ g, const uint16_t* __restrict__ u,
                   uint16_t* __restrict__ gg, uint16_t* __restrict__ gu, int64_t n, int vector_ok) {
  const int64_t i = ((int64_t)blockIdx.x * kThreads + threadIdx.x) * 16;
  if (vector_ok && i + 16 <= n) {
    const V8 c = ld32_stream(gy + i), a = ld32_stream(g + i), b = ld32_stream(u + i);
    V8 oa, ob;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      float ga0, gb0, ga1, gb1;
      silu_pair_grad(lo_f32(c.w[w]), lo_f32(a.w[w]), lo_f32(b.w[w]), ga0, gb0);
      silu_pair_grad(hi_f32(c.w[w]), hi_f32(a.w[w]), hi_f32(b.w[w]), ga1, gb1);
      oa.w[w] = f32x2_to_bf16x2_rne(ga0, ga1);
      ob.w[w] = f32x2_to_bf16x2_rne(gb0, gb1);
    }
    st32(gg + i, oa);
    st32(gu + i, ob);
    return;
  }
  for (int64_t j = i; j < i + 16 && j < n; ++j) {
    float a, b;
    silu_pair_grad(bf16_bits_to_f32(gy[j]), bf16_bits_to_f32(g[j]), bf16_bits_to_f32(u[j]), a, b);
    gg[j] = (uint16_t)f32_to_bf16_rne_bits(a);
    gu[j] = (uint16_t)f32_to_bf16_rne_bits(b);
  }
}

// One thread rotates 8 values of the first half of a head with their partners in the
// second: two 16-byte loads and stores per operand.  The threads of a CTA walk the heads
// of one position after another, so a table row is read from DRAM once and from L1 after.
struct RopeArgs {
  RopeTensor q, k;
  const uint16_t *cos, *sin;
  int64_t seq, items;  // items = batch * seq * (q.heads + k.heads) * (dim / 16)
  int dim, per_head, per_token;
};

template <bool TRANSPOSED>
__global__ void __launch_bounds__(kThreads) rope_kernel(RopeArgs a) {
  const int64_t i = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (i >= a.items) return;
  const int64_t token = i / a.per_token;
  const int r = (int)(i - token * a.per_token);
  int head = r / a.per_head;
  const int col = (r - head * a.per_head) * 8, half = a.dim >> 1;
  const int64_t b = token / a.seq, s = token - b * a.seq;
  const bool is_q = head < a.q.heads;
  if (!is_q) head -= a.q.heads;
  const RopeTensor& t = is_q ? a.q : a.k;
  const uint16_t* x = (const uint16_t*)t.in + b * t.sb + s * t.ss + head * t.sh + col;
  uint16_t* y = (uint16_t*)t.out + (token * t.heads + head) * a.dim + col;
  const uint16_t *c = a.cos + s * a.dim + col, *n = a.sin + s * a.dim + col;
  const uint4 x1 = *reinterpret_cast<const uint4*>(x), x2 = *reinterpret_cast<const uint4*>(x + half);
  const uint4 c1 = __ldg(reinterpret_cast<const uint4*>(c)), c2 = __ldg(reinterpret_cast<const uint4*>(c + half));
  const uint4 n1 = __ldg(reinterpret_cast<const uint4*>(n)), n2 = __ldg(reinterpret_cast<const uint4*>(n + half));
  const uint32_t X1[4] = {x1.x, x1.y, x1.z, x1.w}, X2[4] = {x2.x, x2.y, x2.z, x2.w};
  const uint32_t C1[4] = {c1.x, c1.y, c1.z, c1.w}, C2[4] = {c2.x, c2.y, c2.z, c2.w};
  const uint32_t N1[4] = {n1.x, n1.y, n1.z, n1.w}, N2[4] = {n2.x, n2.y, n2.z, n2.w};
  uint32_t o1[4], o2[4];
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    float p[2], q[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float a1 = h ? hi_f32(X1[w]) : lo_f32(X1[w]), a2 = h ? hi_f32(X2[w]) : lo_f32(X2[w]);
      const float k1 = h ? hi_f32(C1[w]) : lo_f32(C1[w]), k2 = h ? hi_f32(C2[w]) : lo_f32(C2[w]);
      const float s1 = h ? hi_f32(N1[w]) : lo_f32(N1[w]), s2 = h ? hi_f32(N2[w]) : lo_f32(N2[w]);
      if (TRANSPOSED) {
        p[h] = __fmaf_rn(a2, s2, __fmul_rn(a1, k1));
        q[h] = __fmaf_rn(-a1, s1, __fmul_rn(a2, k2));
      } else {
        p[h] = __fmaf_rn(-a2, s1, __fmul_rn(a1, k1));
        q[h] = __fmaf_rn(a1, s2, __fmul_rn(a2, k2));
      }
    }
    o1[w] = f32x2_to_bf16x2_rne(p[0], p[1]);
    o2[w] = f32x2_to_bf16x2_rne(q[0], q[1]);
  }
  *reinterpret_cast<uint4*>(y) = make_uint4(o1[0], o1[1], o1[2], o1[3]);
  *reinterpret_cast<uint4*>(y + half) = make_uint4(o2[0], o2[1], o2[2], o2[3]);
}

bool aligned(const void* p, uintptr_t to) { return (reinterpret_cast<uintptr_t>(p) & (to - 1)) == 0; }
bool rope_ok(const RopeTensor& t) {
  return t.heads == 0 || (t.in != nullptr && t.out != nullptr && aligned(t.in, 16) && aligned(t.out, 16) &&
                          t.sb % 8 == 0 && t.ss % 8 == 0 && t.sh % 8 == 0);
}
constexpr int64_t kMaxGrid = int64_t(1) << 31;

}  // namespace

cudaError_t launch_swiglu(const void* g, const void* u, void* y, int64_t n, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int64_t grid = (n + kThreads * 16 - 1) / (kThreads * 16);
  if (grid >= kMaxGrid) return cudaErrorInvalidValue;
  count_launch();
  swiglu_kernel<<<(unsigned)grid, kThreads, 0, st>>>((const uint16_t*)g, (const uint16_t*)u, (uint16_t*)y, n,
                                                    aligned(g, 32) && aligned(u, 32) && aligned(y, 32));
  return cudaGetLastError();
}

cudaError_t launch_swiglu_grad(const void* gy, const void* g, const void* u, void* gg, void* gu, int64_t n,
                               cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int64_t grid = (n + kThreads * 16 - 1) / (kThreads * 16);
  if (grid >= kMaxGrid) return cudaErrorInvalidValue;
  count_launch();
  swiglu_grad_kernel<<<(unsigned)grid, kThreads, 0, st>>>(
      (const uint16_t*)gy, (const uint16_t*)g, (const uint16_t*)u, (uint16_t*)gg, (uint16_t*)gu, n,
      aligned(gy, 32) && aligned(g, 32) && aligned(u, 32) && aligned(gg, 32) && aligned(gu, 32));
  return cudaGetLastError();
}

cudaError_t launch_rope(const RopeTensor& q, const RopeTensor& k, const void* cos, const void* sin, int64_t batch,
                        int64_t seq, int dim, bool transposed, cudaStream_t st) {
  if (dim <= 0 || dim % 16 != 0 || !rope_ok(q) || !rope_ok(k) || !aligned(cos, 16) || !aligned(sin, 16))
    return cudaErrorInvalidValue;
  RopeArgs a{q, k, (const uint16_t*)cos, (const uint16_t*)sin, seq, 0, dim, dim / 16, (q.heads + k.heads) * (dim / 16)};
  a.items = batch * seq * a.per_token;
  if (a.items <= 0) return cudaSuccess;
  const int64_t grid = (a.items + kThreads - 1) / kThreads;
  if (grid >= kMaxGrid) return cudaErrorInvalidValue;
  count_launch();
  if (transposed) rope_kernel<true><<<(unsigned)grid, kThreads, 0, st>>>(a);
  else rope_kernel<false><<<(unsigned)grid, kThreads, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace oab
