// Elementwise parts of the decoder for sm_100a: SwiGLU and rotary embeddings, forward and
// backward.  Memory bound: each reads its inputs and writes its results once.
//
// Measured on a B200 for 4096 tokens of the 8B shape: SwiGLU 52 us forward (6.8 TB/s) and
// 85 us backward (6.9 TB/s), RoPE of 32 + 8 heads 19.5 us (4.3 TB/s) either way.  As PyTorch
// operations with their intermediate tensors they took 96 and 177 us, and about 170 us each
// way (negate, concatenate, two products and a sum for q and for k).
#include <climits>

#include "common.cuh"
#include "model_ops.h"

namespace oab {
namespace {

constexpr int kThreads = 256;

__device__ __forceinline__ float lo_f32(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_f32(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// fp32 exp and division: the kernels are bound by memory, and approximate ones (error growing
// with |x|) took the same time (forward 55.0 us, now 55.5; backward 89.5 and 89.7).
__device__ __forceinline__ float sigmoid(float x) { return __fdiv_rn(1.0f, __fadd_rn(1.0f, expf(-x))); }
// for x = -inf this is -inf / inf = NaN, as in PyTorch
__device__ __forceinline__ float silu(float x) { return __fdiv_rn(x, __fadd_rn(1.0f, expf(-x))); }

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

// -------------------------------------------------------------------- RMSNorm
// LANES threads share a row (32: a warp, 256: a CTA) and hold it in registers, VPT vectors
// of 8 values each, so that every operand is read once.  Measured on a B200 for 4096 rows of
// 4096: 12 us forward, 23 us with the sum in front (5.9 TB/s; as two operations 30 us), 23 and
// 28 us backward plus 7 us for the weight gradient (as three operations 65 us).
__device__ __forceinline__ void unpack8(const uint4& r, float (&x)[8]) {
  const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) { x[2 * i] = lo_f32(w[i]); x[2 * i + 1] = hi_f32(w[i]); }
}
__device__ __forceinline__ uint4 pack8(const float (&x)[8]) {
  return make_uint4(f32x2_to_bf16x2_rne(x[0], x[1]), f32x2_to_bf16x2_rne(x[2], x[3]), f32x2_to_bf16x2_rne(x[4], x[5]),
                    f32x2_to_bf16x2_rne(x[6], x[7]));
}
// Sum over the LANES threads of a row, in all of them.  `red`: kThreads / 32 floats, two
// sets used in turn, so that one barrier per call is enough.
template <int LANES>
__device__ __forceinline__ float row_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (LANES == 32) return v;
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[0];
#pragma unroll
  for (int i = 1; i < kThreads / 32; ++i) v = __fadd_rn(v, red[i]);
  return v;
}

template <int LANES, int VPT, bool ADD>
__global__ void __launch_bounds__(kThreads)
rms_norm_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ r, const uint16_t* __restrict__ w,
                uint16_t* __restrict__ sum, uint16_t* __restrict__ out, float* __restrict__ rstd, int64_t rows, int cols,
                float eps) {
  __shared__ float red[kThreads / 32];
  const int lane = threadIdx.x % LANES, nvec = cols >> 3;
  const int64_t row = (int64_t)blockIdx.x * (kThreads / LANES) + threadIdx.x / LANES;
  if (row >= rows) return;  // whole warps (LANES == 32) or the whole CTA
  const int64_t base = row * cols;
  float e[VPT][8];
  float ss = 0.f;
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int v = lane + k * LANES;
    if (v >= nvec) continue;
    unpack8(*reinterpret_cast<const uint4*>(x + base + v * 8), e[k]);
    if (ADD) {
      float a[8];
      unpack8(*reinterpret_cast<const uint4*>(r + base + v * 8), a);
#pragma unroll
      for (int i = 0; i < 8; ++i) a[i] = __fadd_rn(e[k][i], a[i]);
      const uint4 packed = pack8(a);
      *reinterpret_cast<uint4*>(sum + base + v * 8) = packed;
      unpack8(packed, e[k]);  // the norm is of the rounded sum, which the residual stream keeps
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) ss = __fmaf_rn(e[k][i], e[k][i], ss);
  }
  ss = row_sum<LANES>(ss, red);
  const float rs = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, (float)cols), eps)));
  if (lane == 0) rstd[row] = rs;
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int v = lane + k * LANES;
    if (v >= nvec) continue;
    float wv[8];
    unpack8(__ldg(reinterpret_cast<const uint4*>(w + v * 8)), wv);
#pragma unroll
    for (int i = 0; i < 8; ++i) wv[i] = __fmul_rn(__fmul_rn(e[k][i], rs), wv[i]);
    *reinterpret_cast<uint4*>(out + base + v * 8) = pack8(wv);
  }
}

// Every group of LANES threads walks rows with stride `groups` and keeps its share of the
// weight gradient in registers; one row of partial sums per group goes to memory.
template <int LANES, int VPT, bool GSUM>
__global__ void __launch_bounds__(kThreads)
rms_norm_grad_kernel(const uint16_t* __restrict__ g, const uint16_t* __restrict__ gsum, const uint16_t* __restrict__ x,
                     const uint16_t* __restrict__ w, const float* __restrict__ rstd, uint16_t* __restrict__ dx,
                     float* __restrict__ partials, int64_t rows, int cols, int groups) {
  __shared__ float red[2][kThreads / 32];
  const int lane = threadIdx.x % LANES, nvec = cols >> 3;
  const int group = blockIdx.x * (kThreads / LANES) + threadIdx.x / LANES;
  if (group >= groups) return;  // whole warps or the whole CTA
  float acc[VPT][8];
#pragma unroll
  for (int k = 0; k < VPT; ++k)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[k][i] = 0.f;
  const float inv_cols = __fdiv_rn(1.0f, (float)cols);
  int turn = 0;
  for (int64_t row = group; row < rows; row += groups, turn ^= 1) {
    const int64_t base = row * cols;
    const float rs = rstd[row];
    uint4 gp[VPT], xp[VPT], sp[VPT];
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int v = lane + k * LANES;
      if (v >= nvec) continue;
      gp[k] = *reinterpret_cast<const uint4*>(g + base + v * 8);
      xp[k] = *reinterpret_cast<const uint4*>(x + base + v * 8);
      if (GSUM) sp[k] = *reinterpret_cast<const uint4*>(gsum + base + v * 8);
    }
    float c = 0.f;
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int v = lane + k * LANES;
      if (v >= nvec) continue;
      float gv[8], xv[8], wv[8];
      unpack8(gp[k], gv);
      unpack8(xp[k], xv);
      unpack8(__ldg(reinterpret_cast<const uint4*>(w + v * 8)), wv);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float h = __fmul_rn(xv[i], rs);
        acc[k][i] = __fmaf_rn(gv[i], h, acc[k][i]);
        c = __fmaf_rn(__fmul_rn(gv[i], wv[i]), h, c);
      }
    }
    c = __fmul_rn(row_sum<LANES>(c, red[turn]), inv_cols);
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int v = lane + k * LANES;
      if (v >= nvec) continue;
      float gv[8], xv[8], wv[8], o[8];
      unpack8(gp[k], gv);
      unpack8(xp[k], xv);
      unpack8(__ldg(reinterpret_cast<const uint4*>(w + v * 8)), wv);
      if (GSUM) unpack8(sp[k], o);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float d = __fmul_rn(rs, __fmaf_rn(-c, __fmul_rn(xv[i], rs), __fmul_rn(gv[i], wv[i])));
        o[i] = GSUM ? __fadd_rn(d, o[i]) : d;
      }
      *reinterpret_cast<uint4*>(dx + base + v * 8) = pack8(o);
    }
  }
  if (partials == nullptr) return;
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int v = lane + k * LANES;
    if (v >= nvec) continue;
    float4* p = reinterpret_cast<float4*>(partials + (int64_t)group * cols + v * 8);
    p[0] = make_float4(acc[k][0], acc[k][1], acc[k][2], acc[k][3]);
    p[1] = make_float4(acc[k][4], acc[k][5], acc[k][6], acc[k][7]);
  }
}

// dw[c] = sum over the groups, 32 columns per CTA: 8 threads a column, then their 8 sums.
__global__ void __launch_bounds__(kThreads)
column_sum_kernel(const float* __restrict__ partials, int groups, int cols, uint16_t* __restrict__ dw) {
  __shared__ float red[8][33];
  const int c = threadIdx.x & 31, part = threadIdx.x >> 5, col = blockIdx.x * 32 + c;
  float s = 0.f;
  if (col < cols) {
#pragma unroll 8
    for (int i = part; i < groups; i += 8) s = __fadd_rn(s, __ldg(partials + (int64_t)i * cols + col));
  }
  red[part][c] = s;
  __syncthreads();
  if (part == 0 && col < cols) {
#pragma unroll
    for (int i = 1; i < 8; ++i) s = __fadd_rn(s, red[i][c]);
    dw[col] = (uint16_t)f32_to_bf16_rne_bits(s);
  }
}

// ------------------------------------------------------------ embedding gradient
// The gradient is dense: writing it is the work (1.05 GB for a 128256 x 4096 table), so the
// kernel that writes the zero rows also sums the others, and no fill comes before it.  The
// tokens of a row are found by counting: with n ids on chip, the position of a token in
// sorted order is the number of smaller ids plus the number of equal ones before it.
// Measured on a B200 for 4096 tokens and a 128256 x 4096 table: 20 us to order, 217 us to write
// (4.8 TB/s of stores); PyTorch's fill, sort, partial sums and scatter took 750 us.
constexpr int kScanThreads = 256, kScanPer = 4;  // threads that share the scan of one token
constexpr int kScanTile = 2048;
constexpr int kLightRows = 8;  // rows named by more tokens than this are summed by a CTA

// order[position] = token; rows[id] = {first position, number of tokens}; ids that many
// tokens share are appended to `heavy` (in any order).
__global__ void __launch_bounds__(kScanThreads)
embed_order_kernel(const int64_t* __restrict__ ids, int n, int vocab, int* __restrict__ order, int2* __restrict__ rows,
                   int* __restrict__ heavy, int* n_heavy) {
  __shared__ int tile[kScanTile];
  const int t = blockIdx.x * (kScanThreads / kScanPer) + threadIdx.x / kScanPer, part = threadIdx.x % kScanPer;
  auto get = [&](int i) {
    const int64_t v = ids[i];
    return v < 0 || v >= vocab ? INT_MAX : (int)v;
  };
  const int id = t < n ? get(t) : INT_MAX;
  int less = 0, before = 0, equal = 0;
  for (int base = 0; base < n; base += kScanTile) {
    __syncthreads();
    for (int i = threadIdx.x; i < kScanTile; i += kScanThreads) tile[i] = base + i < n ? get(base + i) : INT_MAX;
    __syncthreads();
#pragma unroll 8
    for (int i = part; i < kScanTile; i += kScanPer) {
      const int v = tile[i];
      less += v < id;
      equal += v == id;
      before += v == id && base + i < t;
    }
  }
#pragma unroll
  for (int o = 1; o < kScanPer; o <<= 1) {
    less += __shfl_xor_sync(0xffffffffu, less, o);
    before += __shfl_xor_sync(0xffffffffu, before, o);
    equal += __shfl_xor_sync(0xffffffffu, equal, o);
  }
  if (part != 0 || id == INT_MAX) return;  // past the end, or no row of the table
  order[less + before] = t;
  if (before == 0) {
    rows[id] = make_int2(less, equal);
    if (equal > kLightRows) heavy[atomicAdd(n_heavy, 1)] = id;
  }
}

// A warp writes a row: zeros, or the sum of up to kLightRows gradients.
__global__ void __launch_bounds__(kThreads)
embed_rows_kernel(const uint16_t* __restrict__ g, const int* __restrict__ order, const int2* __restrict__ rows,
                  uint16_t* __restrict__ dw, int64_t vocab, int cols) {
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * (kThreads / 32);
  for (int64_t row = (int64_t)blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5); row < vocab; row += stride) {
    const int2 r = __ldg(rows + row);
    uint16_t* out = dw + row * cols;
    if (r.y == 0) {
#pragma unroll 4
      for (int col = lane * 8; col < cols; col += 256) *reinterpret_cast<uint4*>(out + col) = make_uint4(0, 0, 0, 0);
    } else if (r.y <= kLightRows) {
#pragma unroll 2
      for (int col = lane * 8; col < cols; col += 256) {
        float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        for (int i = 0; i < r.y; ++i) {
          float e[8];
          unpack8(*reinterpret_cast<const uint4*>(g + (int64_t)__ldg(order + r.x + i) * cols + col), e);
#pragma unroll
          for (int k = 0; k < 8; ++k) acc[k] = __fadd_rn(acc[k], e[k]);
        }
        *reinterpret_cast<uint4*>(out + col) = pack8(acc);
      }
    }
  }
}

// A CTA sums 256 columns of a row that many tokens share: eight warps, every eighth token
// each, four loads in flight.  Grids of any size finish the list.
__global__ void __launch_bounds__(kThreads)
embed_heavy_kernel(const uint16_t* __restrict__ g, const int* __restrict__ order, const int2* __restrict__ rows,
                   const int* __restrict__ heavy, const int* __restrict__ n_heavy, uint16_t* __restrict__ dw, int cols) {
  __shared__ float part[kThreads / 32][256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, col = blockIdx.y * 256 + lane * 8;
  const int count = *n_heavy;
  for (int h = blockIdx.x; h < count; h += gridDim.x) {
    const int row = heavy[h];
    const int2 r = rows[row];
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (col < cols) {
#pragma unroll 4
      for (int i = warp; i < r.y; i += kThreads / 32) {
        float e[8];
        unpack8(*reinterpret_cast<const uint4*>(g + (int64_t)__ldg(order + r.x + i) * cols + col), e);
#pragma unroll
        for (int k = 0; k < 8; ++k) acc[k] = __fadd_rn(acc[k], e[k]);
      }
    }
    __syncthreads();  // the sums of the row before have been read
#pragma unroll
    for (int k = 0; k < 8; ++k) part[warp][lane * 8 + k] = acc[k];
    __syncthreads();
    const int c = blockIdx.y * 256 + threadIdx.x;
    if (c < cols) {
      float s = part[0][threadIdx.x];
#pragma unroll
      for (int w = 1; w < kThreads / 32; ++w) s = __fadd_rn(s, part[w][threadIdx.x]);
      dw[(int64_t)row * cols + c] = (uint16_t)f32_to_bf16_rne_bits(s);
    }
  }
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
  if (batch <= 0 || seq <= 0) return cudaSuccess;  // before the checks: an empty tensor has no address
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

// A warp holds up to 1024 columns (four vectors a thread), a CTA up to 16384 (eight).
#define OAB_NORM_SHAPE(...)                                                      \
  do {                                                                           \
    if (cols <= 1024) { constexpr int LANES = 32, VPT = 4; __VA_ARGS__; }        \
    else if (cols <= 4096) { constexpr int LANES = kThreads, VPT = 2; __VA_ARGS__; } \
    else if (cols <= 8192) { constexpr int LANES = kThreads, VPT = 4; __VA_ARGS__; } \
    else { constexpr int LANES = kThreads, VPT = 8; __VA_ARGS__; }               \
  } while (0)

cudaError_t launch_rms_norm(const void* x, const void* r, const void* w, void* sum, void* out, float* rstd,
                            int64_t rows, int cols, float eps, cudaStream_t st) {
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  if (cols % 8 != 0 || cols > kNormMaxCols || rows >= kMaxGrid || !aligned(x, 16) || !aligned(r, 16) || !aligned(w, 16) ||
      !aligned(sum, 16) || !aligned(out, 16) || (r != nullptr && sum == nullptr))
    return cudaErrorInvalidValue;
  count_launch();
  OAB_NORM_SHAPE(
      const unsigned grid = (unsigned)((rows + kThreads / LANES - 1) / (kThreads / LANES));
      if (r != nullptr)
        rms_norm_kernel<LANES, VPT, true><<<grid, kThreads, 0, st>>>((const uint16_t*)x, (const uint16_t*)r, (const uint16_t*)w, (uint16_t*)sum, (uint16_t*)out, rstd, rows, cols, eps);
      else
        rms_norm_kernel<LANES, VPT, false><<<grid, kThreads, 0, st>>>((const uint16_t*)x, nullptr, (const uint16_t*)w, nullptr, (uint16_t*)out, rstd, rows, cols, eps));
  return cudaGetLastError();
}

// Groups of threads that share the rows: three CTAs per SM when a CTA holds a row, two CTAs
// of eight warps per SM when a warp does.
int rms_norm_partials(int64_t rows, int cols) {
  const int64_t most = cols <= 1024 ? (int64_t)kNumSMs * 16 : (int64_t)kNumSMs * 3;
  return (int)(rows < most ? rows : most);
}

cudaError_t launch_rms_norm_grad(const void* g, const void* gsum, const void* x, const void* w, const float* rstd,
                                 void* dx, void* dw, float* partials, int64_t rows, int cols, cudaStream_t st) {
  if (rows <= 0 || cols <= 0) return cudaSuccess;
  if (cols % 8 != 0 || cols > kNormMaxCols || !aligned(g, 16) || !aligned(gsum, 16) || !aligned(x, 16) || !aligned(w, 16) ||
      !aligned(dx, 16) || !aligned(partials, 16) || (dw != nullptr && partials == nullptr))
    return cudaErrorInvalidValue;
  const int groups = rms_norm_partials(rows, cols);
  float* part = dw != nullptr ? partials : nullptr;
  count_launch();
  OAB_NORM_SHAPE(
      const unsigned grid = (unsigned)((groups + kThreads / LANES - 1) / (kThreads / LANES));
      if (gsum != nullptr)
        rms_norm_grad_kernel<LANES, VPT, true><<<grid, kThreads, 0, st>>>((const uint16_t*)g, (const uint16_t*)gsum, (const uint16_t*)x, (const uint16_t*)w, rstd, (uint16_t*)dx, part, rows, cols, groups);
      else
        rms_norm_grad_kernel<LANES, VPT, false><<<grid, kThreads, 0, st>>>((const uint16_t*)g, nullptr, (const uint16_t*)x, (const uint16_t*)w, rstd, (uint16_t*)dx, part, rows, cols, groups));
  if (dw != nullptr) {
    count_launch();
    column_sum_kernel<<<(unsigned)((cols + 31) / 32), kThreads, 0, st>>>(partials, groups, cols, (uint16_t*)dw);
  }
  return cudaGetLastError();
}

// rows (two ints each) | order | heavy | n_heavy
int64_t embed_work_ints(int64_t n, int64_t vocab) { return 2 * vocab + 2 * n + 1; }

cudaError_t launch_embed_grad(const void* g, const int64_t* ids, int64_t n, void* dw, int64_t vocab, int cols, int* work,
                              cudaStream_t st) {
  if (vocab <= 0 || cols <= 0) return cudaSuccess;
  if (n < 0 || n > kEmbedMaxTokens || vocab >= INT_MAX || cols % 8 != 0 || !aligned(g, 16) || !aligned(dw, 16) || !aligned(work, 8))
    return cudaErrorInvalidValue;
  int2* rows = reinterpret_cast<int2*>(work);
  int *order = work + 2 * vocab, *heavy = order + n, *n_heavy = heavy + n;
  cudaError_t err = cudaMemsetAsync(work, 0, sizeof(int) * (size_t)embed_work_ints(n, vocab), st);
  if (err != cudaSuccess) return err;
  const int per = kScanThreads / kScanPer, col_blocks = (cols + 255) / 256;
  if (n > 0) {
    count_launch();
    embed_order_kernel<<<(unsigned)((n + per - 1) / per), kScanThreads, 0, st>>>(ids, (int)n, (int)vocab, order, rows, heavy, n_heavy);
  }
  // eight CTAs per SM walk the rows; a short table takes fewer
  const int64_t want = (vocab + kThreads / 32 - 1) / (kThreads / 32);
  count_launch();
  embed_rows_kernel<<<(unsigned)(want < kNumSMs * 8 ? want : kNumSMs * 8), kThreads, 0, st>>>((const uint16_t*)g, order, rows,
                                                                                           (uint16_t*)dw, vocab, cols);
  if (n > kLightRows) {
    const int64_t most = n / (kLightRows + 1);  // ids that can have more tokens than that
    count_launch();
    embed_heavy_kernel<<<dim3((unsigned)(most < kNumSMs ? most : kNumSMs), (unsigned)col_blocks), kThreads, 0, st>>>(
        (const uint16_t*)g, order, rows, heavy, n_heavy, (uint16_t*)dw, cols);
  }
  return cudaGetLastError();
}

}  // namespace oab
