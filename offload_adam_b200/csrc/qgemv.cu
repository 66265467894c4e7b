// y = x W^T (+ bias) for a few tokens and a packed weight, without a dense copy of it.
//
// A linear layer on one to four tokens reads every weight once and does two to eight
// operations with it: the packed bytes are what it cannot do without.  De-quantizing to a
// dense bf16 copy first writes and re-reads four (4-bit formats) or two (int8) times those
// bytes.  Here the weights are decoded to fp32 in registers, multiplied with the bf16
// activations and summed in fp32; the scale of a block is applied to the block's partial
// sum, so no weight is rounded to bf16 on the way.
//
// Row-major formats (NVFP4, NF4, int8): a lane owns 16 consecutive columns of R rows per
// step, a warp 512 columns; the next step's words are loaded before the current ones are
// used.  The R rows share the unpacked activations.  One token through 14336 x 4096 NF4: 19 us
// of GPU time (1.7 TB/s of packed bytes), with a dense copy 43 us.  What bounds it is not the
// bytes but the decoding: the look-ups of 58.7 M indices keep the shared-memory pipe busy for
// 6.5 us and the issue slots 63 % of the time.
#include "qgemv.h"
#include "quant.h"
#include "quant_math.cuh"

namespace oab {
namespace {

using namespace qm;

constexpr int kSplitWarps = 4;  // warps of a CTA that split a row

__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  return ((uint64_t)__float_as_uint(hi) << 32) | __float_as_uint(lo);
}
__device__ __forceinline__ uint64_t unpack_pair(uint32_t w) {  // two bf16
  return pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
// two independent fp32 fused multiply-adds
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float sum2(uint64_t v) {
  return __fadd_rn(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32)));
}

struct Args {
  const uint8_t* w;
  const void* scales;
  const float* global_scale;
  const uint16_t* x;
  const uint16_t* bias;
  uint16_t* y;
  int64_t rows;
  int cols, tokens, block_shift;  // NF4: log2 of the block size
};

// 16 packed weights of a row and the scale they share
template <int FMT>
struct Raw {
  uint32_t w[FMT == kQInt8 ? 4 : 2];
  float scale;
};

template <int FMT>
__device__ __forceinline__ void load_raw(Raw<FMT>& r, const Args& a, int64_t row, int col) {
  const int64_t at = row * a.cols + col;
  if (FMT == kQInt8) {
    const uint4 v = __ldcs(reinterpret_cast<const uint4*>(a.w + at));
    r.w[0] = v.x; r.w[1] = v.y;
    r.w[FMT == kQInt8 ? 2 : 0] = v.z; r.w[FMT == kQInt8 ? 3 : 1] = v.w;
  } else {
    const uint2 v = __ldcs(reinterpret_cast<const uint2*>(a.w + (at >> 1)));
    r.w[0] = v.x; r.w[1] = v.y;
    if (FMT == kQNVFP4) r.scale = __uint_as_float(reinterpret_cast<const uint8_t*>(a.scales)[at >> 4]);  // decoded later
    else r.scale = __ldg(reinterpret_cast<const float*>(a.scales) + (at >> a.block_shift));
  }
}

// the 16 weights without their scale, as 8 pairs (even column in the low half)
template <int FMT>
__device__ __forceinline__ void decode(const Raw<FMT>& r, const float* lut, uint64_t (&v)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    if (FMT == kQInt8) {
      const uint32_t w = r.w[i >> 1] ^ 0x80808080u;
      const uint32_t sel = 0x7650u | (2 * (i & 1));
      // bytes {value, 0, 0, 0x4B}: the float 2^23 + 128 + q
      v[i] = pack2(__fsub_rn(__uint_as_float(__byte_perm(w, 0x4B000000u, sel)), 8388736.0f),
                   __fsub_rn(__uint_as_float(__byte_perm(w, 0x4B000000u, sel + 1)), 8388736.0f));
    } else {
      const uint32_t w = r.w[i >> 2];
      const int b = 8 * (i & 3);
      if (FMT == kQNVFP4) {
        const float2 f = e2m1x2_to_f32((w >> b) & 0xffu);
        v[i] = pack2(f.x, f.y);
      } else {  // even column in the high nibble; 16 table words in 16 banks: no conflicts
        const uint32_t hi = (w >> (b + 2)) & 0x3cu;
        const uint32_t lo = (b ? (w >> (b - 2)) : (w << 2)) & 0x3cu;
        const char* t = reinterpret_cast<const char*>(lut);
        v[i] = pack2(*reinterpret_cast<const float*>(t + hi), *reinterpret_cast<const float*>(t + lo));
      }
    }
  }
}

template <int FMT>
__device__ __forceinline__ float scale_of(const Raw<FMT>& r) {
  if (FMT == kQNVFP4) return e4m3_to_f32((uint8_t)__float_as_uint(r.scale));
  return FMT == kQInt8 ? 1.0f : r.scale;
}

// SPLIT: the four warps of a CTA share its R rows and split the columns.  Otherwise a CTA is
// one warp with R rows of its own: the rows of a layer rarely fill whole waves of larger
// CTAs (14336 rows in CTAs of 16 are 896 of them where 888 fit at a time).
template <int FMT, int R, int M, bool SPLIT>
__global__ void __launch_bounds__(SPLIT ? 32 * kSplitWarps : 32, (M == 4 ? 3 : (M == 2 ? 5 : 6)) * (SPLIT ? 1 : 4)) qgemv_kernel(Args a) {
  constexpr int kWarps = SPLIT ? kSplitWarps : 1, kThreads = 32 * kWarps;
  __shared__ float lut[16];
  __shared__ float part[kWarps][R * M];
  if (FMT == kQNF4) {
    if (threadIdx.x < 16) lut[threadIdx.x] = kNF4[threadIdx.x];
    if (SPLIT) __syncthreads(); else __syncwarp();
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row0 = (int64_t)blockIdx.x * R;
  const int first = SPLIT ? threadIdx.x * 16 : lane * 16;
  const int step = SPLIT ? kThreads * 16 : 512;
  float acc[R][M];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int t = 0; t < M; ++t) acc[r][t] = 0.f;
  // rows past the end repeat the last one and are not stored
  int64_t row[R];
#pragma unroll
  for (int r = 0; r < R; ++r) row[r] = row0 + r < a.rows ? row0 + r : a.rows - 1;

  Raw<FMT> cur[R], nxt[R];
  if (first < a.cols) {
#pragma unroll
    for (int r = 0; r < R; ++r) load_raw<FMT>(nxt[r], a, row[r], first);
  }
  for (int c = first; c < a.cols; c += step) {
#pragma unroll
    for (int r = 0; r < R; ++r) cur[r] = nxt[r];
    if (c + step < a.cols) {
#pragma unroll
      for (int r = 0; r < R; ++r) load_raw<FMT>(nxt[r], a, row[r], c + step);
    }
    if (M <= 2) {  // hold the activations, decode row by row
      uint64_t xp[M][8];
#pragma unroll
      for (int t = 0; t < M; ++t) {
        const V8 xv = ld32(a.x + (int64_t)t * a.cols + c);  // M == tokens here
#pragma unroll
        for (int i = 0; i < 8; ++i) xp[t][i] = unpack_pair(xv.w[i]);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        uint64_t w[8];
        decode<FMT>(cur[r], lut, w);
        const float s = scale_of<FMT>(cur[r]);
#pragma unroll
        for (int t = 0; t < M; ++t) {
          uint64_t p = 0;
#pragma unroll
          for (int i = 0; i < 8; ++i) p = fma2(w[i], xp[t][i], p);
          acc[r][t] = __fmaf_rn(sum2(p), s, acc[r][t]);
        }
      }
    } else {  // hold the decoded weights, unpack token by token
      uint64_t w[R][8];
      float s[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        decode<FMT>(cur[r], lut, w[r]);
        s[r] = scale_of<FMT>(cur[r]);
      }
#pragma unroll
      for (int t = 0; t < M; ++t) {
        // a missing fourth token repeats the last one: no branch between the loads
        const V8 xv = ld32(a.x + (int64_t)(t < a.tokens ? t : a.tokens - 1) * a.cols + c);
        uint64_t p[R];
#pragma unroll
        for (int r = 0; r < R; ++r) p[r] = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const uint64_t xp = unpack_pair(xv.w[i]);
#pragma unroll
          for (int r = 0; r < R; ++r) p[r] = fma2(w[r][i], xp, p[r]);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r][t] = __fmaf_rn(sum2(p[r]), s[r], acc[r][t]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int t = 0; t < M; ++t)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc[r][t] = __fadd_rn(acc[r][t], __shfl_xor_sync(0xffffffffu, acc[r][t], o));
  if (SPLIT) {
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < R * M; ++i) part[warp][i] = acc[i / M][i % M];
    }
    __syncthreads();
  }
  // thread (lane) i writes result i of the warp's (or, split, of the CTA's) R * M
#pragma unroll
  for (int i = 0; i < R * M; ++i) {
    if ((SPLIT ? (int)threadIdx.x : lane) != i) continue;
    const int r = i / M, t = i % M;
    if (row0 + r >= a.rows || t >= a.tokens) continue;
    float v = acc[r][t];
    if (SPLIT) {
      v = part[0][i];
#pragma unroll
      for (int k = 1; k < kWarps; ++k) v = __fadd_rn(v, part[k][i]);
    }
    if (FMT == kQNVFP4) v = __fmul_rn(v, *a.global_scale);
    if (FMT == kQInt8) v = __fmul_rn(v, bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(a.scales)[row0 + r]));
    if (a.bias != nullptr) v = __fadd_rn(v, bf16_bits_to_f32(a.bias[row0 + r]));
    a.y[(int64_t)t * a.rows + row0 + r] = (uint16_t)f32_to_bf16_rne_bits(v);
  }
}

// int4 (GPTQ layout): the words of one input position lie along the output rows, so a lane
// owns a row, a warp reads 128 consecutive bytes per word, and the warps of a CTA split the
// columns in units of 128 (16 words a lane, the next unit's loaded before the current one is
// used).  The activations of a word are the same for all lanes: one broadcast load.
template <int WORDS /* per quantization group */, int M, int WARPS>
__global__ void __launch_bounds__(32 * WARPS) qgemv_int4_kernel(Args a) {
  __shared__ float part[WARPS][M][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row0 = (int64_t)blockIdx.x * 32;
  const int64_t row = row0 + lane < a.rows ? row0 + lane : a.rows - 1;
  const uint32_t* w = reinterpret_cast<const uint32_t*>(a.w) + row;
  const uint16_t* sc = reinterpret_cast<const uint16_t*>(a.scales) + row;
  const int units = a.cols >> 7;
  constexpr int kGroups = 16 / WORDS;
  float acc[M];
#pragma unroll
  for (int t = 0; t < M; ++t) acc[t] = 0.f;
  uint32_t nxt[16];
  uint16_t nxs[kGroups];
  auto load = [&](int u) {
#pragma unroll
    for (int k = 0; k < 16; ++k) nxt[k] = __ldcs(w + ((int64_t)u * 16 + k) * a.rows);
#pragma unroll
    for (int g = 0; g < kGroups; ++g) nxs[g] = __ldg(sc + ((int64_t)u * kGroups + g) * a.rows);
  };
  if (warp < units) load(warp);
  for (int u = warp; u < units; u += WARPS) {
    uint32_t cur[16];
    float s[kGroups];
#pragma unroll
    for (int k = 0; k < 16; ++k) cur[k] = nxt[k];
#pragma unroll
    for (int g = 0; g < kGroups; ++g) s[g] = bf16_bits_to_f32(nxs[g]);
    if (u + WARPS < units) load(u + WARPS);
    const uint16_t* x = a.x + u * 128;
#pragma unroll
    for (int g = 0; g < kGroups; ++g) {
      uint64_t p[M];
#pragma unroll
      for (int t = 0; t < M; ++t) p[t] = 0;
#pragma unroll
      for (int k = 0; k < WORDS; ++k) {
        const uint32_t v = cur[g * WORDS + k];
        uint64_t q[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          q[i] = pack2(small_int_to_f32((v >> (8 * i)) & 0xfu, 8388616.0f), small_int_to_f32((v >> (8 * i + 4)) & 0xfu, 8388616.0f));
#pragma unroll
        for (int t = 0; t < M; ++t) {
          const uint4 xv = __ldg(reinterpret_cast<const uint4*>(x + (int64_t)t * a.cols + (g * WORDS + k) * 8));
          p[t] = fma2(q[0], unpack_pair(xv.x), p[t]);
          p[t] = fma2(q[1], unpack_pair(xv.y), p[t]);
          p[t] = fma2(q[2], unpack_pair(xv.z), p[t]);
          p[t] = fma2(q[3], unpack_pair(xv.w), p[t]);
        }
      }
#pragma unroll
      for (int t = 0; t < M; ++t) acc[t] = __fmaf_rn(sum2(p[t]), s[g], acc[t]);
    }
  }
#pragma unroll
  for (int t = 0; t < M; ++t) part[warp][t][lane] = acc[t];
  __syncthreads();
  for (int i = threadIdx.x; i < 32 * M; i += 32 * WARPS) {
    const int t = i >> 5, l = i & 31;
    if (t >= a.tokens || row0 + l >= a.rows) continue;
    float v = part[0][t][l];
#pragma unroll
    for (int k = 1; k < WARPS; ++k) v = __fadd_rn(v, part[k][t][l]);
    if (a.bias != nullptr) v = __fadd_rn(v, bf16_bits_to_f32(a.bias[row0 + l]));
    a.y[(int64_t)t * a.rows + row0 + l] = (uint16_t)f32_to_bf16_rne_bits(v);
  }
}

template <int WORDS, int M>
cudaError_t launch_int4(const Args& a, cudaStream_t st) {
  // fewer rows than a CTA of 32 per SM: more warps split the columns
  const unsigned grid = (unsigned)((a.rows + 31) / 32);
  if (a.rows >= int64_t(kNumSMs) * 32) qgemv_int4_kernel<WORDS, M, 8><<<grid, 256, 0, st>>>(a);
  else qgemv_int4_kernel<WORDS, M, 16><<<grid, 512, 0, st>>>(a);
  return cudaGetLastError();
}
template <int M>
cudaError_t launch_int4_group(const Args& a, int group, cudaStream_t st) {
  if (group == 32) return launch_int4<4, M>(a, st);
  if (group == 64) return launch_int4<8, M>(a, st);
  return launch_int4<16, M>(a, st);
}

template <int FMT, int M>
cudaError_t launch_rows(const Args& a, cudaStream_t st) {
  // Four rows per warp share the activations as long as that still gives every SM eight
  // warps; fewer rows: the warps of a CTA split the columns, so that a row's reads are in
  // flight together; very few rows: one row per CTA.
  auto ctas = [&](int64_t per) { return (unsigned)((a.rows + per - 1) / per); };
  if (a.rows >= int64_t(kNumSMs) * 32) qgemv_kernel<FMT, 4, M, false><<<ctas(4), 32, 0, st>>>(a);
  else if (a.rows >= int64_t(kNumSMs) * 4) qgemv_kernel<FMT, 4, M, true><<<ctas(4), 32 * kSplitWarps, 0, st>>>(a);
  else qgemv_kernel<FMT, 1, M, true><<<ctas(1), 32 * kSplitWarps, 0, st>>>(a);
  return cudaGetLastError();
}

template <int FMT>
cudaError_t launch_tokens(const Args& a, cudaStream_t st) {
  if (a.tokens == 1) return launch_rows<FMT, 1>(a, st);
  if (a.tokens == 2) return launch_rows<FMT, 2>(a, st);
  return launch_rows<FMT, 4>(a, st);
}

}  // namespace

bool qgemv_supported(int format, int64_t rows, int64_t cols, int64_t tokens, int group) {
  if (rows <= 0 || rows >= (int64_t(1) << 31) || cols <= 0 || cols % 16 != 0 || cols >= (int64_t(1) << 30)) return false;
  if (tokens < 1 || tokens > kQGemvMaxTokens) return false;
  if (format == kQInt4) return tokens <= 2 && rows >= 1024 && cols % 128 == 0 && (group == 32 || group == 64 || group == 128);
  if (format == kQNF4) return group >= 16 && group <= 512 && (group & (group - 1)) == 0 && cols % group == 0;
  return format == kQNVFP4 || format == kQInt8;
}

cudaError_t launch_qgemv(int format, const void* packed, const void* scales, const float* global_scale, int group,
                         const void* x, int64_t tokens, const void* bias, void* y, int64_t rows, int64_t cols,
                         cudaStream_t st) {
  if (!qgemv_supported(format, rows, cols, tokens, group)) return cudaErrorInvalidValue;
  if ((reinterpret_cast<uintptr_t>(x) & 31u) || (reinterpret_cast<uintptr_t>(packed) & (qgemv_packed_align(format) - 1)))
    return cudaErrorInvalidValue;
  Args a{(const uint8_t*)packed, scales, global_scale, (const uint16_t*)x, (const uint16_t*)bias, (uint16_t*)y,
         rows, (int)cols, (int)tokens, 0};
  while (format == kQNF4 && (1 << a.block_shift) < group) ++a.block_shift;
  count_launch();
  switch (format) {
    case kQInt4:
      return a.tokens == 1 ? launch_int4_group<1>(a, group, st) : launch_int4_group<2>(a, group, st);
    case kQNVFP4: return launch_tokens<kQNVFP4>(a, st);
    case kQNF4: return launch_tokens<kQNF4>(a, st);
    default: return launch_tokens<kQInt8>(a, st);
  }
}

}  // namespace oab
