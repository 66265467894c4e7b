// Fused Adam/AdamW step kernels for sm_100a.
//
// One kernel template covers the four parameter-precision schemes of the
// reference optimizer (reference: src/offload_adam/kernels/*.py) and folds in
// the work the reference does in separate passes around its step kernel:
//   * the clip coefficient is read from a device scalar and applied in fp32
//     (reference: grad.mul_(clip_coef), src/offload_adam/offload_adam.py:451);
//   * an optional second gradient term is added and rounded to bf16 exactly as
//     an in-place bf16 `add_` would (reference: offload_adam.py:398), so the
//     accumulated host gradient never has to be materialised on the device;
//   * an optional running max of |master| feeds the NVFP4 tensor scale.
//
// The kernel is a grid-stride stream over groups of 16 elements.  Every operand
// moves with Blackwell's 256-bit global loads/stores (one 32-byte request per
// bf16 stream, two for the fp32 master), all issued before the first use, so a
// thread keeps 160-224 bytes in flight and a warp request always covers whole,
// contiguous 1 KiB runs; that is what both HBM3e and a PCIe link (when operands
// are mapped host memory) need to stay busy.
#include <algorithm>
#include <utility>

#include "adam_vec.cuh"

namespace oab {

std::atomic<unsigned long long> g_launch_count{0};

namespace {

using namespace vec;

template <int MODE, bool DECOUPLED, bool HAS_G2, bool PEERS, bool AMAX>
__global__ void __launch_bounds__(kThreads, PEERS ? ((MODE == kModeSR || AMAX) ? 1 : 2) : 3)
adam_step_kernel(Ptrs t, Peers pr, int64_t n, AdamScalars s, const float* __restrict__ clip_ptr,
                 uint64_t seed, int64_t elem_offset, float* amax_out, int vector_ok,
                 const int* abort_flag) {
  __shared__ float red[kThreads / 32];
  if (abort_flag != nullptr && *reinterpret_cast<const volatile int*>(abort_flag) != 0) return;
  const float clip = clip_ptr ? *clip_ptr : 1.0f;
  float amax = 0.f;
  const int64_t tid = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  const int64_t nthreads = (int64_t)gridDim.x * kThreads;
  int64_t scalar_begin = 0;
  if (vector_ok) {
    const int64_t nvec = n / kVec;
    scalar_begin = nvec * kVec;
    for (int64_t vec = tid; vec < nvec; vec += nthreads) {
      VecRegs<MODE> r;
      load_vec<MODE, HAS_G2, PEERS>(r, t, pr, vec);
      const float a = compute_vec<MODE, DECOUPLED, HAS_G2 && !PEERS, AMAX>(r, vec, clip, s, seed, elem_offset);
      if (AMAX) amax = fmaxf(amax, a);
      store_vec<MODE, PEERS>(r, t, pr, vec);
    }
  }
  for (int64_t i = scalar_begin + tid; i < n; i += nthreads)
    amax = fmaxf(amax, scalar_element<MODE, DECOUPLED, PEERS>(t, i, HAS_G2, clip, s, seed, elem_offset, &pr));

  if (AMAX && amax_out != nullptr) {
    float bm = block_max<kThreads>(amax, red);
    if (threadIdx.x == 0 && bm > 0.f) atomicMax(reinterpret_cast<unsigned int*>(amax_out), __float_as_uint(bm));
  }
}

template <int MODE>
cudaError_t dispatch(const AdamStepArgs& a, const Ptrs& t, const Peers& pr, const AdamScalars& s,
                     int grid, int vector_ok, cudaStream_t st) {
#define OAB_LAUNCH2(DEC, G2, PE, AM)                                                           \
  adam_step_kernel<MODE, DEC, G2, PE, AM><<<grid, kThreads, 0, st>>>(                          \
      t, pr, a.n, s, a.clip_coef, a.seed, a.elem_offset, a.amax_out, vector_ok, a.abort_flag)
  // the running max of |master| only exists for fp32_master (it feeds the NVFP4 tensor scale)
#define OAB_LAUNCH(DEC, G2, PE)                                                                \
  do {                                                                                         \
    if (MODE == kModeFP32Master && a.amax_out != nullptr) OAB_LAUNCH2(DEC, G2, PE, (MODE == kModeFP32Master)); \
    else OAB_LAUNCH2(DEC, G2, PE, false);                                                      \
  } while (0)
  const bool peers = a.n_g_peers > 0 || a.n_p_peers > 0;
  if (peers) {
    if (a.decoupled) OAB_LAUNCH(true, false, true); else OAB_LAUNCH(false, false, true);
  } else if (a.decoupled) {
    if (a.g2) OAB_LAUNCH(true, true, false); else OAB_LAUNCH(true, false, false);
  } else {
    if (a.g2) OAB_LAUNCH(false, true, false); else OAB_LAUNCH(false, false, false);
  }
#undef OAB_LAUNCH2
#undef OAB_LAUNCH
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_adam_step(const AdamStepArgs& a, cudaStream_t stream) {
  if (a.n <= 0) return cudaSuccess;
  if (a.mode != kModeFP32Master && a.p == nullptr) return cudaErrorInvalidValue;
  if (a.mode != kModeSR && a.extra == nullptr) return cudaErrorInvalidValue;
  if (a.amax_out != nullptr && a.mode != kModeFP32Master) return cudaErrorInvalidValue;
  if (a.extra_copy != nullptr && a.mode != kModeFP32Master) return cudaErrorInvalidValue;
  Ptrs t{(uint16_t*)a.p, (const uint16_t*)a.g, (const uint16_t*)a.g2,
         (uint16_t*)a.m, (uint16_t*)a.v, a.extra, a.extra_copy};
  if (a.n_g_peers > kMaxPeers || a.n_p_peers > kMaxPeers) return cudaErrorInvalidValue;
  if (a.n_g_peers == 0 && a.g == nullptr) return cudaErrorInvalidValue;
  Peers pr;
  pr.n_g = a.n_g_peers;
  pr.n_p = a.n_p_peers;
  pr.g_scale = a.g_scale;
  for (int j = 0; j < kMaxPeers; ++j) {
    pr.g[j] = (const uint16_t*)a.g_peers[j];
    pr.p[j] = (uint16_t*)a.p_peers[j];
  }
  // with a pulled gradient the local `g` is unused; point it somewhere valid
  if (a.n_g_peers > 0) { t.g = pr.g[0]; t.g2 = nullptr; }
  AdamScalars s;
  s.lr = a.lr;
  s.wd = a.wd;
  s.lr_wd = a.lr * a.wd;  // fp32 product, same as the device's __fmul_rn
  s.one_m_b1h = 1.0f - a.beta1_hat;
  s.one_m_b2h = 1.0f - a.beta2_hat;
  s.eps = a.eps;
  auto al = [](const void* p) { return p == nullptr || (reinterpret_cast<uintptr_t>(p) & 31u) == 0; };
  int vector_ok = al(a.p) && al(t.g) && al(t.g2) && al(a.m) && al(a.v) && al(a.extra) && al(a.extra_copy) &&
                  ((a.elem_offset & 7) == 0);
  for (int j = 0; j < a.n_g_peers; ++j) vector_ok = vector_ok && al(a.g_peers[j]);
  for (int j = 0; j < a.n_p_peers; ++j) vector_ok = vector_ok && al(a.p_peers[j]);
  const int64_t nvec = (a.n + kVec - 1) / kVec;
  int64_t want = (nvec + kThreads - 1) / kThreads;
  int cap = a.max_ctas > 0 ? a.max_ctas : kNumSMs * 8;
  int grid = (int)(want < 1 ? 1 : (want > cap ? cap : want));
  count_launch();
  switch (a.mode) {
    case kModeSR: return dispatch<kModeSR>(a, t, pr, s, grid, vector_ok, stream);
    case kModeFP32Master: return dispatch<kModeFP32Master>(a, t, pr, s, grid, vector_ok, stream);
    case kModeFP31: return dispatch<kModeFP31>(a, t, pr, s, grid, vector_ok, stream);
    case kModeCustom: return dispatch<kModeCustom>(a, t, pr, s, grid, vector_ok, stream);
    default: return cudaErrorInvalidValue;
  }
}

// ----------------------------------------------------------------------------
// Many tensors, one launch: the optimizer whose state lives on the GPU.
//
// A launch per tensor leaves the chip idle twice: small tensors (a norm weight is a
// fraction of one wave) cost a launch each, and every large one ends in a partly filled
// wave.  Here a CTA takes `chunk` consecutive elements of one tensor, whichever tensor
// that is, and all tensors share one tail.  Measured on a B200, a step of 20 tensors of a
// tiny model: 220 -> 117 us (host bound); 62 M parameters in 11 tensors, fp31_master: 238 ->
// 178 us; 1.27 G parameters in 12 tensors, fp32_master: 4008 -> 3769 us (6.7 TB/s).
// ----------------------------------------------------------------------------
namespace {
struct ManyTable {
  int count;
  int64_t chunk;  // elements per CTA, a multiple of kThreads * kVec
  ManyEntry e[kManyTensors];
};

template <int MODE, bool DECOUPLED>
__global__ void __launch_bounds__(kThreads, 3)
adam_step_many_kernel(const __grid_constant__ ManyTable table, AdamScalars s) {
  int lo = 0, hi = table.count - 1;  // the last tensor whose first CTA is not after this one
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (table.e[mid].first_block <= blockIdx.x) lo = mid; else hi = mid - 1;
  }
  const ManyEntry& e = table.e[lo];
  const Ptrs t{(uint16_t*)e.p, (const uint16_t*)e.g, nullptr, (uint16_t*)e.m, (uint16_t*)e.v, e.extra, nullptr};
  const Peers none{};
  const int64_t begin = (int64_t)(blockIdx.x - e.first_block) * table.chunk;
  const int64_t end = begin + table.chunk < e.n ? begin + table.chunk : e.n;
  const uint64_t seed = e.seed;
  int64_t scalar_begin = begin;
  if (e.vector_ok) {
    const int64_t vec_end = end / kVec;
    scalar_begin = vec_end * kVec;
    for (int64_t vec = begin / kVec + threadIdx.x; vec < vec_end; vec += kThreads) {
      VecRegs<MODE> r;
      load_vec<MODE, false, false>(r, t, none, vec);
      compute_vec<MODE, DECOUPLED, false, false>(r, vec, 1.0f, s, seed, 0);
      store_vec<MODE, false>(r, t, none, vec);
    }
  }
  for (int64_t i = scalar_begin + threadIdx.x; i < end; i += kThreads)
    scalar_element<MODE, DECOUPLED>(t, i, false, 1.0f, s, seed, 0);
}

// True when a tensor of the table writes what another one reads or writes: parameters that
// are views of one storage, a state loaded for both.  (At most 480 ranges to sort: 2 us of
// host time for 20 tensors.)
bool share_memory(const ManyTable& t, int mode) {
  using Range = std::pair<uintptr_t, uintptr_t>;
  Range written[4 * kManyTensors];
  int k = 0;
  auto range = [](const void* p, int64_t bytes) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(p);
    return Range(at, at + (uintptr_t)bytes);
  };
  for (int i = 0; i < t.count; ++i) {
    const ManyEntry& e = t.e[i];
    if (e.p != nullptr) written[k++] = range(e.p, 2 * e.n);
    written[k++] = range(e.m, 2 * e.n);
    written[k++] = range(e.v, 2 * e.n);
    if (e.extra != nullptr) written[k++] = range(e.extra, (mode == kModeFP32Master ? 4 : 2) * e.n);
  }
  std::sort(written, written + k);
  for (int i = 1; i < k; ++i)
    if (written[i].first < written[i - 1].second) return true;
  for (int i = 0; i < t.count; ++i) {
    const Range g = range(t.e[i].g, 2 * t.e[i].n);
    const Range* next = std::upper_bound(written, written + k, g);  // the first that begins after g begins
    if ((next != written + k && next->first < g.second) || (next != written && (next - 1)->second > g.first)) return true;
  }
  return false;
}

template <int MODE>
void launch_many(const ManyTable& t, unsigned grid, bool decoupled, const AdamScalars& s, cudaStream_t st) {
  if (decoupled) adam_step_many_kernel<MODE, true><<<grid, kThreads, 0, st>>>(t, s);
  else adam_step_many_kernel<MODE, false><<<grid, kThreads, 0, st>>>(t, s);
}
}  // namespace

cudaError_t launch_adam_step_many(ManyEntry* entries, int count, int mode, bool decoupled, float lr, float wd,
                                  float beta1_hat, float beta2_hat, float eps, cudaStream_t stream) {
  AdamScalars s;
  s.lr = lr; s.wd = wd; s.lr_wd = lr * wd;
  s.one_m_b1h = 1.0f - beta1_hat; s.one_m_b2h = 1.0f - beta2_hat; s.eps = eps;
  auto al = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; };
  for (int at = 0; at < count; at += kManyTensors) {
    ManyTable t;
    t.count = 0;
    int64_t total = 0;
    for (int i = at; i < count && i < at + kManyTensors; ++i) {
      const ManyEntry& e = entries[i];
      if (e.g == nullptr || e.m == nullptr || e.v == nullptr) return cudaErrorInvalidValue;
      if (mode != kModeFP32Master && e.p == nullptr) return cudaErrorInvalidValue;
      if (mode != kModeSR && e.extra == nullptr) return cudaErrorInvalidValue;
      if (e.n <= 0) continue;
      total += e.n;
      ManyEntry& o = t.e[t.count++];
      o = e;
      o.vector_ok = al(e.p) && al(e.g) && al(e.m) && al(e.v) && al(e.extra);
    }
    if (t.count == 0) continue;
    if (t.count > 1 && share_memory(t, mode)) {  // one after the other, as adam_step would
      for (int i = 0; i < t.count; ++i) {
        const cudaError_t err = launch_adam_step_many(&t.e[i], 1, mode, decoupled, lr, wd, beta1_hat, beta2_hat, eps, stream);
        if (err != cudaSuccess) return err;
      }
      continue;
    }
    // one vector per thread while that does not fill the chip several times over, four
    // after that (a CTA's fixed cost is then a small part of its 10 us)
    const int64_t unit = kThreads * kVec;
    t.chunk = total >= unit * 4 * kNumSMs * 12 ? unit * 4 : unit;
    int64_t blocks = 0;
    for (int i = 0; i < t.count; ++i) {
      t.e[i].first_block = (uint32_t)blocks;
      blocks += (t.e[i].n + t.chunk - 1) / t.chunk;
    }
    if (blocks >= (int64_t(1) << 31)) return cudaErrorInvalidValue;
    count_launch();
    switch (mode) {
      case kModeSR: launch_many<kModeSR>(t, (unsigned)blocks, decoupled, s, stream); break;
      case kModeFP32Master: launch_many<kModeFP32Master>(t, (unsigned)blocks, decoupled, s, stream); break;
      case kModeFP31: launch_many<kModeFP31>(t, (unsigned)blocks, decoupled, s, stream); break;
      case kModeCustom: launch_many<kModeCustom>(t, (unsigned)blocks, decoupled, s, stream); break;
      default: return cudaErrorInvalidValue;
    }
    const cudaError_t err = cudaGetLastError();
    if (err != cudaSuccess) return err;
  }
  return cudaSuccess;
}

// ----------------------------------------------------------------------------
// Multi-tensor variant: one launch updates every small (GPU-resident) tensor.
// block_map[b] = {tensor index, chunk index}; each block handles kChunk elements.
// (reference: the per-parameter loop of OffloadAdam._step_inplace,
//  src/offload_adam/offload_adam.py:456-467, one kernel + one zero_ per tensor)
// ----------------------------------------------------------------------------
namespace {
constexpr int kChunk = 8192;

template <int MODE, bool DECOUPLED>
__global__ void __launch_bounds__(kThreads)
multi_tensor_adam_kernel(const MultiTensorEntry* __restrict__ table,
                         const int2* __restrict__ block_map, AdamScalars s,
                         const float* __restrict__ clip_ptr, uint64_t seed, int zero_grad) {
  const int2 bm = block_map[blockIdx.x];
  const MultiTensorEntry e = table[bm.x];
  const float clip = clip_ptr ? *clip_ptr : 1.0f;
  Ptrs t{(uint16_t*)e.p, (const uint16_t*)e.g, nullptr, (uint16_t*)e.m, (uint16_t*)e.v, e.extra, nullptr};
  const int64_t begin = (int64_t)bm.y * kChunk;
  int64_t end = begin + kChunk;
  if (end > e.n) end = e.n;
  for (int64_t i = begin + threadIdx.x; i < end; i += kThreads) {
    scalar_element<MODE, DECOUPLED>(t, i, false, clip, s, seed, e.elem_offset);
    if (zero_grad) const_cast<uint16_t*>(t.g)[i] = 0;
  }
}
}  // namespace

cudaError_t launch_multi_tensor_adam(const MultiTensorEntry* dev_table, int n_tensors,
                                     const int2* dev_block_map, int n_blocks, int mode,
                                     bool decoupled, float lr, float wd, float beta1_hat,
                                     float beta2_hat, float eps, const float* clip_coef,
                                     uint64_t seed, bool zero_grad, cudaStream_t stream) {
  if (n_blocks <= 0 || n_tensors <= 0) return cudaSuccess;
  AdamScalars s;
  s.lr = lr; s.wd = wd; s.lr_wd = lr * wd;
  s.one_m_b1h = 1.0f - beta1_hat; s.one_m_b2h = 1.0f - beta2_hat; s.eps = eps;
  count_launch();
#define OAB_MT(M)                                                                              \
  if (decoupled)                                                                               \
    multi_tensor_adam_kernel<M, true><<<n_blocks, kThreads, 0, stream>>>(                      \
        dev_table, dev_block_map, s, clip_coef, seed, zero_grad ? 1 : 0);                      \
  else                                                                                         \
    multi_tensor_adam_kernel<M, false><<<n_blocks, kThreads, 0, stream>>>(                     \
        dev_table, dev_block_map, s, clip_coef, seed, zero_grad ? 1 : 0)
  switch (mode) {
    case kModeSR: OAB_MT(kModeSR); break;
    case kModeFP32Master: OAB_MT(kModeFP32Master); break;
    case kModeFP31: OAB_MT(kModeFP31); break;
    case kModeCustom: OAB_MT(kModeCustom); break;
    default: return cudaErrorInvalidValue;
  }
#undef OAB_MT
  return cudaGetLastError();
}

int multi_tensor_chunk() { return kChunk; }

}  // namespace oab
