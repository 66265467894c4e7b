// Python bindings of the cross-entropy kernels.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <optional>

#include "loss_ops.h"

namespace py = pybind11;
using at::Tensor;

namespace {

cudaStream_t cur() { return at::cuda::getCurrentCUDAStream().stream(); }
void ok(cudaError_t e, const char* what) { TORCH_CHECK(e == cudaSuccess, what, ": ", cudaGetErrorString(e)); }

void check_logits(const Tensor& x, const Tensor& labels, const char* what) {
  TORCH_CHECK(x.is_cuda() && x.scalar_type() == at::kBFloat16 && x.dim() == 2 && x.stride(1) == 1, what,
              ": logits must be a 2-D bf16 CUDA tensor with unit column stride");
  TORCH_CHECK(x.size(0) <= 1 || x.stride(0) % oab::kCePitchAlign == 0, what, ": rows must start 32-byte aligned");
  TORCH_CHECK(labels.is_cuda() && labels.scalar_type() == at::kLong && labels.is_contiguous() &&
                  labels.numel() == x.size(0), what, ": one contiguous int64 label per row");
}
// the last row, too, is read and written in whole 16-value vectors
int64_t pitch_of(const Tensor& x) {
  const int64_t pitch = x.size(0) > 1 ? x.stride(0) : (x.size(1) + oab::kCePitchAlign - 1) / oab::kCePitchAlign * oab::kCePitchAlign;
  const int64_t end = x.storage_offset() + (x.size(0) - 1) * pitch + (x.size(1) + 15) / 16 * 16;
  TORCH_CHECK(end * x.element_size() <= (int64_t)x.storage().nbytes(), "logits buffer ends inside its last vector");
  return pitch;
}
void check_f32(const Tensor& t, int64_t n, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous() && t.numel() >= n, name, ": CUDA fp32");
}

// Where the kernel leaves a label that the vocabulary does not have.  The host sees it when
// that kernel has run: the call itself returns NaN, and the next one (its backward, or the
// next loss) raises.  PyTorch's operations end the context with a device assertion instead,
// which the next call that looks reports as late.
int64_t* bad_label() {
  static int64_t* const at = [] {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // the first call may be captured
    ok(cudaThreadExchangeStreamCaptureMode(&mode), "label report");
    void* p = nullptr;
    const cudaError_t e = cudaHostAlloc(&p, sizeof(int64_t), cudaHostAllocPortable | cudaHostAllocMapped);
    ok(cudaThreadExchangeStreamCaptureMode(&mode), "label report");
    ok(e, "label report");
    *static_cast<int64_t*>(p) = -1;
    return static_cast<int64_t*>(p);
  }();
  return at;
}
void raise_bad_label() {
  if (__atomic_load_n(bad_label(), __ATOMIC_RELAXED) < 0) return;
  const int64_t label = __atomic_exchange_n(bad_label(), int64_t(-1), __ATOMIC_RELAXED);
  TORCH_CHECK_INDEX(label < 0, "label ", std::to_string(label), " of an earlier cross-entropy is outside its vocabulary; that loss is NaN");
}

// An (n, V) bf16 view whose rows start 32-byte aligned.
Tensor ce_logits_buffer(const Tensor& like, int64_t n, int64_t V) {
  c10::cuda::CUDAGuard guard(like.device());
  const int64_t pitch = (V + oab::kCePitchAlign - 1) / oab::kCePitchAlign * oab::kCePitchAlign;
  return at::empty({n, pitch}, like.options().dtype(at::kBFloat16)).narrow(1, 0, V);
}

// stats: 3 n floats (max, 1 / sum, row loss); see loss_ops.h
void ce_stats(const Tensor& logits, const Tensor& labels, const Tensor& stats) {
  if (logits.size(0) == 0) return;
  check_logits(logits, labels, "ce_stats");
  check_f32(stats, 3 * logits.size(0), "stats");
  c10::cuda::CUDAGuard guard(logits.device());
  raise_bad_label();
  ok(oab::launch_ce_stats(logits.data_ptr(), pitch_of(logits), labels.data_ptr<int64_t>(), logits.size(0),
                          logits.size(1), stats.data_ptr<float>(), bad_label(), cur()), "ce_stats");
}

void ce_finish(const std::optional<Tensor>& row_loss, const Tensor& labels, const std::optional<Tensor>& loss, const Tensor& inv) {
  TORCH_CHECK(labels.is_cuda() && labels.scalar_type() == at::kLong && labels.is_contiguous(), "ce_finish: contiguous int64 labels");
  check_f32(inv, 1, "inv");
  const bool has = row_loss.has_value() && row_loss->defined();
  if (has) {
    check_f32(*row_loss, labels.numel(), "row_loss");
    TORCH_CHECK(loss.has_value(), "ce_finish: row_loss without loss");
    check_f32(*loss, 1, "loss");
  }
  c10::cuda::CUDAGuard guard(labels.device());
  ok(oab::launch_ce_finish(has ? row_loss->data_ptr<float>() : nullptr, labels.data_ptr<int64_t>(), labels.numel(),
                           has ? loss->data_ptr<float>() : nullptr, inv.data_ptr<float>(), cur()), "ce_finish");
}

void ce_grad(const Tensor& logits, const Tensor& labels, const Tensor& stats, const Tensor& inv,
             const std::optional<Tensor>& g, const Tensor& grad) {
  const int64_t n = logits.size(0);
  if (n == 0) return;
  check_logits(logits, labels, "ce_grad");
  check_logits(grad, labels, "ce_grad");
  check_f32(stats, 2 * n, "stats");
  check_f32(inv, 1, "inv");
  TORCH_CHECK(grad.sizes() == logits.sizes() && pitch_of(grad) == pitch_of(logits), "ce_grad: grad like logits");
  const float* gp = nullptr;
  if (g.has_value() && g->defined()) {
    check_f32(*g, 1, "g");
    gp = g->data_ptr<float>();
  }
  c10::cuda::CUDAGuard guard(logits.device());
  raise_bad_label();
  const float* s = stats.data_ptr<float>();
  ok(oab::launch_ce_grad(logits.data_ptr(), pitch_of(logits), labels.data_ptr<int64_t>(), n, logits.size(1), s, s + n,
                         inv.data_ptr<float>(), gp, grad.data_ptr(), cur()), "ce_grad");
}

// fp32(acc) + fp32(g), in fp32 (into `acc` when it is fp32) or rounded to bf16 (into `to` when
// it is given; it may be g); g is bf16
Tensor sum_bf16(const Tensor& acc, const Tensor& g, bool round, const std::optional<Tensor>& to) {
  TORCH_CHECK(acc.is_cuda() && g.device() == acc.device() && acc.is_contiguous() && g.is_contiguous() && acc.sizes() == g.sizes() &&
                  g.scalar_type() == at::kBFloat16 && (acc.scalar_type() == at::kBFloat16 || acc.scalar_type() == at::kFloat),
              "sum_bf16: contiguous CUDA tensors of one shape");
  c10::cuda::CUDAGuard guard(acc.device());
  const bool f32 = acc.scalar_type() == at::kFloat;
  const bool given = round && to.has_value() && to->defined();
  TORCH_CHECK(!given || (to->sizes() == g.sizes() && to->scalar_type() == at::kBFloat16 && to->is_contiguous() && to->device() == g.device()),
              "sum_bf16: `to` like g");
  Tensor out = given ? *to : round ? at::empty_like(g) : (f32 ? acc : at::empty(g.sizes(), g.options().dtype(at::kFloat)));
  ok(oab::launch_sum_bf16(acc.data_ptr(), f32, g.data_ptr(), round ? nullptr : out.data_ptr<float>(),
                          round ? out.data_ptr() : nullptr, g.numel(), cur()), "sum_bf16");
  return out;
}

}  // namespace

void bind_loss(py::module_& m) {
  m.def("ce_logits_buffer", &ce_logits_buffer);
  m.def("ce_stats", &ce_stats);
  m.def("ce_finish", &ce_finish, py::arg("row_loss"), py::arg("labels"), py::arg("loss"), py::arg("inv"));
  m.def("sum_bf16", &sum_bf16, py::arg("acc"), py::arg("g"), py::arg("round"), py::arg("to") = py::none());
  m.def("ce_grad", &ce_grad, py::arg("logits"), py::arg("labels"), py::arg("stats"), py::arg("inv"), py::arg("g"),
        py::arg("grad"));
}
