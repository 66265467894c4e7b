// Python bindings of the quantization kernels.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <optional>

#include "qgemv.h"
#include "quant.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

int qdtype(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return oab::kF32;
    case at::kBFloat16: return oab::kBF16;
    case at::kHalf: return oab::kF16;
    default: TORCH_CHECK(false, "unsupported dtype ", t.scalar_type());
  }
  return -1;
}
cudaStream_t cur() { return at::cuda::getCurrentCUDAStream().stream(); }
void ok(cudaError_t e, const char* what) { TORCH_CHECK(e == cudaSuccess, what, ": ", cudaGetErrorString(e)); }
void dense(const Tensor& t, const char* n) { TORCH_CHECK(t.is_cuda() && t.is_contiguous(), n, " must be a contiguous CUDA tensor"); }

// max |x| of disjoint parts of x; the largest is the tensor's
Tensor absmax_partials(const Tensor& x) {
  dense(x, "x");
  Tensor out = at::empty({oab::absmax_partials(x.numel())}, x.options().dtype(at::kFloat));
  ok(oab::launch_absmax_partials(x.data_ptr(), qdtype(x), x.numel(), out.data_ptr<float>(), cur()), "absmax_partials");
  return out;
}

void nvfp4_quantize(const Tensor& x, const std::optional<Tensor>& amax_in, Tensor packed, Tensor scales, Tensor global_scale) {
  dense(x, "x"); dense(packed, "packed"); dense(scales, "scales");
  const Tensor amax = amax_in.has_value() && amax_in->defined() ? *amax_in : absmax_partials(x);
  TORCH_CHECK(x.numel() % 16 == 0 && packed.numel() * 2 == x.numel() && scales.numel() * 16 == x.numel(), "nvfp4 shapes");
  TORCH_CHECK(packed.element_size() == 1 && scales.element_size() == 1, "nvfp4 payload dtypes");
  TORCH_CHECK(amax.is_contiguous() && amax.numel() >= 1, "amax: one or more contiguous values");
  TORCH_CHECK(amax.is_cuda() && amax.scalar_type() == at::kFloat && global_scale.is_cuda() && global_scale.scalar_type() == at::kFloat, "scalars: CUDA fp32");
  ok(oab::launch_nvfp4_quantize(x.data_ptr(), qdtype(x), x.numel(), amax.data_ptr<float>(), (int)amax.numel(),
                                (uint8_t*)packed.data_ptr(), (uint8_t*)scales.data_ptr(),
                                global_scale.data_ptr<float>(), cur()), "nvfp4_quantize");
}

void nvfp4_dequantize(const Tensor& packed, const Tensor& scales, const Tensor& global_scale, Tensor out) {
  dense(packed, "packed"); dense(scales, "scales"); dense(out, "out");
  TORCH_CHECK(out.numel() == packed.numel() * 2 && scales.numel() * 16 == out.numel(), "nvfp4 shapes");
  ok(oab::launch_nvfp4_dequantize((const uint8_t*)packed.data_ptr(), (const uint8_t*)scales.data_ptr(),
                                  global_scale.data_ptr<float>(), out.numel(), out.data_ptr(), qdtype(out), cur()), "nvfp4_dequantize");
}

void nf4_quantize(const Tensor& x, int64_t blocksize, Tensor packed, Tensor absmax_out) {
  dense(x, "x"); dense(packed, "packed"); dense(absmax_out, "absmax");
  TORCH_CHECK(x.numel() % blocksize == 0 && packed.numel() * 2 == x.numel() && absmax_out.numel() * blocksize == x.numel(), "nf4 shapes");
  TORCH_CHECK(absmax_out.scalar_type() == at::kFloat, "absmax: fp32");
  ok(oab::launch_nf4_quantize(x.data_ptr(), qdtype(x), x.numel(), (int)blocksize, (uint8_t*)packed.data_ptr(),
                              absmax_out.data_ptr<float>(), cur()), "nf4_quantize");
}

void nf4_dequantize(const Tensor& packed, const Tensor& absmax_in, int64_t blocksize, Tensor out) {
  dense(packed, "packed"); dense(absmax_in, "absmax"); dense(out, "out");
  TORCH_CHECK(out.numel() == packed.numel() * 2 && absmax_in.numel() * blocksize == out.numel(), "nf4 shapes");
  ok(oab::launch_nf4_dequantize((const uint8_t*)packed.data_ptr(), absmax_in.data_ptr<float>(), out.numel(),
                                (int)blocksize, out.data_ptr(), qdtype(out), cur()), "nf4_dequantize");
}

void int8_quantize(const Tensor& x, Tensor q, Tensor scales) {
  dense(x, "x"); dense(q, "q"); dense(scales, "scales");
  TORCH_CHECK(x.dim() == 2 && q.sizes() == x.sizes() && q.scalar_type() == at::kChar && scales.numel() == x.size(0), "int8 shapes");
  ok(oab::launch_int8_quantize(x.data_ptr(), qdtype(x), x.size(0), x.size(1), q.data_ptr<int8_t>(),
                               scales.data_ptr(), qdtype(scales), cur()), "int8_quantize");
}

void int8_dequantize(const Tensor& q, const Tensor& scales, Tensor out) {
  dense(q, "q"); dense(scales, "scales"); dense(out, "out");
  TORCH_CHECK(q.dim() == 2 && out.sizes() == q.sizes() && out.scalar_type() == scales.scalar_type(), "int8 shapes/dtypes");
  ok(oab::launch_int8_dequantize(q.data_ptr<int8_t>(), scales.data_ptr(), qdtype(scales), q.size(0), q.size(1),
                                 out.data_ptr(), cur()), "int8_dequantize");
}

void int4_quantize(const Tensor& x, int64_t group, Tensor qweight, Tensor scales) {
  dense(x, "x"); dense(qweight, "qweight"); dense(scales, "scales");
  const int64_t out_f = x.size(0), in_f = x.size(1);
  TORCH_CHECK(in_f % 128 == 0 && (group == 32 || group == 64 || group == 128), "int4 kernel: in_f % 128 == 0, group in {32,64,128}");
  TORCH_CHECK(qweight.scalar_type() == at::kInt && qweight.size(0) == in_f / 8 && qweight.size(1) == out_f, "qweight shape");
  TORCH_CHECK(scales.size(0) == in_f / group && scales.size(1) == out_f, "scales shape");
  ok(oab::launch_int4_quantize(x.data_ptr(), qdtype(x), out_f, in_f, (int)group, qweight.data_ptr<int32_t>(),
                               scales.data_ptr(), qdtype(scales), cur()), "int4_quantize");
}

void int4_dequantize(const Tensor& qweight, const Tensor& scales, int64_t group, Tensor out) {
  dense(qweight, "qweight"); dense(scales, "scales"); dense(out, "out");
  const int64_t out_f = out.size(0), in_f = out.size(1);
  TORCH_CHECK(in_f % 128 == 0 && (group == 32 || group == 64 || group == 128), "int4 kernel: in_f % 128 == 0, group in {32,64,128}");
  TORCH_CHECK(out.scalar_type() == scales.scalar_type(), "int4 dequant output dtype = scale dtype");
  ok(oab::launch_int4_dequantize(qweight.data_ptr<int32_t>(), scales.data_ptr(), qdtype(scales), out_f, in_f,
                                 (int)group, out.data_ptr(), cur()), "int4_dequantize");
}

void fake_quant(int64_t format, const Tensor& x, Tensor out, int64_t group, int64_t scale_dtype, const std::optional<Tensor>& amax) {
  dense(x, "x"); dense(out, "out");
  TORCH_CHECK(x.dim() == 2 && out.sizes() == x.sizes() && out.scalar_type() == x.scalar_type(), "fake_quant: out like x (2-D)");
  const float* ap = nullptr;
  int n_amax = 0;
  if (amax.has_value() && amax->defined()) {
    TORCH_CHECK(amax->is_cuda() && amax->scalar_type() == at::kFloat && amax->is_contiguous() && amax->numel() >= 1,
                "amax: contiguous CUDA fp32");
    ap = amax->data_ptr<float>();
    n_amax = (int)amax->numel();
  }
  ok(oab::launch_fake_quant((int)format, x.data_ptr(), out.data_ptr(), qdtype(x), x.size(0), x.size(1), (int)group,
                            (int)scale_dtype, ap, n_amax, cur()), "fake_quant");
}

// ---------------------------------------------------------------------------
// Linear layer on a packed weight
// ---------------------------------------------------------------------------
struct Packed {
  int64_t format = 0, group = 0, rows = 0, cols = 0;
  Tensor packed, scales, global_scale;
};

// Fills in rows and cols; false unless the kernels read exactly what these tensors hold
// (bf16 arithmetic: int4 and int8 scales are bf16).
bool packed_ok(Packed& w, const at::Device& dev) {
  auto here = [&](const Tensor& t) { return t.device() == dev && t.is_contiguous(); };
  if (!here(w.packed) || !here(w.scales)) return false;
  if (w.format == oab::kQInt8) {
    if (w.packed.dim() != 2 || w.packed.scalar_type() != at::kChar) return false;
    w.rows = w.packed.size(0);
    w.cols = w.packed.size(1);
    return w.scales.numel() == w.rows && w.scales.scalar_type() == at::kBFloat16;
  }
  if (w.format == oab::kQInt4) {
    if (w.packed.dim() != 2 || w.packed.scalar_type() != at::kInt) return false;
    w.rows = w.packed.size(1);
    w.cols = w.packed.size(0) * 8;
    return w.cols % 128 == 0 && (w.group == 32 || w.group == 64 || w.group == 128) && w.scales.dim() == 2 &&
           w.scales.size(0) == w.cols / w.group && w.scales.size(1) == w.rows && w.scales.scalar_type() == at::kBFloat16;
  }
  if (w.packed.dim() != 2 || w.packed.scalar_type() != at::kByte) return false;
  w.rows = w.packed.size(0);
  w.cols = w.packed.size(1) * 2;
  const int64_t n = w.rows * w.cols;
  if (reinterpret_cast<uintptr_t>(w.packed.data_ptr()) & 7u) return false;
  if (w.format == oab::kQNF4)
    return w.group >= 16 && w.group <= 512 && (w.group & (w.group - 1)) == 0 && w.cols % w.group == 0 &&
           w.scales.numel() * w.group == n && w.scales.scalar_type() == at::kFloat;
  return w.format == oab::kQNVFP4 && w.cols % 16 == 0 && w.scales.numel() * 16 == n && w.scales.element_size() == 1 &&
         w.global_scale.defined() && w.global_scale.device() == dev && w.global_scale.scalar_type() == at::kFloat;
}

Tensor packed_dense(const Packed& w) {
  Tensor out = at::empty({w.rows, w.cols}, w.packed.options().dtype(at::kBFloat16));
  switch (w.format) {
    case oab::kQNVFP4: nvfp4_dequantize(w.packed, w.scales, w.global_scale, out); break;
    case oab::kQNF4: nf4_dequantize(w.packed, w.scales, w.group, out); break;
    case oab::kQInt4: int4_dequantize(w.packed, w.scales, w.group, out); break;
    default: int8_dequantize(w.packed, w.scales, out);
  }
  return out;
}

// The few-token kernel's result, undefined when it does not take the call.
Tensor qgemv(const Packed& w, const Tensor& x, const Tensor& bias) {
  const int64_t tokens = x.numel() / w.cols;
  if (!oab::qgemv_supported((int)w.format, w.rows, w.cols, tokens, (int)w.group)) return Tensor();
  const Tensor xc = x.contiguous();
  if ((reinterpret_cast<uintptr_t>(xc.data_ptr()) & 31u) ||
      (reinterpret_cast<uintptr_t>(w.packed.data_ptr()) & (oab::qgemv_packed_align((int)w.format) - 1)))
    return Tensor();
  auto shape = x.sizes().vec();
  shape.back() = w.rows;
  Tensor y = at::empty(shape, x.options());
  ok(oab::launch_qgemv((int)w.format, w.packed.data_ptr(), w.scales.data_ptr(),
                       w.global_scale.defined() ? w.global_scale.data_ptr<float>() : nullptr, (int)w.group, xc.data_ptr(),
                       tokens, bias.defined() ? bias.data_ptr() : nullptr, y.data_ptr(), w.rows, w.cols, cur()), "qgemv");
  return y;
}

// The weight that a saved-tensor hook returned in place of forward's, another one or a dense
// tensor: its Python object is asked for its payload, as the Python node does.
Tensor other_weight(const Tensor& weight, at::ScalarType dtype) {
  at::NoGradGuard no_grad;
  Packed w;
  {
    py::gil_scoped_acquire gil;
    try {
      const py::object o = py::cast(weight);
      if (!py::hasattr(o, "KERNEL_PAYLOAD")) return weight.to(dtype);
      const py::tuple names = o.attr("KERNEL_PAYLOAD");
      w.format = o.attr("KERNEL_FORMAT").cast<int64_t>();
      w.group = o.attr("kernel_group")().cast<int64_t>();
      w.packed = o.attr(py::object(names[0])).cast<Tensor>();
      w.scales = o.attr(py::object(names[1])).cast<Tensor>();
      if (w.format == oab::kQNVFP4) w.global_scale = o.attr("global_scale").cast<Tensor>();
      if (!w.packed.is_cuda() || !packed_ok(w, w.packed.device()))
        return o.attr("dequantize")(py::cast(dtype)).cast<Tensor>();
    } catch (const py::error_already_set& e) {
      TORCH_CHECK(false, e.what());
    }
  }
  c10::cuda::CUDAGuard guard(w.packed.device());
  return packed_dense(w).to(dtype);
}

// y = x W^T + b.  `weight` is the wrapper that autograd knows; its packed tensors travel
// beside it.  The wrapper is saved as an input is: changing it in place before backward is an
// error, and saved-tensor hooks see it.  The products of backward are ordinary operations (they can
// be differentiated again).  333 tokens through 2816 x 1024 int4 with bias, forward and
// backward, a whole call (35 us of kernels): 189 us with the Python node, 135 with this one.
struct QLinear : torch::autograd::Function<QLinear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const std::optional<Tensor>& bias, const Packed& w) {
    c10::cuda::CUDAGuard guard(x.device());
    ctx->save_for_backward({x, weight});
    // One entry: seven of this map cost 2 us more per forward and backward (and asking the
    // Python object for the payload 10 to 20).
    ctx->saved_data["of"] = c10::ivalue::Tuple::create(std::vector<c10::IValue>{
        weight, w.packed, w.scales, w.global_scale, w.format, w.group, bias.has_value() && bias->defined()});
    const Tensor b = bias.has_value() ? *bias : Tensor();
    const Tensor few = qgemv(w, x, b);
    return few.defined() ? few : at::linear(x, packed_dense(w), bias);
  }
  static Tensor dense_weight(c10::ArrayRef<c10::IValue> of, const Tensor& weight, at::ScalarType dtype) {
    if (!weight.is_same(of[0].toTensor())) return other_weight(weight, dtype);
    Packed w;
    w.packed = of[1].toTensor();
    w.scales = of[2].toTensor();
    w.global_scale = of[3].toTensor();
    w.format = of[4].toInt();
    w.group = of[5].toInt();
    at::NoGradGuard no_grad;
    c10::cuda::CUDAGuard guard(w.packed.device());
    TORCH_CHECK(packed_ok(w, w.packed.device()), "the packed weight changed its layout between forward and backward");
    return packed_dense(w).to(dtype);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &weight = saved[1], &gy = grads[0];
    if (!gy.defined()) return {Tensor(), Tensor(), Tensor(), Tensor()};
    c10::cuda::CUDAGuard guard(gy.device());
    const c10::IValue kept = ctx->saved_data["of"];
    const c10::ArrayRef<c10::IValue> of = kept.toTupleRef().elements();
    const Tensor g2 = gy.reshape({-1, weight.size(0)});
    Tensor gx, gw, gb;
    if (ctx->needs_input_grad(0)) gx = g2.mm(dense_weight(of, weight, gy.scalar_type())).view(x.sizes());
    if (ctx->needs_input_grad(1)) gw = g2.t().mm(x.reshape({-1, weight.size(1)}));
    if (of[6].toBool() && ctx->needs_input_grad(2)) gb = g2.sum(0);
    return {gx, gw, gb, Tensor()};
  }
};

// nullopt when the call is not one for the kernels
std::optional<Tensor> qlinear(const Tensor& x, const Tensor& weight, const std::optional<Tensor>& bias, int64_t format, int64_t group,
                              const Tensor& packed, const Tensor& scales, const std::optional<Tensor>& global_scale) {
  if (!x.is_cuda() || x.scalar_type() != at::kBFloat16 || x.dim() < 1 || x.numel() == 0) return std::nullopt;
  Packed w;
  w.format = format;
  w.group = group;
  w.packed = packed;
  w.scales = scales;
  if (global_scale.has_value()) w.global_scale = *global_scale;
  if (!packed_ok(w, x.device()) || w.rows <= 0 || x.size(-1) != w.cols) return std::nullopt;
  if (bias.has_value() && bias->defined() &&
      (bias->device() != x.device() || bias->scalar_type() != at::kBFloat16 || bias->dim() != 1 || bias->numel() != w.rows ||
       !bias->is_contiguous()))
    return std::nullopt;
  return QLinear::apply(x, weight, bias, w);
}

}  // namespace

void bind_quant(py::module_& m) {
  m.def("absmax_partials", &absmax_partials);
  m.def("nvfp4_quantize", &nvfp4_quantize);
  m.def("nvfp4_dequantize", &nvfp4_dequantize);
  m.def("nf4_quantize", &nf4_quantize);
  m.def("nf4_dequantize", &nf4_dequantize);
  m.def("int8_quantize", &int8_quantize);
  m.def("int8_dequantize", &int8_dequantize);
  m.def("int4_quantize", &int4_quantize);
  m.def("int4_dequantize", &int4_dequantize);
  m.def("qlinear", &qlinear);
  m.def("fake_quant", &fake_quant, py::arg("format"), py::arg("x"), py::arg("out"), py::arg("group"),
        py::arg("scale_dtype"), py::arg("amax") = py::none());
}
