// Autograd functions of the elementwise model kernels and their Python bindings.  The
// graph nodes are C++ so that a call costs the host about what one PyTorch operation does.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include "model_ops.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

cudaStream_t cur() { return at::cuda::getCurrentCUDAStream().stream(); }
void ok(cudaError_t e, const char* what) { TORCH_CHECK(e == cudaSuccess, what, ": ", cudaGetErrorString(e)); }
void check_bf16(const Tensor& t, const char* name) {
  TORCH_CHECK(t.is_cuda() && t.scalar_type() == at::kBFloat16, name, " must be a bf16 CUDA tensor");
}

// --------------------------------------------------------------------- SwiGLU
struct SwiGLU : torch::autograd::Function<SwiGLU> {
  static Tensor forward(AutogradContext* ctx, const Tensor& g, const Tensor& u) {
    check_bf16(g, "gate");
    check_bf16(u, "up");
    TORCH_CHECK(g.sizes() == u.sizes() && g.device() == u.device(), "gate and up must have one shape and device");
    c10::cuda::CUDAGuard guard(g.device());
    const Tensor gc = g.contiguous(), uc = u.contiguous();
    Tensor y = at::empty_like(gc);
    ok(oab::launch_swiglu(gc.data_ptr(), uc.data_ptr(), y.data_ptr(), y.numel(), cur()), "swiglu");
    ctx->save_for_backward({g, u});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &g = saved[0], &u = saved[1], &gy = grads[0];
    if (!gy.defined()) return {Tensor(), Tensor()};
    if (at::GradMode::is_enabled()) {  // a graph of the gradient is asked for
      const Tensor s = at::sigmoid(g);
      return {gy * u * s * (1 + g * (1 - s)), gy * at::silu(g)};
    }
    c10::cuda::CUDAGuard guard(g.device());
    const Tensor c = gy.to(at::kBFloat16).contiguous(), gc = g.contiguous(), uc = u.contiguous();
    Tensor gg = at::empty_like(gc), gu = at::empty_like(uc);
    ok(oab::launch_swiglu_grad(c.data_ptr(), gc.data_ptr(), uc.data_ptr(), gg.data_ptr(), gu.data_ptr(), gc.numel(), cur()),
       "swiglu_grad");
    return {gg, gu};
  }
};

// ----------------------------------------------------------------------- RoPE
// (batch, seq, heads, dim) with unit stride along dim and 16-byte aligned heads
Tensor rope_layout(const Tensor& x) {
  const bool fits = x.stride(3) == 1 && x.stride(0) % 8 == 0 && x.stride(1) % 8 == 0 && x.stride(2) % 8 == 0 &&
                    (reinterpret_cast<uintptr_t>(x.data_ptr()) & 15u) == 0;
  return fits ? x : x.clone(at::MemoryFormat::Contiguous);
}
oab::RopeTensor rope_arg(const Tensor& x, const Tensor& y) {
  oab::RopeTensor t;
  if (!x.defined()) return t;
  t.in = x.data_ptr();
  t.out = y.data_ptr();
  t.sb = x.stride(0);
  t.ss = x.stride(1);
  t.sh = x.stride(2);
  t.heads = (int)x.size(2);
  return t;
}
// either of q, k may be undefined
variable_list rope_run(const Tensor& q, const Tensor& k, const Tensor& cos, const Tensor& sin, bool transposed) {
  const Tensor& any = q.defined() ? q : k;
  if (!any.defined()) return {Tensor(), Tensor()};
  c10::cuda::CUDAGuard guard(any.device());
  const Tensor qi = q.defined() ? rope_layout(q) : q, ki = k.defined() ? rope_layout(k) : k;
  const Tensor qo = q.defined() ? at::empty(q.sizes(), q.options()) : q;
  const Tensor ko = k.defined() ? at::empty(k.sizes(), k.options()) : k;
  ok(oab::launch_rope(rope_arg(qi, qo), rope_arg(ki, ko), cos.data_ptr(), sin.data_ptr(), any.size(0), any.size(1),
                      (int)any.size(3), transposed, cur()), "rope");
  return {qo, ko};
}
Tensor rope_grad_graph(const Tensor& g, const Tensor& cos, const Tensor& sin) {
  if (!g.defined()) return g;
  const int64_t half = g.size(3) / 2;
  const Tensor z = g * sin.unsqueeze(1);
  return g * cos.unsqueeze(1) + at::cat({z.narrow(3, half, half), -z.narrow(3, 0, half)}, 3);
}

struct Rope : torch::autograd::Function<Rope> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& cos, const Tensor& sin) {
    check_bf16(q, "q");
    check_bf16(k, "k");
    check_bf16(cos, "cos");
    check_bf16(sin, "sin");
    TORCH_CHECK(q.dim() == 4 && k.dim() == 4 && q.size(0) == k.size(0) && q.size(1) == k.size(1) &&
                    q.size(3) == k.size(3) && q.size(3) % 16 == 0, "rope: (batch, seq, heads, dim), dim % 16 == 0");
    TORCH_CHECK(cos.dim() == 2 && cos.sizes() == sin.sizes() && cos.size(0) == q.size(1) && cos.size(1) == q.size(3) &&
                    cos.is_contiguous() && sin.is_contiguous(), "rope: contiguous (seq, dim) tables");
    ctx->set_materialize_grads(false);  // either head tensor may go unused
    ctx->save_for_backward({cos, sin});
    return rope_run(q, k, cos, sin, false);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    if (at::GradMode::is_enabled())
      return {rope_grad_graph(grads[0], saved[0], saved[1]), rope_grad_graph(grads[1], saved[0], saved[1]), Tensor(), Tensor()};
    auto out = rope_run(grads[0], grads[1], saved[0], saved[1], true);
    return {out[0], out[1], Tensor(), Tensor()};
  }
};

// -------------------------------------------------------------------- RMSNorm
bool norm_layout(const Tensor& t) {
  return t.is_contiguous() && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0;
}
Tensor norm_operand(const Tensor& t) { return norm_layout(t) ? t : t.clone(at::MemoryFormat::Contiguous); }

// r defined: {x + r, norm(x + r) * w}; else {norm(x) * w}
variable_list norm_forward(AutogradContext* ctx, const Tensor& x, const Tensor& r, const Tensor& w, double eps) {
  check_bf16(x, "x");
  check_bf16(w, "weight");
  const int64_t cols = x.size(-1);
  TORCH_CHECK(cols % 8 == 0 && cols <= oab::kNormMaxCols && w.dim() == 1 && w.size(0) == cols, "rms_norm: unsupported shape");
  const bool add = r.defined();
  if (add) {
    check_bf16(r, "residual");
    TORCH_CHECK(r.sizes() == x.sizes() && r.device() == x.device(), "rms_norm: residual like x");
  }
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t rows = x.numel() / cols;
  const Tensor xc = norm_operand(x), rc = add ? norm_operand(r) : r, wc = norm_operand(w);
  Tensor out = at::empty(x.sizes(), x.options()), sum = add ? at::empty(x.sizes(), x.options()) : Tensor();
  Tensor rstd = at::empty({rows}, x.options().dtype(at::kFloat));
  ok(oab::launch_rms_norm(xc.data_ptr(), add ? rc.data_ptr() : nullptr, wc.data_ptr(), add ? sum.data_ptr() : nullptr,
                          out.data_ptr(), rstd.data_ptr<float>(), rows, (int)cols, (float)eps, cur()), "rms_norm");
  ctx->set_materialize_grads(false);
  ctx->saved_data["eps"] = eps;
  ctx->save_for_backward({add ? sum : x, w, rstd});
  if (add) return {sum, out};
  return {out};
}
// {dx, dw} from the gradients of the sum (may be undefined) and of the norm
variable_list norm_backward(AutogradContext* ctx, const Tensor& gsum, const Tensor& g, bool want_w) {
  if (!g.defined()) return {gsum, Tensor()};
  const auto saved = ctx->get_saved_variables();
  const Tensor &x = saved[0], &w = saved[1], &rstd = saved[2];
  Tensor dx, dw;
  if (at::GradMode::is_enabled()) {  // a graph of the gradient is asked for
    const Tensor x32 = x.to(at::kFloat);
    const Tensor rs = at::rsqrt(x32.square().mean({-1}, true) + ctx->saved_data["eps"].toDouble());
    const Tensor h = x32 * rs, gw = g.to(at::kFloat) * w.to(at::kFloat);
    dx = (rs * (gw - h * (gw * h).mean({-1}, true))).to(x.scalar_type());
    if (gsum.defined()) dx = dx + gsum;
    dw = (g.to(at::kFloat) * h).reshape({-1, w.size(0)}).sum(0).to(w.scalar_type());
    return {dx, dw};
  }
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t cols = x.size(-1), rows = x.numel() / cols;
  const Tensor gc = norm_operand(g.to(at::kBFloat16)), xc = norm_operand(x), wc = norm_operand(w), rc = rstd.contiguous();
  const Tensor sc = gsum.defined() ? norm_operand(gsum.to(at::kBFloat16)) : gsum;
  dx = at::empty(x.sizes(), x.options());
  Tensor partials;
  if (want_w) {
    dw = at::empty(w.sizes(), w.options());
    partials = at::empty({(int64_t)oab::rms_norm_partials(rows, (int)cols) * cols}, rstd.options());
  }
  ok(oab::launch_rms_norm_grad(gc.data_ptr(), sc.defined() ? sc.data_ptr() : nullptr, xc.data_ptr(), wc.data_ptr(),
                               rc.data_ptr<float>(), dx.data_ptr(), want_w ? dw.data_ptr() : nullptr,
                               want_w ? partials.data_ptr<float>() : nullptr, rows, (int)cols, cur()), "rms_norm_grad");
  return {dx, dw};
}

struct RmsNorm : torch::autograd::Function<RmsNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, double eps) {
    return norm_forward(ctx, x, Tensor(), w, eps)[0];
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto d = norm_backward(ctx, Tensor(), grads[0], ctx->needs_input_grad(1));
    return {d[0], d[1], Tensor()};
  }
};

struct AddRmsNorm : torch::autograd::Function<AddRmsNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& r, const Tensor& w, double eps) {
    return norm_forward(ctx, x, r, w, eps);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    auto d = norm_backward(ctx, grads[0], grads[1], ctx->needs_input_grad(2));
    return {d[0], d[0], d[1], Tensor()};
  }
};

// ------------------------------------------------------------------ embedding
struct Embedding : torch::autograd::Function<Embedding> {
  static Tensor forward(AutogradContext* ctx, const Tensor& weight, const Tensor& ids) {
    check_bf16(weight, "embedding table");
    TORCH_CHECK(weight.dim() == 2 && weight.size(1) % 8 == 0 && ids.scalar_type() == at::kLong && ids.device() == weight.device() &&
                    ids.numel() <= oab::kEmbedMaxTokens, "embedding: unsupported call");
    ctx->save_for_backward({ids});
    ctx->saved_data["vocab"] = weight.size(0);
    return at::embedding(weight, ids);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor ids = ctx->get_saved_variables()[0], &g = grads[0];
    const int64_t vocab = ctx->saved_data["vocab"].toInt();
    if (!g.defined()) return {Tensor(), Tensor()};
    if (at::GradMode::is_enabled()) return {at::embedding_dense_backward(g, ids, vocab, -1, false), Tensor()};
    c10::cuda::CUDAGuard guard(g.device());
    const int64_t cols = g.size(-1), n = ids.numel();
    const Tensor gc = norm_operand(g.to(at::kBFloat16)), ic = ids.contiguous();
    Tensor dw = at::empty({vocab, cols}, gc.options());
    Tensor work = at::empty({oab::embed_work_ints(n, vocab)}, gc.options().dtype(at::kInt));
    ok(oab::launch_embed_grad(gc.data_ptr(), ic.data_ptr<int64_t>(), n, dw.data_ptr(), vocab, (int)cols, work.data_ptr<int>(), cur()),
       "embed_grad");
    return {dw, Tensor()};
  }
};

}  // namespace

void bind_model(py::module_& m) {
  m.def("swiglu", [](const Tensor& g, const Tensor& u) { return SwiGLU::apply(g, u); });
  m.def("rms_norm", [](const Tensor& x, const Tensor& w, double eps) { return RmsNorm::apply(x, w, eps); });
  m.def("add_rms_norm", [](const Tensor& x, const Tensor& r, const Tensor& w, double eps) {
    auto out = AddRmsNorm::apply(x, r, w, eps);
    return std::make_pair(out[0], out[1]);
  });
  m.def("embedding", [](const Tensor& weight, const Tensor& ids) { return Embedding::apply(weight, ids); });
  m.def("embed_kernel_wins", &oab::embed_kernel_wins);
  m.attr("EMBED_MAX_TOKENS") = oab::kEmbedMaxTokens;
  m.attr("NORM_MAX_COLS") = oab::kNormMaxCols;
  m.def("rope", [](const Tensor& q, const Tensor& k, const Tensor& cos, const Tensor& sin) {
    auto out = Rope::apply(q, k, cos, sin);
    return std::make_pair(out[0], out[1]);
  });
}
