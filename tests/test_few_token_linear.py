"""Linear layers on packed weights: a few tokens straight from the packed words, against
fp64, and the autograd node."""

import pytest
import torch
import torch.nn.functional as F

from offload_adam_b200.qweight import Int4QWeight, Int8QWeight, NF4QWeight, NVFP4QWeight

pytestmark = pytest.mark.gpu


def _case(cls, rows, cols, tokens, bias, **kw):
    gen = torch.Generator(device="cuda").manual_seed(rows + cols + tokens)

    def normal(*shape, std=1.0):
        return (torch.randn(*shape, device="cuda", generator=gen) * std).to(torch.bfloat16)

    w = torch.nn.Parameter(cls.from_float(normal(rows, cols, std=0.02), **kw), requires_grad=False)
    return w, normal(tokens, cols), normal(rows) if bias else None


def _takes_packed_words(w, x, b=None):
    """Whether ``F.linear`` multiplies with the packed words: no dense bf16 copy of the weight is
    allocated (what it does allocate is smaller: the result, and x made contiguous)."""
    with torch.no_grad():
        F.linear(x, w, b)  # the library's workspace
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        y = F.linear(x, w, b)
    return torch.cuda.max_memory_allocated() - before < 2 * w.shape[0] * w.shape[1], y


def _check(w, x, b, y):
    dense = w.data.dequantize(torch.float32).double()
    want = x.double() @ dense.T + (0 if b is None else b.double())
    # one rounding to bf16, plus fp32 rounding of a sum of cols products
    slack = 2.0 ** -20 * (x.double().abs() @ dense.abs().T + 1e-30)
    assert y.shape == (*x.shape[:-1], w.shape[0]) and y.dtype == torch.bfloat16
    assert ((y.double() - want).abs() <= 1.01 * 2.0 ** -8 * want.abs() + slack).all()


# rows around the launch shapes (1, 592 and 4736 rows) and their remainders; columns
# around one warp step (512) and one CTA step (2048)
@pytest.mark.parametrize("cls,kw", [(NVFP4QWeight, {}), (NF4QWeight, {}), (NF4QWeight, {"blocksize": 16}),
                                    (NF4QWeight, {"blocksize": 512}), (Int8QWeight, {}), (Int4QWeight, {}),
                                    (Int4QWeight, {"group_size": 64}), (Int4QWeight, {"group_size": 32})])
@pytest.mark.parametrize("rows,cols", [(1, 512), (5, 1024), (591, 2048), (593, 4608), (4741, 512), (4736, 2560)])
@pytest.mark.parametrize("tokens", [1, 2, 3, 4])
def test_few_tokens(cls, kw, rows, cols, tokens):
    w, x, b = _case(cls, rows, cols, tokens, bias=tokens % 2 == 0, **kw)
    few, y = _takes_packed_words(w, x, b)
    if cls is Int4QWeight and (rows < 1024 or tokens > 2):
        assert not few
        dense = x @ w.data.dequantize(torch.bfloat16).T  # the dense route
        assert torch.equal(y, dense if b is None else F.linear(x, w.data.dequantize(torch.bfloat16), b))
        return
    assert few
    _check(w, x, b, y)


@pytest.mark.parametrize("cls,cols", [(NVFP4QWeight, 16), (NF4QWeight, 64), (Int8QWeight, 48)])
def test_narrow_weights(cls, cols):
    w, x, b = _case(cls, 33, cols, 4, bias=True)
    few, y = _takes_packed_words(w, x.view(2, 2, cols), b)
    assert few
    _check(w, x.view(2, 2, cols), b, y)


def test_other_calls_keep_the_dense_route():
    """More tokens, other dtypes, ragged columns, other scale types, non-contiguous
    or misaligned activations: same result as before."""
    for cls, cols, tokens, kw in ((NF4QWeight, 256, 5, {}), (Int8QWeight, 36, 2, {}),
                                  (Int4QWeight, 256, 1, {"scale_dtype": torch.float32})):
        w, x, b = _case(cls, 40, cols, tokens, bias=False, **kw)
        few, y = _takes_packed_words(w, x)
        assert not few and torch.equal(y, x @ w.data.dequantize(torch.bfloat16).T)
    w, x, b = _case(NF4QWeight, 40, 256, 2, bias=False)
    with torch.no_grad():
        assert torch.equal(F.linear(x.half(), w), x.half() @ w.data.dequantize(torch.float16).T)
        _check(w, x, None, F.linear(x.T.contiguous().T, w))          # strided
        shifted = torch.empty(513, device="cuda", dtype=torch.bfloat16)[1:].view(2, 256).copy_(x)
        few, y = _takes_packed_words(w, shifted)                     # not 32-byte aligned
        assert not few and torch.equal(y, x @ w.data.dequantize(torch.bfloat16).T)
        few, _ = _takes_packed_words(w, x.T.contiguous().T)
        assert few


def test_gradients_of_a_few_tokens():
    w, x, b = _case(NF4QWeight, 96, 256, 3, bias=True)
    w.requires_grad_(True)
    x.requires_grad_(True)
    y = F.linear(x, w, b)
    gy = torch.ones_like(y)
    y.backward(gy)
    dense = w.data.dequantize(torch.bfloat16)
    assert torch.equal(x.grad, gy @ dense)
    assert torch.equal(w.grad, gy.T @ x.detach())


@pytest.mark.parametrize("cls,kw", [(NVFP4QWeight, {}), (NF4QWeight, {}), (Int4QWeight, {"group_size": 64}), (Int8QWeight, {})])
@pytest.mark.parametrize("shape", [(37,), (3, 11)])
@pytest.mark.parametrize("bias", [False, True])
def test_autograd_node_matches_the_general_one(cls, kw, shape, bias):
    """More tokens than the few-token kernel takes: the C++ node against the Python node."""
    from offload_adam_b200.qweight.base import _WeightOnlyLinear

    rows, cols = 96, 256
    n = torch.Size(shape).numel()
    w, x, b = _case(cls, rows, cols, n, bias, **kw)
    x, gy = x.view(*shape, cols), _case(cls, rows, rows * 4, n, False)[1][:, :rows].reshape(*shape, rows)
    out = []
    for fn in (F.linear, _WeightOnlyLinear.apply):
        wi = torch.nn.Parameter(w.data)
        xi = x.clone().requires_grad_(True)
        bi = torch.nn.Parameter(b.clone()) if bias else None
        y = fn(xi, wi, bi)
        y.backward(gy)
        out.append([y.detach(), xi.grad, wi.grad] + ([bi.grad] if bias else []))
    for i, (a, c) in enumerate(zip(*out)):
        if i == 0 and bias:  # the sum with the bias rounds once, there twice
            assert ((a.double() - c.double()).abs() <= 2.0 ** -7 * c.double().abs() + 2.0 ** -7).all()
        else:
            assert torch.equal(a, c)


def test_autograd_node_with_frozen_inputs_and_second_derivative():
    w, x, _ = _case(NF4QWeight, 64, 128, 20, False)
    frozen = torch.nn.Parameter(w.data, requires_grad=False)
    x.requires_grad_(True)
    y = F.linear(x, frozen)
    gx, = torch.autograd.grad(y.float().square().sum(), x, create_graph=True)
    hx, = torch.autograd.grad(gx.float().sum(), x)
    assert frozen.grad is None and hx.isfinite().all() and hx.abs().max() > 0
    trained = torch.nn.Parameter(w.data)
    F.linear(x.detach(), trained).sum().backward()  # only the weight needs a gradient
    assert trained.grad.shape == (64, 128)
    with torch.no_grad():
        assert not F.linear(x, trained).requires_grad
    mixed = torch.autograd.graph.save_on_cpu()
    with mixed:
        z = F.linear(x, trained)
    g1, = torch.autograd.grad(z.sum(), x)
    g2, = torch.autograd.grad(F.linear(x, trained).sum(), x)
    assert torch.equal(g1, g2)


@pytest.mark.parametrize("cls,kw", [(NVFP4QWeight, {}), (NF4QWeight, {}), (Int4QWeight, {}), (Int8QWeight, {})])
@pytest.mark.parametrize("tokens", [1, 20])
def test_weight_changed_in_place_before_backward_is_an_error(cls, kw, tokens):
    """As for a dense weight: the gradient would belong to another weight than the result."""
    w, x, _ = _case(cls, 64, 128, tokens, False, **kw)
    x.requires_grad_(True)
    y = F.linear(x, w)
    with torch.no_grad():
        w.copy_(torch.ones(64, 128, device="cuda", dtype=torch.bfloat16))
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()


@pytest.mark.parametrize("cls,kw", [(NVFP4QWeight, {}), (NF4QWeight, {}), (Int4QWeight, {}), (Int8QWeight, {})])
def test_saved_tensor_hooks_see_the_weight(cls, kw):
    w, x, _ = _case(cls, 64, 128, 20, False, **kw)
    other, _, _ = _case(cls, 64, 128, 21, False, **kw)
    x.requires_grad_(True)
    seen = []

    def pack(t):
        seen.append(t)
        return t

    # backward uses what the hook returns: another packed weight, or a dense one
    for back, want in ((lambda t: other.data, other), (lambda t: t.detach().dequantize(), w)):
        seen.clear()
        with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: back(t) if isinstance(t, cls) else t):
            y = F.linear(x, w)
            gx, = torch.autograd.grad(y.sum(), x)
        assert any(isinstance(t, cls) for t in seen)
        assert torch.equal(gx, torch.ones_like(y) @ want.data.dequantize(torch.bfloat16))
