"""Elementwise model kernels against the same formulas in fp64 PyTorch."""

import pytest
import torch
import torch.nn.functional as F

from offload_adam_b200 import _ext
from offload_adam_b200.models import llama
from offload_adam_b200.models.llama import _apply_rope, _rope_tables, build_llama, tiny_llama

pytestmark = pytest.mark.gpu


def _rand(*shape, seed=0, std=1.0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=gen) * std).to(torch.bfloat16)


def _close(got, want, slack=1.01):
    """One rounding to bf16 (8 significant bits: 2^-8 of the value) on top of a few fp32 ulp."""
    err = (got.double() - want).abs()
    assert (err <= slack * 2.0 ** -8 * want.abs() + 1e-6 * want.abs().max() + 1e-37).all(), err.max().item()


@pytest.mark.parametrize("n", [1, 15, 16, 17, 4096, 4097, 100003])
def test_swiglu(n):
    C = _ext.load(required=True)
    g, u, gy = _rand(n, seed=1, std=4.0), _rand(n, seed=2), _rand(n, seed=3)
    g[0] = -80.0
    a, b = g.clone().requires_grad_(True), u.clone().requires_grad_(True)
    y = C.swiglu(a, b)
    y.backward(gy)
    a64, b64 = g.double().requires_grad_(True), u.double().requires_grad_(True)
    y64 = F.silu(a64) * b64
    y64.backward(gy.double())
    _close(y.detach(), y64.detach())
    _close(a.grad, a64.grad)
    _close(b.grad, b64.grad)


def test_swiglu_keeps_fp32_precision():
    """Where an approximate exponential is off by more: for large negative gates."""
    C = _ext.load(required=True)
    gen = torch.Generator(device="cuda").manual_seed(0)
    g = (-40 - 46 * torch.rand(1 << 20, device="cuda", generator=gen)).to(torch.bfloat16)
    u = (1 + torch.rand(1 << 20, device="cuda", generator=gen)).to(torch.bfloat16)
    want = F.silu(g.double()) * u.double()
    # three fp32 roundings and exp's: 2^-22 in all, which changes that / 2^-8 of the bf16 roundings
    assert (C.swiglu(g, u) != want.float().to(torch.bfloat16)).double().mean() <= 3e-4


def test_swiglu_views_and_second_derivative():
    C = _ext.load(required=True)
    base = _rand(64, 70, seed=4)
    g, u = base[:, 1:33], base.t()[:64, :32].contiguous()[:, :32]
    _close(C.swiglu(g, u), F.silu(g.double()) * u.double())
    a = _rand(40, seed=5).requires_grad_(True)
    b = _rand(40, seed=6)
    d, = torch.autograd.grad(C.swiglu(a, b).float().sum(), a, create_graph=True)
    dd, = torch.autograd.grad(d.float().sum(), a)
    a64 = a.detach().double().requires_grad_(True)
    d64, = torch.autograd.grad((F.silu(a64) * b.double()).sum(), a64, create_graph=True)
    dd64, = torch.autograd.grad(d64.sum(), a64)
    assert (dd.double() - dd64).norm() <= 2e-2 * dd64.norm()


@pytest.mark.parametrize("dim", [16, 32, 64, 96, 128])
@pytest.mark.parametrize("batch,seq,heads,kv", [(1, 1, 1, 1), (2, 17, 4, 2), (1, 300, 5, 5)])
def test_rope(dim, batch, seq, heads, kv):
    C = _ext.load(required=True)
    cos, sin = (t.to(torch.bfloat16) for t in _rope_tables(seq, dim, 1e4, "cuda"))
    q, k = _rand(batch, seq, heads, dim, seed=1), _rand(batch, seq, kv, dim, seed=2)
    gq = _rand(batch, heads, seq, dim, seed=3).transpose(1, 2)  # as attention hands it back
    gk = _rand(batch, seq, kv, dim, seed=4)
    a, b = q.clone().requires_grad_(True), k.clone().requires_grad_(True)
    for use in ("both", "q"):
        a.grad = b.grad = None
        qo, ko = C.rope(a, b, cos, sin)
        torch.autograd.backward([qo, ko] if use == "both" else [qo], [gq, gk] if use == "both" else [gq])
        for x, y, grad, g in ((q, qo, a.grad, gq), (k, ko, b.grad, gk)):
            x64 = x.double().requires_grad_(True)
            y64 = _apply_rope(x64.transpose(1, 2), cos.double(), sin.double()).transpose(1, 2)
            y64.backward(g.double())
            # the two products cancel: one rounding of the larger of them
            bound = 1.01 * 2.0 ** -8 * y64.detach().abs() + 1e-6
            assert ((y.detach().double() - y64.detach()).abs() <= bound).all()
            if use == "q" and x is k:
                assert grad is None or grad.abs().max() == 0
            else:
                assert ((grad.double() - x64.grad).abs() <= 1.01 * 2.0 ** -8 * x64.grad.abs() + 1e-6).all()


def _norm64(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


# a warp's row ends at 1024 columns, a CTA's with 2, 4 and 8 vectors a thread at 4096, 8192
# and 16384; rows around the groups that share them in backward (444 CTAs, 2368 warps)
@pytest.mark.parametrize("cols", [8, 256, 840, 1024, 1032, 4096, 4104, 8192, 16384])
@pytest.mark.parametrize("rows", [1, 9, 445, 2371])
@pytest.mark.parametrize("add", [False, True])
def test_rms_norm(cols, rows, add):
    C = _ext.load(required=True)
    x, r, g, gs = (_rand(rows, cols, seed=s) for s in range(4))
    w = (1 + 0.1 * _rand(cols, seed=9).float()).to(torch.bfloat16).requires_grad_(True)
    a, b = x.clone().requires_grad_(True), r.clone().requires_grad_(True)
    if add:
        s, n = C.add_rms_norm(a, b, w, 1e-5)
        assert torch.equal(s.detach(), x + r)
        torch.autograd.backward([s, n], [gs, g])
    else:
        n = C.rms_norm(a, w, 1e-5)
        n.backward(g)
    y = (x + r if add else x).double().requires_grad_(True)
    w64 = w.detach().double().requires_grad_(True)
    n64 = _norm64(y, w64, 1e-5)
    torch.autograd.backward([n64, y * 1.0] if add else [n64], [g.double(), gs.double()] if add else [g.double()])
    _close(n.detach(), n64.detach())
    # fp32 sums over a row and over the rows: relative to what is summed
    assert ((a.grad.double() - y.grad).abs() <= 1.01 * 2.0 ** -8 * y.grad.abs() + 1e-5).all()
    slack = 2.0 ** -20 * (g.double() * y.detach()).abs().sum(0)
    assert ((w.grad.double() - w64.grad).abs() <= 1.01 * 2.0 ** -8 * w64.grad.abs() + slack).all()
    assert not add or torch.equal(a.grad, b.grad)


def test_rms_norm_of_which_one_output_is_used_and_second_derivative():
    C = _ext.load(required=True)
    x, r = _rand(5, 64, seed=1).requires_grad_(True), _rand(5, 64, seed=2).requires_grad_(True)
    w = torch.ones(64, device="cuda", dtype=torch.bfloat16)
    s, n = C.add_rms_norm(x, r, w, 1e-5)
    gx, = torch.autograd.grad(s, x, torch.ones_like(s), retain_graph=True)
    assert torch.equal(gx, torch.ones_like(gx))
    gx, = torch.autograd.grad(n, x, torch.ones_like(n), create_graph=True)
    hx, = torch.autograd.grad(gx.float().square().sum(), x)
    y = (x + r).detach().double().requires_grad_(True)
    g64, = torch.autograd.grad(_norm64(y, w.double(), 1e-5).sum(), y, create_graph=True)
    h64, = torch.autograd.grad(g64.square().sum(), y)
    assert (hx.double() - h64).norm() <= 5e-2 * h64.norm()


def test_hooks_on_a_norm_still_see_its_calls():
    model = build_llama(tiny_llama(), device="cuda", seed=1)
    ids = torch.randint(0, 1024, (1, 9), device="cuda")
    plain, seen = model(ids), []
    model.model.layers[0].post_attention_layernorm.register_forward_hook(lambda m, i, o: seen.append(o))
    assert torch.equal(model(ids), plain) and len(seen) == 1 and seen[0].shape == (1, 9, 256)


@pytest.mark.parametrize("where", ["instance", "class"])
def test_replaced_forward_is_called(where, monkeypatch):
    """As adapters do it: a norm's or the embedding's ``forward`` is put in its place."""
    model = build_llama(tiny_llama(), device="cuda", seed=1)
    ids = torch.randint(0, 1024, (1, 9), device="cuda")
    seen = []
    for module in (model.model.layers[1].post_attention_layernorm, model.model.embed_tokens):
        cls, original = type(module), type(module).forward

        def forward(self, x, original=original):
            seen.append(type(self))
            return original(self, x)

        if where == "instance":
            module.forward = forward.__get__(module)
        else:
            monkeypatch.setattr(cls, "forward", forward)
    model(ids, labels=ids).backward()
    norms = [c for c in seen if c is llama.RMSNorm]
    assert len(norms) == (1 if where == "instance" else 5) and seen.count(torch.nn.Embedding) == 1


def test_model_takes_the_torch_route_where_kernels_may_not_run():
    """Autocast, function modes and second derivatives of the whole model still work, and
    the two routes agree."""
    model = build_llama(tiny_llama(), device="cuda", seed=1)
    ids = torch.randint(0, 1024, (2, 33), device="cuda")

    class Watch(torch.overrides.TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    C = _ext.load(required=True)
    with torch.no_grad():
        n0 = C.launch_count()
        kernels = model(ids)
        n1 = C.launch_count()
        with Watch():
            torch_route = model(ids)
        assert n1 > n0 and C.launch_count() == n1
        with torch.autocast("cuda", dtype=torch.bfloat16):
            assert torch.allclose(model(ids).float(), torch_route.float(), rtol=0.1, atol=0.1)
    assert (kernels.float() - torch_route.float()).norm() <= 2e-2 * torch_route.float().norm()
    w = model.model.layers[0].mlp.gate_proj.weight
    g, = torch.autograd.grad(model(ids).float().square().mean(), w, create_graph=False)
    assert g.isfinite().all()
    assert torch.func.jvp(lambda x: model.model.layers[0].mlp(x), (_rand(3, 256),), (_rand(3, 256),))[1].isfinite().all()


def test_model_on_an_empty_sequence():
    model = build_llama(tiny_llama(), device="cuda", seed=1)
    ids = torch.zeros(2, 0, dtype=torch.int64, device="cuda")
    logits = model(ids)
    assert logits.shape == (2, 0, 1024)
    logits.sum().backward()
    assert model.model.layers[0].self_attn.q_proj.weight.grad.abs().max() == 0


def test_rope_of_an_empty_batch():
    C = _ext.load(required=True)
    cos, sin = (t.to(torch.bfloat16) for t in _rope_tables(8, 32, 1e4, "cuda"))
    q, k = _rand(0, 8, 4, 32).requires_grad_(True), _rand(0, 8, 2, 32).requires_grad_(True)
    qo, ko = C.rope(q, k, cos, sin)
    assert qo.shape == q.shape and ko.shape == k.shape
    (qo.sum() + ko.sum()).backward()
    assert q.grad.shape == q.shape and k.grad.shape == k.shape


# columns around a warp's 256; tokens around the order kernel's tile (2048) and its CTAs (64);
# rows with none, some, more than 8 and all tokens; ids drawn from a few rows or all
@pytest.mark.parametrize("cols", [8, 256, 264, 1000])
@pytest.mark.parametrize("n,vocab,spread", [(1, 5, 5), (63, 1000, 1000), (65, 40, 3), (2049, 3001, 3001), (2048, 700, 1),
                                            (5000, 131, 131)])
def test_embedding_gradient(cols, n, vocab, spread):
    C = _ext.load(required=True)
    w = _rand(vocab, cols, seed=1).requires_grad_(True)
    ids = torch.randint(0, spread, (n,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    g = _rand(n, cols, seed=2)
    y = C.embedding(w, ids)
    assert torch.equal(y, w[ids])
    y.backward(g)
    want = torch.zeros(vocab, cols, device="cuda", dtype=torch.float64).index_add_(0, ids, g.double())
    slack = 2.0 ** -20 * torch.zeros_like(want).index_add_(0, ids, g.double().abs())  # fp32 sums
    assert ((w.grad.double() - want).abs() <= 1.01 * 2.0 ** -8 * want.abs() + slack).all()


def test_embedding_of_the_model_and_its_limits():
    C = _ext.load(required=True)
    model = build_llama(tiny_llama(tie_embeddings=False), device="cuda", seed=1)
    ids = torch.randint(0, 1024, (2, 40), device="cuda")
    table = model.model.embed_tokens.weight
    out = []
    for watched in (False, True):
        if watched:  # a hook on the module: PyTorch's own gradient
            model.model.embed_tokens.register_forward_hook(lambda m, i, o: None)
        table.grad = None
        n0 = C.launch_count()
        model(ids, labels=ids).backward()
        out.append((table.grad.clone(), C.launch_count() - n0))
    assert out[0][1] == out[1][1] + 3
    assert (out[0][0].float() - out[1][0].float()).norm() <= 1e-2 * out[1][0].float().norm()
    with pytest.raises(RuntimeError):
        C.embedding(table, torch.zeros(C.EMBED_MAX_TOKENS + 1, dtype=torch.int64, device="cuda"))


@pytest.mark.parametrize("n,vocab,cols,kernel", [(12288, 1024, 64, True), (12289, 1024, 64, False), (16384, 8000, 1000, True),
                                                 (16385, 8000, 1000, False), (24576, 100000, 1000, True),
                                                 (24577, 100000, 1000, False)])
def test_embedding_gradient_takes_the_kernel_where_it_wins(n, vocab, cols, kernel):
    C = _ext.load(required=True)
    module = torch.nn.Embedding(vocab, cols, device="cuda", dtype=torch.bfloat16)
    ids = torch.randint(0, vocab, (n,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    n0 = C.launch_count()
    llama._embed(module, ids).backward(torch.ones(n, cols, device="cuda", dtype=torch.bfloat16))
    assert (C.launch_count() > n0) == kernel
    counts = torch.bincount(ids, minlength=vocab)
    # PyTorch sums in fp32 too; whole numbers up to 256 are exact in bf16
    assert counts.max() <= 256 and torch.equal(module.weight.grad, counts.to(torch.bfloat16)[:, None].expand(-1, cols))
