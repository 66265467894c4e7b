"""Cross-entropy kernels against the same loss in fp64 PyTorch."""

import math

import pytest
import torch

from offload_adam_b200 import _ext
from offload_adam_b200.models import llama
from offload_adam_b200.models.llama import chunked_linear_cross_entropy

pytestmark = pytest.mark.gpu


def _inputs(n, hidden, vocab, ignored=0.2, scale=1.0, seed=0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    h = torch.randn(n, hidden, device="cuda", generator=gen).to(torch.bfloat16)
    w = (torch.randn(vocab, hidden, device="cuda", generator=gen) * scale / math.sqrt(hidden)).to(torch.bfloat16)
    labels = torch.randint(0, vocab, (n,), device="cuda", generator=gen)
    labels[torch.rand(n, device="cuda", generator=gen) < ignored] = -100
    return h, w, labels


def _run(fn, h, w, labels, chunk, g=1.0):
    h, w = h.clone().requires_grad_(True), w.clone().requires_grad_(True)
    loss = fn(h, w, labels, chunk)
    (loss * g).backward()
    return loss.detach().double(), h.grad.double(), w.grad.double()


def _fp64(h, w, labels, g=1.0):
    h, w = h.double().requires_grad_(True), w.double().requires_grad_(True)
    loss = torch.nn.functional.cross_entropy(h @ w.T, labels, ignore_index=-100, reduction="sum")
    loss = loss / max(1, int((labels != -100).sum()))
    (loss * g).backward()
    return loss.detach(), h.grad, w.grad


def _rel(a, b):
    return ((a - b).norm() / b.norm().clamp_min(1e-30)).item()


# vocabularies around a 16-value vector, a pair of vectors per thread and the CTA sizes;
# rows in one group, in several and a ragged last one
@pytest.mark.parametrize("vocab", [1, 15, 16, 17, 1000, 4095, 8192, 8193, 32003, 128256])
@pytest.mark.parametrize("n,chunk", [(1, 128), (37, 128), (300, 50), (300, 15)])
def test_linear_cross_entropy_matches_fp64(vocab, n, chunk):
    h, w, labels = _inputs(n, 64, vocab)
    got = _run(chunked_linear_cross_entropy, h, w, labels, chunk, g=0.25)
    want = _fp64(h, w, labels, g=0.25)
    old = _run(llama._ChunkedLinearCE.apply, h, w, labels, chunk, g=0.25)
    # bf16 logits round by up to 2^-8 of their value, a few units here
    assert abs(got[0] - want[0]) <= 2.0 ** -8 * max(1.0, abs(want[0].item()))
    for k in (1, 2):
        if want[k].norm() == 0:  # one class, or no label: every gradient is zero
            assert got[k].abs().max() <= 2.0 ** -8
            continue
        # logits, their gradient and the result each round to bf16, by up to 2^-8; and not
        # worse than the PyTorch route
        assert _rel(got[k], want[k]) <= 3 * 2.0 ** -8
        assert _rel(got[k], want[k]) <= 1.1 * _rel(old[k], want[k]) + 1e-4


# products large enough for the library to split: few tiles, long sums, vocabularies of every
# alignment; one group of rows, two, and several
@pytest.mark.parametrize("vocab,hidden,n,chunk", [(1001, 2048, 4096, 2048), (1001, 256, 8192, 1024), (32003, 64, 60, 15),
                                                  (32003, 64, 4096, 256), (32003, 840, 3000, 512), (32004, 256, 3000, 512),
                                                  (32000, 256, 3000, 512), (5001, 512, 777, 64), (8192, 1024, 600, 128),
                                                  (1001, 100, 300, 64)])
def test_no_less_precise_and_no_larger_than_the_pytorch_route(vocab, hidden, n, chunk):
    """At the chunk that the caller passes."""
    h, w, labels = _inputs(n, hidden, vocab)
    want = _fp64(h, w, labels)
    got, old, peak = [], [], []
    for fn, out in ((chunked_linear_cross_entropy, got), (llama._ChunkedLinearCE.apply, old)):
        for turn in range(2):  # the library takes its workspace in the first
            a = b = None
            torch.cuda.reset_peak_memory_stats()
            before = torch.cuda.memory_allocated()
            a, b = h.detach().requires_grad_(True), w.detach().requires_grad_(True)
            fn(a, b, labels, chunk).backward()
            peak.append(torch.cuda.max_memory_allocated() - before)
        out += [a.grad.double(), b.grad.double()]
        del a, b
    for k in (0, 1):
        assert _rel(got[k], want[k + 1]) <= 1.1 * _rel(old[k], want[k + 1]) + 1e-4
    # labels' statistics (three floats a row) and 512-byte blocks of the allocator on top
    assert peak[1] <= peak[3] + 16 * n + 16384


@pytest.mark.parametrize("n", [1, 15, 16, 4096, 4113])
def test_sum_of_bf16_tensors(n):
    C = _ext.load(required=True)
    a, b, c = (torch.randn(n, device="cuda").to(torch.bfloat16) for _ in range(3))
    ab = C.sum_bf16(a, b, False)
    assert torch.equal(ab, a.float() + b.float())
    assert torch.equal(C.sum_bf16(a, b, True), (a.float() + b.float()).to(torch.bfloat16))
    assert torch.equal(C.sum_bf16(ab, c, True), (a.float() + b.float() + c.float()).to(torch.bfloat16))
    into = c.clone()
    assert C.sum_bf16(ab, into, True, into) is into
    assert torch.equal(into, (a.float() + b.float() + c.float()).to(torch.bfloat16))
    assert torch.equal(C.sum_bf16(ab, c, False), a.float() + b.float() + c.float())


def test_loss_without_gradient_and_all_ignored():
    h, w, labels = _inputs(64, 64, 1000)
    with torch.no_grad():
        a = chunked_linear_cross_entropy(h, w, labels, 16)   # two groups
        b = chunked_linear_cross_entropy(h, w, labels, 128)  # one group
    assert torch.allclose(a, b, rtol=1e-6) and not a.requires_grad
    labels.fill_(-100)
    loss, gh, gw = _run(chunked_linear_cross_entropy, h, w, labels, 128)
    assert loss == 0 and gh.abs().max() == 0 and gw.abs().max() == 0


def test_non_finite_logits_as_in_pytorch():
    h, w, labels = _inputs(8, 32, 100, ignored=0.0)
    labels.clamp_(min=8)
    h[1].fill_(float("nan"))
    h[2].fill_(float("inf"))
    for row in range(8):
        one = h[row:row + 1], w, labels[row:row + 1], 128
        got, want = _run(chunked_linear_cross_entropy, *one), _run(llama._ChunkedLinearCE.apply, *one)
        for a, b in zip(got, want):
            assert torch.equal(a.isfinite(), b.isfinite())


def test_backward_twice_and_through_the_incoming_gradient():
    h, w, labels = _inputs(32, 64, 1000)
    h.requires_grad_(True)
    scale = torch.tensor(3.0, device="cuda", requires_grad=True)
    loss = chunked_linear_cross_entropy(h, w, labels, 128)
    a, = torch.autograd.grad(loss, h, retain_graph=True)
    b, = torch.autograd.grad(loss, h, retain_graph=True)
    assert torch.equal(a, b)
    c, = torch.autograd.grad(loss * scale, h, create_graph=True)
    c.float().sum().backward()
    assert torch.allclose(scale.grad, a.float().sum(), rtol=2e-2, atol=1e-3)


def test_saved_tensors_may_move():
    h, w, labels = _inputs(33, 64, 1001)
    plain = _run(chunked_linear_cross_entropy, h, w, labels, 128)
    with torch.autograd.graph.save_on_cpu():
        moved = _run(chunked_linear_cross_entropy, h, w, labels, 128)
    for a, b in zip(plain, moved):
        assert torch.equal(a, b)


@pytest.mark.parametrize("n,chunk", [(20, 128), (300, 15)])
def test_label_outside_the_vocabulary_is_refused(n, chunk):
    """It is seen when the kernel has run: this call's loss is NaN, the next call raises."""
    h, w, labels = _inputs(n, 64, 1000)
    good = _run(chunked_linear_cross_entropy, h, w, labels, chunk)
    bad = labels.clone()
    bad[n // 2] = 1000
    with torch.no_grad():
        loss = chunked_linear_cross_entropy(h, w, bad, n)
        assert loss.isnan()  # waits for it
        with pytest.raises(IndexError, match="label 1000 .* outside its vocabulary"):
            chunked_linear_cross_entropy(h, w, labels, chunk)
    for a, b in zip(good, _run(chunked_linear_cross_entropy, h, w, labels, chunk)):
        assert torch.equal(a, b)  # reported once
    a = h.clone().requires_grad_(True)
    loss = chunked_linear_cross_entropy(a, w, bad, n)
    torch.cuda.synchronize()
    with pytest.raises(IndexError, match="label 1000"):
        loss.backward()


def test_probabilities_keep_fp32_precision():
    """Far below the row's maximum, where an approximate exponential is off by more, down to
    what only a subnormal bf16 holds."""
    C = _ext.load(required=True)
    n, V = 512, 16384
    x = C.ce_logits_buffer(torch.empty(0, device="cuda", dtype=torch.bfloat16), n, V)
    gen = torch.Generator(device="cuda").manual_seed(0)
    x.copy_(-40 - 48 * torch.rand(n, V, device="cuda", generator=gen))
    top = torch.rand(n, device="cuda", generator=gen).to(torch.bfloat16)  # the maximum of its row
    x[:, 0] = top
    labels = torch.zeros(n, dtype=torch.int64, device="cuda")
    stats, inv = torch.empty(3 * n, device="cuda"), torch.ones((), device="cuda")
    grad = C.ce_logits_buffer(x, n, V)
    C.ce_stats(x, labels, stats)
    C.ce_grad(x, labels, stats, inv, None, grad)
    d = (x.float() - top.float()[:, None]).double()[:, 1:]  # the difference rounds to fp32 first
    want = d.exp()  # the sum of a row is 1 to within 1e-13
    normal = want > 1.2e-38
    wrong = grad[:, 1:] != want.float().to(torch.bfloat16)
    # a relative error of e changes the rounding of about e / 2^-8 of the values; e is 2^-22 here
    assert wrong[normal].double().mean() <= 3e-4
    tiny = ~normal
    assert tiny.any()
    assert ((grad[:, 1:].double() - want).abs()[tiny] <= 2.0 ** -8 * want[tiny] + 2.0 ** -133).all()
