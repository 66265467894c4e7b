"""One launch over many tensors gives the bits of a launch per tensor."""

import warnings

import pytest
import torch

from offload_adam_b200 import Adam, _ext
from offload_adam_b200.adam import STATE_DTYPES
from offload_adam_b200.ops.adam_step import _EXTRA_KEY, adam_step, adam_step_many
from offload_adam_b200.ops.oracle import MODE_IDS
from offload_adam_b200.qweight import NF4QWeight

pytestmark = pytest.mark.gpu

# around a vector (16), a CTA's chunk (4096 with this much work), and one element
SIZES = [1, 15, 16, 17, 4095, 4096, 4097, 100003]


def _items(mode, sizes, shift):
    gen = torch.Generator(device="cuda").manual_seed(len(sizes))
    items = []
    for i, n in enumerate(sizes):
        def t(dtype, scale=1.0):
            x = torch.randn(n + shift, device="cuda", generator=gen) * scale
            return (x * 100).to(dtype)[shift:] if dtype == torch.int16 else x.to(dtype)[shift:]
        st = {k: t(d, 1e-3) for k, d in STATE_DTYPES[mode].items()}
        st["exp_avg_sq"] = st["exp_avg_sq"].abs()
        st["grad"] = t(torch.bfloat16, 1e-2)
        no_image = mode == "fp32_master" and i % 3 == 2
        items.append((None if no_image else t(torch.bfloat16), st, 1000 + i))
    return items


@pytest.mark.parametrize("mode", list(STATE_DTYPES))
@pytest.mark.parametrize("decoupled", [True, False])
@pytest.mark.parametrize("sizes,shift", [(SIZES, 0), (SIZES, 1), ([33] * 250 + [70000], 0), ([30_000_001, 5], 0)])
def test_many_tensors_bit_for_bit(mode, decoupled, sizes, shift):
    one, many = _items(mode, sizes, shift), _items(mode, sizes, shift)
    hp = (1e-2, 0.1, 0.9, 0.99, 1e-8, 3)
    for p, st, seed in one:
        adam_step(mode, p, st, *hp, decoupled_weight_decay=decoupled, seed=seed)
    C = _ext.load(required=True)
    n0 = C.launch_count()
    adam_step_many(mode, many, *hp, decoupled_weight_decay=decoupled)
    assert C.launch_count() - n0 == -(-len(sizes) // 120)
    key = _EXTRA_KEY[MODE_IDS[mode]]
    for (p, a, _), (q, b, _) in zip(one, many):
        assert p is None or torch.equal(p, q)
        for k in ("exp_avg", "exp_avg_sq") + ((key,) if key else ()):
            assert torch.equal(a[k], b[k])


def test_optimizer_with_uneven_step_counts():
    """Parameters that joined later have another step count: their own launch, same result
    as an optimizer each."""
    def make():
        torch.manual_seed(0)
        return [torch.nn.Parameter(torch.randn(n, device="cuda").to(torch.bfloat16)) for n in (64, 1000, 17)]

    together, alone = make(), make()
    opt = Adam(together, lr=1e-2, mode="fp31_master")
    opts = [Adam([p], lr=1e-2, mode="fp31_master") for p in alone]
    for it in range(3):
        for i, (p, q) in enumerate(zip(together, alone)):
            if i == 1 and it == 0:
                continue  # no gradient in the first step
            p.grad = torch.full_like(p, 0.01 * (i + 1) * (it + 1))
            q.grad = p.grad.clone()
        opt.step()
        for o in opts:
            o.step()
    assert [opt.state[p]["step"] for p in together] == [3, 2, 3]
    for p, q in zip(together, alone):
        assert torch.equal(p, q)


@pytest.mark.parametrize("mode", list(STATE_DTYPES))
@pytest.mark.parametrize("shared", ["parameter", "state", "gradient"])
def test_tensors_that_share_memory_are_stepped_in_order(mode, shared):
    """A launch over both would update the same elements twice at once."""
    def make():
        a, b, c = _items(mode, [300_000, 200_000, 100_000], 0)
        if shared == "parameter":
            b = (a[0][100_000:], *b[1:]) if b[0] is not None else b
        elif shared == "state":
            b[1]["exp_avg"] = a[1]["exp_avg"][:200_000]
        else:  # written by a, read by b
            b[1]["grad"] = a[0][50_000:250_000]
        return [a, b, c]

    one, many = make(), make()
    hp = (1e-2, 0.1, 0.9, 0.99, 1e-8, 3)
    for p, st, seed in one:
        adam_step(mode, p, st, *hp, seed=seed)
    C = _ext.load(required=True)
    n0 = C.launch_count()
    adam_step_many(mode, many, *hp)
    assert C.launch_count() - n0 == 3
    for (p, a, _), (q, b, _) in zip(one, many):
        assert p is None or torch.equal(p, q)
        for k in a:
            assert torch.equal(a[k], b[k])


def _params(*sizes):
    return [torch.nn.Parameter(torch.ones(n, device="cuda", dtype=torch.bfloat16)) for n in sizes]


def test_an_error_stops_at_its_parameter():
    """Those before it are stepped, those after it keep their step count."""
    a, b, c = [torch.nn.Parameter(torch.ones(8, 4, device="cuda", dtype=torch.bfloat16)) for _ in range(3)]
    opt = Adam([a, b, c], lr=1e-2, mode="fp32_master")
    for p in (a, b, c):
        p.grad = torch.ones_like(p)
    opt.step()
    before = a.clone(), b.clone(), c.clone()
    b.grad = torch.ones(4, 8, device="cuda", dtype=torch.bfloat16).t()
    with pytest.raises(RuntimeError, match="contiguous"):
        opt.step()
    assert [opt.state[p]["step"] for p in (a, b, c)] == [2, 2, 1]
    assert (a < before[0]).all() and torch.equal(b, before[1]) and torch.equal(c, before[2])


def test_an_empty_parameter_is_refused_as_in_a_launch_of_its_own():
    ps = _params(17, 0, 5)
    opt = Adam(ps, lr=1e-2, mode="fp31_master")
    for p in ps:
        p.grad = torch.ones_like(p)
        opt._init_state_if_empty(p, opt.state[p])
    with pytest.raises(RuntimeError, match="needs a gradient"):
        opt.step()
    assert (ps[0] < 1).all() and (ps[2] == 1).all() and [opt.state[p]["step"] for p in ps] == [1, 1, 0]


def test_new_state_steps_at_once():
    """What is allocated for a later parameter may fail; and the GPU need not wait for it."""
    ps = _params(100, 200, 300)
    opt = Adam(ps, lr=1e-2, mode="fp32_master")
    init = opt._init_state_if_empty

    def out_of_memory(p, state):
        if p is ps[2]:
            raise torch.cuda.OutOfMemoryError("planted")
        init(p, state)

    opt._init_state_if_empty = out_of_memory
    for p in ps:
        p.grad = torch.ones_like(p)
    with pytest.raises(torch.cuda.OutOfMemoryError):
        opt.step()
    assert (ps[0] < 1).all() and (ps[1] < 1).all() and [opt.state[p]["step"] for p in ps[:2]] == [1, 1]
    opt._init_state_if_empty = init
    n0 = _ext.load(required=True).launch_count()
    opt.step()
    assert [opt.state[p]["step"] for p in ps] == [2, 2, 1]
    assert _ext.load(required=True).launch_count() - n0 == 2  # the two that have state, and the third


def test_one_copy_of_a_gradient_in_another_dtype_at_a_time():
    ws = [torch.nn.Parameter(NF4QWeight.from_float(torch.randn(512, 1024, device="cuda"))) for _ in range(6)]
    opt = Adam(ws, lr=1e-2, mode="fp32_master")
    opt._quant_master_warned = True
    for turn in range(2):
        for w in ws:
            w.grad = torch.randn(512, 1024, device="cuda")
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        opt.step()
    assert torch.cuda.max_memory_allocated() - before <= 1.5 * 2 * 512 * 1024
    assert all(w.grad is None for w in ws)


def test_a_parameter_listed_twice_is_stepped_twice():
    p, q = _params(1000, 1000)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        twice = Adam([{"params": [p, p]}], lr=1e-2, mode="fp31_master")
    once = Adam([q], lr=1e-2, mode="fp31_master")
    for _ in range(2):
        p.grad, q.grad = torch.ones_like(p), torch.ones_like(q)
        twice.step()
        once.step()
        once.step()
    assert twice.state[p]["step"] == 4 and torch.equal(p, q)
