"""One launch over many tensors gives the bits of a launch per tensor."""

import pytest
import torch

from offload_adam_b200 import Adam, _ext
from offload_adam_b200.adam import STATE_DTYPES
from offload_adam_b200.ops.adam_step import _EXTRA_KEY, adam_step, adam_step_many
from offload_adam_b200.ops.oracle import MODE_IDS

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
