"""Layers of the model under the tracers of PyTorch (CPU)."""

import copy
import warnings

import pytest
import torch

from offload_adam_b200.models.llama import build_llama, tiny_llama

MODULES = ["input_layernorm", "self_attn", "mlp", ""]


def _module(name):
    model = build_llama(tiny_llama(), device="cpu", dtype=torch.float32, seed=1)
    layer = model.model.layers[0]
    x = torch.randn(2, 5, 256, generator=torch.Generator().manual_seed(0))
    cos, sin = model._rope_for(5, x.device, x.dtype)
    return getattr(layer, name) if name else layer, (x, cos, sin) if name in ("self_attn", "") else (x,)


@pytest.mark.parametrize("name", MODULES)
def test_symbolic_trace(name):
    module, args = _module(name)
    assert torch.allclose(torch.fx.symbolic_trace(copy.deepcopy(module))(*args), module(*args), atol=1e-6)


@pytest.mark.parametrize("name", MODULES)
def test_script(name):
    module, args = _module(name)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")  # torch.jit.script is deprecated
        scripted = torch.jit.script(module)
    assert torch.allclose(scripted(*args), module(*args), atol=1e-6)
