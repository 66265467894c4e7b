"""When the model code may call a CUDA kernel in place of PyTorch operations.

The kernels read raw pointers, so nothing that watches or rewrites PyTorch operations sees
them.  They are used for plain bf16 CUDA tensors in ordinary eager execution; everything
else (other dtypes and devices, tensor subclasses, ``torch.func`` transforms, forward-mode
differentiation, tracing, compilation, autocast, dispatch and function modes) runs the
PyTorch operations."""

from __future__ import annotations

import torch
from torch import nn
from torch.autograd import forward_ad

_PLAIN = (torch.Tensor, nn.Parameter)


def eager():
    """True in ordinary eager execution: no transform, mode or tracer is active."""
    if torch.compiler.is_compiling():  # first: a tracer need not look at the rest
        return False
    return (torch._C._functorch.peek_interpreter_stack() is None
            and forward_ad._current_level < 0
            and not torch._C._len_torch_dispatch_stack()
            and not torch._C._len_torch_function_stack()
            and not torch.is_autocast_enabled("cuda")
            and not torch.jit.is_tracing())


def use_kernels(*tensors):
    """True when all of ``tensors`` are plain bf16 CUDA tensors in eager execution."""
    for t in tensors:
        if type(t) not in _PLAIN or not t.is_cuda or t.dtype is not torch.bfloat16:
            return False
    return eager()
