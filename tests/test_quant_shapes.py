"""Quantization kernels at the sizes where their launch rules change, bit for bit against
the PyTorch restatements."""

import pytest
import torch

from offload_adam_b200.qweight import Int8QWeight, NVFP4QWeight, fake_quantize
from offload_adam_b200.qweight.int8 import _quantize_int8_cuda, quantize_int8_per_channel
from offload_adam_b200.qweight.nvfp4 import _quantize_nvfp4_cuda, quantize_nvfp4_blockwise

pytestmark = pytest.mark.gpu


def _rand(rows, cols, dtype, shift=0):
    gen = torch.Generator(device="cuda").manual_seed(rows * 131 + cols)
    flat = torch.randn(rows * cols + shift, device="cuda", generator=gen).to(dtype)[shift:]
    return flat.view(rows, cols)  # `shift` elements past a 512-byte boundary


def _bits(t):
    return t.cpu().contiguous().reshape(-1).view(torch.uint8)


# quads of a warp end at 2048 columns, vectors of a CTA at 16384, quads of a CTA at 16384
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("cols", [4, 124, 1100, 2044, 2048, 2052, 4096, 16380, 16384, 16388])
@pytest.mark.parametrize("rows", [1, 7, 9, 300])
@pytest.mark.parametrize("shift", [0, 1, 4])
def test_int8_rows(dtype, cols, rows, shift):
    x = _rand(rows, cols, dtype, shift)
    if rows > 1:
        x[1] = 0
    q, s = _quantize_int8_cuda(x, torch.bfloat16)
    q_ref, s_ref = quantize_int8_per_channel(x.cpu(), scale_dtype=torch.bfloat16)
    assert torch.equal(q.cpu(), q_ref) and torch.equal(s.cpu(), s_ref)
    fake = fake_quantize(x, Int8QWeight)
    assert torch.equal(_bits(fake), _bits(Int8QWeight(q, s).dequantize(dtype)))


# one block; around a warp's 32 blocks; several CTAs; more than one sweep of the grid
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(1, 16), (1, 496), (3, 176), (33, 512), (130, 4112), (2500, 4096)])
def test_nvfp4_two_passes(dtype, rows, cols):
    x = _rand(rows, cols, dtype)
    x[-1, -1] = 40.0  # the maximum is in the last value
    got = _quantize_nvfp4_cuda(x)
    want = quantize_nvfp4_blockwise(x.cpu())
    for a, b in zip(got, want):
        assert torch.equal(_bits(a.reshape(b.shape)), _bits(b))
    q = NVFP4QWeight(*got, cols, dtype)
    assert torch.equal(_bits(fake_quantize(x, NVFP4QWeight)), _bits(q.dequantize(dtype)))


def test_misaligned_source_of_nvfp4_is_refused_before_any_launch():
    """The pass for the tensor's maximum reads 32-byte vectors, as the quantization does."""
    x = torch.randn(64 * 64 + 1, device="cuda")[1:].view(64, 64)
    w = NVFP4QWeight.from_float(torch.randn(64, 64, device="cuda"))
    payload = [t.clone() for t in w._payload()]
    with pytest.raises(RuntimeError, match="invalid argument"):
        w.copy_(x)
    with pytest.raises(RuntimeError, match="invalid argument"):
        fake_quantize(x, NVFP4QWeight)
    torch.cuda.synchronize()
    assert all(torch.equal(_bits(a), _bits(b)) for a, b in zip(payload, w._payload()))


# results around 96 MB, where a thread takes one vector; rows of 16 columns and others
@pytest.mark.parametrize("rows,cols", [(11717, 4096), (11720, 4096), (12000, 4004), (1, 16), (37, 20)])
def test_dequantize_on_every_grid(rows, cols):
    x = _rand(rows, cols, torch.bfloat16)
    q, s = _quantize_int8_cuda(x, torch.bfloat16)
    assert torch.equal(Int8QWeight(q, s).dequantize(torch.bfloat16), (q.float() * s.float().reshape(-1, 1)).to(torch.bfloat16))
    if cols % 16 == 0:
        w = NVFP4QWeight(*_quantize_nvfp4_cuda(x), cols, torch.bfloat16)
        half = rows // 2 + 1  # a slice below the limit against the whole
        part = NVFP4QWeight(w.weight_packed[:half], w.block_scale_fp8[:half], w.global_scale, cols, torch.bfloat16)
        assert torch.equal(w.dequantize()[:half], part.dequantize())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,cols", [(592, 2048), (593, 2048), (592, 16), (593, 16), (2369, 4348), (2369, 4352), (2369, 4356),
                                       (2500, 2052), (2400, 4096)])
def test_int8_rows_around_the_limits_of_a_grid(dtype, rows, cols):
    x = _rand(rows, cols, dtype)
    q, s = _quantize_int8_cuda(x, torch.bfloat16)
    q_ref, s_ref = quantize_int8_per_channel(x.cpu(), scale_dtype=torch.bfloat16)
    assert torch.equal(q.cpu(), q_ref) and torch.equal(s.cpu(), s_ref)
    assert torch.equal(_bits(fake_quantize(x, Int8QWeight)), _bits(Int8QWeight(q, s).dequantize(dtype)))
