"""The row packer's 16-bit form against the oracle where a near quotient could go wrong: values on and next to the
rounding bounds of the codes, maxima on and next to those of the scales, zeros of either sign, NaN, infinities."""
import numpy as np
import pytest
import torch

from helpers import u8
from oracle import nvfp4_oracle as O

pytestmark = pytest.mark.gpu


def _check(w):
    from svdquant_kernels_b200 import ops
    packed, scales = ops.quantize_nvfp4_rows(w.cuda(), pad_size=1)
    o_p, o_s = O.quantize_nvfp4_rows(w.float().numpy(), 1)
    assert (u8(scales) == o_s).all() and (u8(packed) == o_p).all()


def _neighbours(v, dtype):
    """v rounded to dtype and the values just below and above it"""
    bits = v.to(dtype).view(torch.int16)
    return torch.stack([(bits + d).view(dtype) for d in (-1, 0, 1)], -1)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_bounds_of_codes(dtype):
    scale = torch.arange(1, 0x7E, dtype=torch.uint8).view(torch.float8_e4m3fn).float()
    bounds = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0])
    v = _neighbours(scale[:, None] * bounds, dtype).reshape(len(scale), 21)
    v = torch.cat([v, v[:, :9]], 1).reshape(-1, 2, 15)
    top = (scale * 6).to(dtype)[:, None, None].expand(-1, 2, 1)
    w = torch.cat([top, v], 2).reshape(-1, 32)
    _check(torch.cat([w, -w]))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_bounds_of_scales(dtype):
    g = torch.Generator().manual_seed(1)
    scale = torch.arange(0, 0x7F, dtype=torch.uint8).view(torch.float8_e4m3fn).float()
    top = _neighbours(torch.cat([(scale[1:] + scale[:-1]) * 3, scale * 6]).clamp_min(1e-4), dtype).reshape(-1, 1)
    _check(torch.cat([top, (torch.rand(len(top), 15, generator=g) * top.float()).to(dtype)], 1))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_special_values(dtype):
    w = torch.zeros(6, 32)
    w[0, ::2] = -0.0
    w[1] = torch.linspace(-1, 1, 32)
    w[1, 7:9] = torch.tensor([-0.0, 0.0])
    w[2] = 1e-7
    w[3, 3] = -1e-7
    w[4] = 60000.0
    w[5, :16] = torch.linspace(-6e-3, 6e-3, 16)
    _check(w.to(dtype))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_non_finite_values(dtype):
    from svdquant_kernels_b200 import ops
    w = torch.ones(3, 32)
    w[0, 3], w[1, 20], w[1, 21], w[2, :16] = float("nan"), float("inf"), float("-inf"), 0.0
    w[2, 5] = float("nan")
    packed, scales = ops.quantize_nvfp4_rows(w.to(dtype).cuda(), pad_size=1)
    codes = np.stack([u8(packed) & 15, u8(packed) >> 4], axis=-1).reshape(3, 32)
    assert codes[0, 3] == 0 and (codes[0, [0, 1, 2, 4]] == 7).all()
    assert u8(scales)[1, 1] == 0x7E and codes[1, 20] == 7 and codes[1, 21] == 15
    assert u8(scales)[0, 2] == 0 and (codes[2, :16] == 0).all()
