"""The fp16 copy of a bf16 lora_up made on the device: every bf16 value against the host's conversion, sizes around the eight
values of a thread, a source that is not 16-byte aligned, and values that fp16 does not hold."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _host(t):
    from svdquant_kernels_b200 import _lib
    src = t.contiguous().view(torch.int16).numpy()
    out = np.zeros(src.shape, dtype=np.float16)
    return _lib.load().svdq_lora_up_to_f16(src.ctypes.data, out.ctypes.data, src.size), out


def test_every_value_that_fits_converts_as_on_the_host():
    from svdquant_kernels_b200 import ops
    every = torch.arange(1 << 16, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    fits = every[every.float().abs() <= 65504].clone()            # subnormals and both zeros among them, no NaN
    rc, want = _host(fits)
    assert rc == 0
    got = ops._lora_up_f16(fits.cuda()).cpu().numpy()
    assert np.array_equal(got.view(np.uint16), want.view(np.uint16))


@pytest.mark.parametrize("n,skip", [(1, 0), (7, 0), (8, 0), (9, 0), (4099, 0), (16, 1), (30001, 3)])
def test_sizes_and_alignments(n, skip):
    from svdquant_kernels_b200 import ops
    flat = torch.randn(n + skip, generator=torch.Generator().manual_seed(n)).to(torch.bfloat16).cuda()
    src = flat[skip:].view(1, n)
    assert np.array_equal(ops._lora_up_f16(src).cpu().numpy(), src.cpu().float().numpy().astype(np.float16))


@pytest.mark.parametrize("bad", [65536.0, -131072.0, float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("at", [0, 4095, 70000, 99999])
def test_values_that_do_not_fit_leave_no_copy(bad, at):
    from svdquant_kernels_b200 import ops
    src = torch.zeros(100000, dtype=torch.bfloat16)
    src[at] = bad
    assert _host(src)[0] != 0
    assert ops._lora_up_f16(src.cuda()) is None
