"""How a host call moves its rows: kernels for short copies, the copy engine for long or misaligned ones,
chunks for tall calls.  None of it may show in y."""
import pytest
import torch

from helpers import assert_device_clean
from test_plan_gpu import _setup

pytestmark = pytest.mark.gpu


def _pinned(rows, cols, dtype, offset):
    return torch.empty(rows * cols + offset, dtype=dtype).pin_memory()[offset:].view(rows, cols)


@pytest.mark.parametrize("K,N,rows", [
    (128, 128, (1, 3, 256)),
    (4096, 512, (256, 257)),          # x of exactly 2 MB, and one row more in two chunks
    (512, 4096, (255, 256, 700)),     # y of just under 2 MB, of exactly 2 MB, in chunks
    (1536, 1024, (2048, 1900)),
])
@pytest.mark.parametrize("offset", [0, 1])
def test_forward_host_copies(K, N, rows, offset):
    dtype = torch.float16
    plan, device_path, g = _setup(max(rows), K, N, 32, dtype, 3)
    try:
        other_x, other_y = _pinned(2, K, dtype, 0), _pinned(2, N, dtype, 0)
        other_x.copy_(torch.randn(2, K, generator=g))
        for M in rows:
            for x_pinned, y_pinned in ((True, True), (False, True), (True, False)):
                x = _pinned(M, K, dtype, offset) if x_pinned else torch.empty(M, K, dtype=dtype)
                y = _pinned(M, N, dtype, offset) if y_pinned else torch.empty(M, N, dtype=dtype)
                x.copy_(torch.randn(M, K, generator=g))
                y.fill_(7.0)
                plan.submit(other_x, other_y)                # a call of the other slot still in flight
                plan.forward_host(x, y)
                assert torch.equal(y, device_path(x)), (M, x_pinned, y_pinned)
                assert torch.equal(other_y, device_path(other_x))
    finally:
        plan.close()
    assert_device_clean()
