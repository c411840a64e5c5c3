"""The row packer at the edges of its 128-row x 4-group tiles, all input types, against the oracle."""
import numpy as np
import pytest
import torch

from helpers import u8
from oracle import nvfp4_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
@pytest.mark.parametrize("rows,K,pad", [(1, 16, 1), (127, 112, 1), (129, 144, 1), (128, 128, 1), (130, 64, 128), (3, 4112, 4), (1000, 192, 256)])
def test_packer_tile_edges(rows, K, pad, dtype):
    from svdquant_kernels_b200 import ops
    g = torch.Generator().manual_seed(rows + K)
    w = torch.randn(rows, K, generator=g) * torch.exp2(torch.randint(-12, 12, (rows, 1), generator=g).float())
    w[0, :3] = torch.tensor([-0.0, 0.0, 1e-30])
    w = w.to(dtype)
    packed, scales = ops.quantize_nvfp4_rows(w.cuda(), pad_size=pad)
    o_p, o_s = O.quantize_nvfp4_rows(w.float().numpy(), pad)
    assert (u8(packed) == o_p).all() and (u8(scales) == o_s).all()
    twin = ops._attached(scales)
    if o_p.shape[0] % 128 == 0 and K % 64 == 0:
        assert (twin.cpu().numpy() == O.swizzle_scales(o_s)).all()
    else:
        assert twin is None


def test_packer_non_finite_values():
    """NaN counts as zero, an infinity saturates its group's scale: as the comparisons of the definition have it."""
    from svdquant_kernels_b200 import ops
    w = torch.ones(2, 32)
    w[0, 3], w[1, 20], w[1, 21] = float("nan"), float("inf"), float("-inf")
    packed, scales = ops.quantize_nvfp4_rows(w.cuda(), pad_size=1)
    codes = np.stack([u8(packed) & 15, u8(packed) >> 4], axis=-1).reshape(2, 32)
    assert codes[0, 3] == 0 and (codes[0, [0, 1, 2, 4]] == 7).all()
    assert u8(scales)[1, 1] == 0x7E and codes[1, 20] == 7 and codes[1, 21] == 15
