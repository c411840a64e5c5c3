"""The quantizer's K splits over clusters of 3 to 16 CTAs, ragged row counts included, against the oracle: codes, scales, LoRA sums
and (bf16) the words that tell which 32-row blocks of lora_act fit fp16."""
import pytest
import torch

from test_quantize_gpu import FUSED, _check, _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,slabs,R", [(256, 5, 16), (256, 6, 136), (200, 7, 128), (256, 10, 40), (130, 12, 32), (256, 14, 64), (256, 16, 256), (77, 33, 128),
                                       (640, 20, 96), (900, 17, 128), (1003, 12, 64), (1500, 11, 8), (2048, 9, 128), (256, 1, 128), (1, 3, 16)])
def test_cluster_splits_match_oracle(M, slabs, R, dtype):
    x, ld, sm = _inputs(M, 64 * slabs, R, dtype, M + slabs)
    if dtype == torch.bfloat16:
        x[M // 2:M // 2 + 3] *= 1e7                          # a block or two whose LoRA sums are beyond fp16
    _check(x, ld, sm, FUSED)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,slabs,R", [(256, 160, 256), (700, 100, 136), (1500, 44, 200), (300, 240, 128), (1003, 75, 64)])
def test_cluster_splits_over_many_ring_revolutions(M, slabs, R, dtype):
    """Every rank's share of K goes round both rings several times, at ranks of all three widths and with receive buffers
    whose shares do and do not divide evenly."""
    x, ld, sm = _inputs(M, 64 * slabs, R, dtype, M + slabs)
    _check(x, ld, sm, FUSED)


def test_cluster_split_is_deterministic():
    from svdquant_kernels_b200 import ops
    x, ld, sm = _inputs(256, 3840, 128, torch.float16, 3)
    first = ops.quantize_w4a4_act_fuse_lora(x, ld, sm)[2].clone()
    for _ in range(10):
        assert torch.equal(first, ops.quantize_w4a4_act_fuse_lora(x, ld, sm)[2])
