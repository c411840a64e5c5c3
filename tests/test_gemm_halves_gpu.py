"""Last rounds of 256-column tiles that are worked on as halves: at the edges of the rule (one tile left, half of the pairs
left, one more than that), with short K, ragged last slabs and every LoRA form, plain and with the next layer's codes.  The
sums of a half are those of a 128-column tile in the same order, so the bits have to be equal; 128-column tiles are compared
with the oracle, and so are the smallest of these."""
import pytest
import torch

from helpers import assert_device_clean, oracle_gemm, rel_l2_vs_bits, u8

pytestmark = pytest.mark.gpu


def _layer(M, K, N, R, dtype, wc, bias):
    from svdquant_kernels_b200 import ops
    g = torch.Generator().manual_seed(M + K + N + R)
    x = torch.randn(M, K, generator=g).to(dtype)
    if dtype == torch.bfloat16 and R:
        x[:3] *= 1e7                                     # a tile whose lora_act does not fit fp16: two LoRA passes
    ld = (torch.randn(K, R, generator=g) / K ** 0.5).to(dtype)
    lu = (torch.randn(N, R, generator=g) * 0.01).to(dtype)
    c = (torch.rand(N, generator=g) + 0.5).to(dtype) if wc else None
    b = (torch.randn(N, generator=g) * 0.01).to(dtype) if bias else None
    act, asc, la = ops.quantize_w4a4_act_fuse_lora(x.cuda(), ld.cuda(), None)
    wgt, wsc = ops.quantize_nvfp4_rows((torch.randn(N, K, generator=g) * 0.02).cuda())
    host = (u8(act), u8(wgt), u8(asc), u8(wsc), la.cpu().numpy() if R else None, lu if R else None, c, b, dtype)
    dev = (act, wgt, asc, wsc, la if R else None, lu.cuda() if R else None, None if c is None else c.cuda(), None if b is None else b.cuda(), dtype)
    return dev, host


# pairs of 148 SMs: 74; tiles 75, 76, 111 = 74 + 37, 112 = 74 + 38 (not halved), 148 + 37
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("mt,nt,K,R", [(5, 15, 64, 0), (4, 19, 320, 48), (3, 37, 576, 128), (7, 16, 256, 16), (5, 37, 512, 256)])
def test_halved_rounds_equal_narrow_tiles(mt, nt, K, R, dtype):
    from svdquant_kernels_b200 import ops
    M, N = 256 * mt, 256 * nt
    args, host = _layer(M, K, N, R, dtype, wc=R != 48, bias=R != 16)
    want = ops.gemm_w4a4(*args, tiler_mn=(256, 128))
    got = ops.gemm_w4a4(*args, tiler_mn=(256, 256))
    assert torch.equal(got, want)
    sn = (torch.rand(N, generator=torch.Generator().manual_seed(1)) + 0.5).to(dtype).cuda()
    for a, b in zip(ops.gemm_w4a4(*args, tiler_mn=(256, 256), smooth_next=sn), ops.gemm_w4a4(*args, tiler_mn=(256, 128), smooth_next=sn)):
        assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    assert torch.equal(ops.gemm_w4a4(*args, tiler_mn=(256, 256), lora_schedule="interleaved"),
                       ops.gemm_w4a4(*args, tiler_mn=(256, 128), lora_schedule="interleaved"))
    assert_device_clean()
    if mt * nt <= 76:
        assert rel_l2_vs_bits(got, oracle_gemm(*host)[0]) <= 1e-3
