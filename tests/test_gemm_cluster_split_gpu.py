"""Split-K within clusters: the S pairs of a cluster share a tile's K loop.  Forced for every S on shapes with short and ragged last
slabs, against the oracle; chosen by the library on long-K shapes; deterministic."""
import pytest
import torch

from helpers import assert_device_clean, oracle_gemm, rel_l2_vs_bits, u8

pytestmark = pytest.mark.gpu


def _run(M, K, N, R, dtype, variant, wc=True, bias=True, repeat=2):
    from svdquant_kernels_b200 import _lib, ops
    g = torch.Generator().manual_seed(M + K + N)
    x = torch.randn(M, K, generator=g).to(dtype).cuda()
    ld = (torch.randn(K, R, generator=g) / K ** 0.5).to(dtype).cuda()
    lu = (torch.randn(N, R, generator=g) * 0.01).to(dtype)
    c = (torch.rand(N, generator=g) + 0.5).to(dtype) if wc else None
    b = (torch.randn(N, generator=g) * 0.01).to(dtype) if bias else None
    act, asc, la = ops.quantize_w4a4_act_fuse_lora(x, ld, None)
    wgt, wsc = ops.quantize_nvfp4_rows((torch.randn(N, K, generator=g) * 0.02).cuda())
    lud, cd, bd = lu.cuda(), None if c is None else c.cuda(), None if b is None else b.cuda()
    p = ops._ptr
    lu16 = ops._lora_up_f16(lud) if dtype == torch.bfloat16 and R else None
    ys = []
    for _ in range(repeat):
        y = torch.full((M, N), float("nan"), dtype=dtype, device="cuda")
        rc = _lib.load().svdq_gemm_w4a4(p(act), p(wgt), p(ops.swizzle_scales(asc)), p(ops.swizzle_scales(wsc)), p(ops._attached(la)) if R else None,
                                        p(lud) if R else None, p(lu16), p(cd), p(bd), p(y), M, N, K, R, ops._DT[dtype], variant, ops._stream(x.device))
        assert rc == 0, rc
        ys.append(y)
    torch.cuda.synchronize()
    assert_device_clean()
    assert all(torch.equal(ys[0], y) for y in ys)
    y_bits, _ = oracle_gemm(u8(act), u8(wgt), u8(asc), u8(wsc), la.cpu().numpy() if R else None, lu if R else None, c, b, dtype)
    assert rel_l2_vs_bits(ys[0], y_bits) <= 1e-3


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("S,M,K,N,R", [(2, 256, 512, 128, 0), (3, 512, 832, 256, 16), (4, 256, 1088, 384, 128), (5, 256, 1280, 128, 80), (6, 256, 1600, 256, 32),
                                       (7, 256, 1792, 128, 0), (8, 256, 2048, 256, 256)])
def test_forced_cluster_splits_match_oracle(S, M, K, N, R, dtype):
    _run(M, K, N, R, dtype, 10000 * S + 2128)
    _run(M, K, N, R, dtype, 10000 * S + 2128, wc=False, bias=S % 2 == 0, repeat=1)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,K,N,R", [(256, 10240, 1280, 48), (768, 6592, 512, 128), (256, 5824, 384, 16)])
def test_chosen_cluster_splits(M, K, N, R, dtype):
    _run(M, K, N, R, dtype, 0)


def test_what_does_not_fit_is_refused():
    from svdquant_kernels_b200 import _lib
    lib = _lib.load()
    buf = torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")
    p = buf.data_ptr()
    for S, M, K in ((9, 256, 2560), (1, 256, 2560), (4, 256, 512), (2, 384, 2560)):
        assert lib.svdq_gemm_w4a4(p, p, p, p, None, None, None, None, None, p, M, 128, K, 0, 0, 10000 * S + 2128, None) == 7
