"""The native host path of the operators (csrc/host_ops.cpp) against the checked Python bodies it stands in for: the same
outputs where it takes a call, the same errors where it does not."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(dtype, M=300, K=512, N=384, R=32):
    from svdquant_kernels_b200 import ops
    g = torch.Generator().manual_seed(6)
    x = torch.randn(M, K, generator=g).to(dtype).cuda()
    sm = (torch.rand(K, generator=g) + 0.5).to(dtype).cuda()
    ld = (torch.randn(K, R, generator=g) / K ** 0.5).to(dtype).cuda()
    lu = (torch.randn(N, R, generator=g) * 0.01).to(dtype).cuda()
    wc = (torch.rand(N, generator=g) + 0.5).to(dtype).cuda()
    wgt, wsc = ops.quantize_nvfp4_rows((torch.randn(N, K, generator=g) * 0.02).cuda())
    return x, sm, ld, lu, wc, wgt, wsc


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_native_calls_equal_the_checked_ones(dtype):
    from svdquant_kernels_b200 import _lib, ops
    x, sm, ld, lu, wc, wgt, wsc = _layer(dtype)
    host = _lib.host()
    q0 = ops._quantize_checked(x, ld, sm)                      # makes the smooth table
    y0 = ops._gemm_checked(q0[0], wgt, q0[1], wsc, q0[2], lu, wc, None, dtype, smooth_next=wc)
    q1 = host.quantize(x, ld, sm, 256, None)
    y1 = host.gemm(q1[0], wgt, q1[1], wsc, q1[2], lu, wc, None, dtype, wc, None)
    assert q1 is not None and y1 is not None
    q2 = host.quantize(x, ld, sm, 256, q1)                     # into the tensors of the last call
    assert q2 is q1
    into = torch.empty_like(y0[0])
    y2 = host.gemm(q2[0], wgt, q2[1], wsc, q2[2], lu, wc, None, dtype, None, into)
    assert y2 is into
    torch.cuda.synchronize()
    for a, b in zip((*q0, *y0, y0[0]), (*q1, *y1, y2)):
        assert a.dtype == b.dtype and torch.equal(a.view(torch.uint8), b.view(torch.uint8))


def test_other_calls_are_left_to_the_checked_body():
    from svdquant_kernels_b200 import _lib, ops
    x, sm, ld, lu, wc, wgt, wsc = _layer(torch.float16)
    host = _lib.host()
    assert host.quantize(x, ld, sm, 256, None) is None         # no smooth table yet
    act, asc, la = ops.quantize_w4a4_act_fuse_lora(x, ld, sm)
    assert host.quantize(x, ld, sm, 256, None) is not None
    sm.mul_(1.0)                                               # edited in place: the table is out of date
    assert host.quantize(x, ld, sm, 256, None) is None
    strided = x.repeat(1, 2)[:, :512]
    assert host.quantize(strided, ld, None, 256, None) is None
    assert torch.equal(ops.quantize_w4a4_act_fuse_lora(strided, ld, sm)[0], act)
    asc.view(torch.uint8).add_(0)                              # so is the twin of the scales
    assert host.gemm(act, wgt, asc, wsc, la, lu, wc, None, torch.float16, None, None) is None
    with pytest.raises(AssertionError):
        ops.gemm_w4a4(act, wgt[:, :-32], asc, wsc, la, lu)
    with pytest.raises(AssertionError):
        torch.ops.svdq_b200.quantize_w4a4_act_fuse_lora(x, ld.float(), sm)


def test_registered_ops_have_no_backward():
    from svdquant_kernels_b200 import torch_ops  # noqa: F401
    x, sm, ld, lu, wc, wgt, wsc = _layer(torch.float16)
    act, asc, la = torch.ops.svdq_b200.quantize_w4a4_act_fuse_lora(x.requires_grad_(), ld, sm)
    assert la.requires_grad and not act.requires_grad
    with pytest.raises(RuntimeError):
        la.sum().backward()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,K", [(64, 128), (300, 512), (4352, 512)])
def test_outputs_have_storages_of_their_own(M, K, dtype):
    """None of a call's outputs shares memory with another or holds more than its own bytes: what is saved, shared or
    kept of one does not bring the others along, and dropping the others gives their memory back."""
    from svdquant_kernels_b200 import ops, torch_ops  # noqa: F401
    x, sm, ld, *_ = _layer(dtype, M=M, K=K)
    for call in (ops.quantize_w4a4_act_fuse_lora, torch.ops.svdq_b200.quantize_w4a4_act_fuse_lora):
        call(x, ld, sm)                                        # makes the smooth table
        held = lambda: torch.cuda.memory_stats()["requested_bytes.all.current"]
        before = held()
        out = call(x, ld, sm)
        stores = [t.untyped_storage() for t in out]
        assert len({s.data_ptr() for s in stores}) == 3
        assert [s.nbytes() for s in stores] == [t.numel() * t.element_size() for t in out]
        act = out[0]
        del out, stores
        assert held() - before == act.numel()                  # the twins went with their owners
        del act


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,K", [(64, 128), (300, 512)])
def test_a_kept_output_keeps_its_own_twin_only(M, K, dtype):
    """An output that outlives the others of its call holds its own bytes and those of its own twin: the scales do not keep
    the planes of lora_act, nor lora_act the scales' second form, nor the codes either."""
    from svdquant_kernels_b200 import ops, torch_ops  # noqa: F401
    x, sm, ld, *_ = _layer(dtype, M=M, K=K)
    nbytes = lambda t: 0 if t is None else t.numel() * t.element_size()
    held = lambda: torch.cuda.memory_stats()["requested_bytes.all.current"]
    for call in (ops.quantize_w4a4_act_fuse_lora, torch.ops.svdq_b200.quantize_w4a4_act_fuse_lora):
        call(x, ld, sm)                                        # makes the smooth table
        for kept in range(3):
            before = held()
            out = call(x, ld, sm)[kept]
            twin = ops._attached(out)
            assert (twin is None) == (kept == 0)
            assert held() - before == nbytes(out) + nbytes(twin), kept
            del out, twin


def test_out_tensors_that_change_type_keep_their_twins_right():
    """The outputs' own types do not depend on the input's, so a call may write into those of a call of the other type:
    the 16-bit form of lora_act that the GEMM reads is then the last call's, in either order."""
    from svdquant_kernels_b200 import ops
    g = torch.Generator().manual_seed(9)
    M, K, N, R = 256, 512, 256, 32
    wgt, wsc = ops.quantize_nvfp4_rows((torch.randn(N, K, generator=g) * 0.02).cuda())
    x, ld, lu = (torch.randn(M, K, generator=g), torch.randn(K, R, generator=g) / K ** 0.5, torch.randn(N, R, generator=g) * 0.01)
    at = {t: (x.to(t).cuda(), ld.to(t).cuda(), lu.to(t).cuda()) for t in (torch.float16, torch.bfloat16)}
    out = ops.quantize_w4a4_act_fuse_lora(*at[torch.float16][:2], None)
    for i, t in enumerate((torch.bfloat16, torch.float16, torch.bfloat16)):
        xt, ldt, lut = at[t]
        xt = xt * (i + 1)
        want = ops.quantize_w4a4_act_fuse_lora(xt, ldt, None)
        got = ops.quantize_w4a4_act_fuse_lora(xt, ldt, None, out=out)
        for u in (torch.float16, torch.bfloat16):
            y0, y1 = (ops.gemm_w4a4(q[0], wgt, q[1], wsc, q[2], at[u][2], None, None, u) for q in (want, got))
            assert torch.equal(y0, y1), (i, t, u)


def test_views_of_one_buffer_are_known_side_by_side():
    """Smoothing factors (or weights) kept as views of one flat buffer: the native table has an entry for each.  With the
    records on the buffer's storage object taken away it is the table alone that answers."""
    from svdquant_kernels_b200 import _lib, ops
    x, _, ld, *_ = _layer(torch.float16)
    host = _lib.host()
    flat = torch.rand(4 * 512, generator=torch.Generator().manual_seed(3)).add_(0.5).half().cuda()
    views = flat.chunk(4)
    want = [ops.quantize_w4a4_act_fuse_lora(x, ld, v.clone()) for v in views]
    for v in views:
        ops.quantize_w4a4_act_fuse_lora(x, ld, v)              # makes the record
        assert host.quantize(x, ld, v, 256, None) is not None  # finds it
    twins = [ops._attached(v) for v in views]
    del flat.untyped_storage()._svdq_twins
    for v, w in zip(views, want):
        got = host.quantize(x, ld, v, 256, None)
        assert got is not None
        assert all(torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(got, w))
    flat.mul_(1.0)                                             # a new version: no entry is good any more
    assert all(host.quantize(x, ld, v, 256, None) is None for v in views)
    del twins


def test_replaced_weights_are_told_apart():
    """More short-lived owners than the native table sweeps at a time, most of them at an address an earlier one had:
    every call uses the factors it is given."""
    from svdquant_kernels_b200 import _lib, ops
    g = torch.Generator().manual_seed(8)
    x, ld = torch.randn(64, 128, generator=g).half().cuda(), torch.randn(128, 16, generator=g).half().cuda()
    kept, seen = [], set()
    for i in range(600):
        sm = (torch.rand(128, generator=g) + 0.5).half().cuda()
        seen.add(sm.data_ptr())
        want = ops.quantize_w4a4_act_fuse_lora(x, ld, sm, _force=_lib.QUANT_FORCE_GENERIC)
        for _ in range(2):                                     # with the table made by this call, and with a known one
            got = ops.quantize_w4a4_act_fuse_lora(x, ld, sm)
            assert torch.equal(got[0], want[0]) and torch.equal(got[1].view(torch.uint8), want[1].view(torch.uint8)), i
        if i % 3 == 0:
            kept.append((sm, want[0]))
    assert len(seen) < 600
    for sm, want in kept:
        assert torch.equal(ops.quantize_w4a4_act_fuse_lora(x, ld, sm)[0], want)
