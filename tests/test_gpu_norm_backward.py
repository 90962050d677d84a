"""The norm's gradient where its blocks have no row, one or several, and one vector a thread or four: against fp64, the weight gradient added or written."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,c", [(1, 4), (3, 256), (296, 256), (297, 256), (1193, 768), (593, 2048), (700, 4096), (297, 4100), (5, 16384)])
@pytest.mark.parametrize("up_given,da_given", [(True, True), (False, False)])
def test_norm_backward_matches_fp64(n, c, up_given, da_given):
    from tagseq2tagseq_b200 import _lib
    dev, L = torch.device("cuda"), _lib.lib()
    g = torch.Generator(device=dev).manual_seed(n + c)
    x, up = (torch.randn(n, c, device=dev, generator=g) for _ in range(2))
    dh = torch.randn(n, c, device=dev, generator=g).bfloat16()
    w = torch.rand(c, device=dev, generator=g) + 0.5
    rstd = torch.rsqrt(x.double().square().mean(-1) + 1e-6).float()
    xh, gw = x.double() * rstd.double()[:, None], dh.double() * w.double()
    want = rstd.double()[:, None] * (gw - xh * (gw * xh).mean(-1, keepdim=True)) + (up.double() if up_given else 0.0)
    want_dw = (dh.double() * xh).sum(0)
    size = rstd.double()[:, None] * (gw.abs() + xh.abs() * (gw * xh).abs().mean(-1, keepdim=True)) + up.double().abs()
    ws = torch.empty(L.ts2ts_add_rmsnorm_bwd_workspace_bytes(n, c), dtype=torch.uint8, device=dev)
    for fn, before in ((L.ts2ts_add_rmsnorm_bwd, 3.0), (L.ts2ts_add_rmsnorm_bwd_set, 0.0)):
        dx, dw = torch.empty(n, c, device=dev), torch.full((c,), 3.0, device=dev)
        da = torch.empty(n, c, device=dev, dtype=torch.bfloat16) if da_given else None
        _lib.check(fn(dh.data_ptr(), up.data_ptr() if up_given else None, x.data_ptr(), w.data_ptr(), rstd.data_ptr(), dx.data_ptr(),
                      da.data_ptr() if da_given else None, dw.data_ptr(), ws.data_ptr(), ws.numel(), n, c, torch.cuda.current_stream().cuda_stream), "norm")
        # fp32: a few roundings of each term, the mean's sum over c in a tree of at most 5 + 5 + c / 1024 steps
        assert ((dx.double() - want).abs() <= 2.0 ** -23 * (16 + c / 1024) * size).all()
        if da_given:
            assert torch.equal(da, dx.bfloat16())
        # products of a row each, a block's rows one after the other, the blocks' sums by rows of 128
        assert ((dw.double() - before - want_dw).abs() <= 2.0 ** -23 * (16 + n / 64) * ((dh.double() * xh).abs().sum(0) + before)).all()
