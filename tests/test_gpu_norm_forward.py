"""The norm's forward with one vector a thread and with up to four, a branch to add or none: against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one vector a thread up to 4096 columns; beyond, two to four of them and a remainder
@pytest.mark.parametrize("n,c", [(1, 4), (3, 256), (700, 4096), (301, 4100), (5, 5504), (300, 8192), (7, 12284), (300, 16384)])
@pytest.mark.parametrize("a_given", [True, False])
def test_norm_forward_matches_fp64(n, c, a_given):
    from tagseq2tagseq_b200 import _lib
    dev, L = torch.device("cuda"), _lib.lib()
    g = torch.Generator(device=dev).manual_seed(n + c)
    x, a = torch.randn(n, c, device=dev, generator=g), torch.randn(n, c, device=dev, generator=g).bfloat16()
    w = torch.rand(c, device=dev, generator=g) + 0.5
    out, h, rstd = torch.full((n + 1, c), 7.0, device=dev), torch.full((n + 1, c), 7.0, device=dev, dtype=torch.bfloat16), torch.full((n + 1,), 7.0, device=dev)
    _lib.check(L.ts2ts_add_rmsnorm_fwd(x.data_ptr(), a.data_ptr() if a_given else None, w.data_ptr(), out.data_ptr(), h.data_ptr(), rstd.data_ptr(), n, c, 1e-6,
                                       torch.cuda.current_stream().cuda_stream), "norm")
    want = x + a if a_given else x                                    # one fp32 addition each
    r = torch.rsqrt(want.double().square().mean(-1) + 1e-6)
    assert torch.equal(out[:n], want)
    # the mean of squares: a rounding of each square, at most 16 additions in a thread and ten in the trees, all of one sign; the quotient, the sum with eps and the root
    assert ((rstd[:n].double() - r).abs() <= 2.0 ** -24 * (27 / 2 + 4) * r).all()
    full = want.double() * r[:, None] * w.double()
    # half a bf16 step, which is 2^-8 of a value whose eight bits are 10000000, behind rstd's error and two products' roundings
    assert ((h[:n].double() - full).abs() <= (2.0 ** -8 + 2.0 ** -24 * 20) * full.abs() * (1 + 2.0 ** -8)).all()
    assert (out[n] == 7).all() and (h[n] == 7).all() and rstd[n] == 7  # nothing behind the last row
