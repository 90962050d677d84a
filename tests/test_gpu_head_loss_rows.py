"""Loss and gradient of a row of logits in one pass, around the row lengths at which a block's threads and chunks change."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


# 256, 1024, 2048 and 4096 vectors of eight, one more, and the ends of the range
@pytest.mark.parametrize("V", [8, 24, 2048, 2056, 8192, 8200, 16384, 16392, 32768, 32776, 50304, 110592])
def test_loss_and_gradient_of_a_row_match_fp64(V):
    from tagseq2tagseq_b200 import _lib
    dev, n = torch.device("cuda"), 9
    g = torch.Generator(device=dev).manual_seed(V)
    x = (torch.randn(n, V, device=dev, generator=g) * 3).bfloat16()
    target = torch.randint(0, V, (n,), device=dev, generator=g)
    x[1, V // 2:] = float("-inf")                              # classes that are ruled out
    target[1] = 0
    x[2] = float("-inf")
    x[2, V - 1], target[2] = 1.5, V - 1                        # one class left
    x[3] *= 30                                                 # far apart
    x[4, target[4]] = 60.0                                     # as good as certain
    target[5], target[6] = -100, V                             # no loss, no gradient
    y, loss = x.clone(), torch.empty(n, device=dev)
    _lib.check(_lib.lib().ts2ts_ce_fwd_grad(y.data_ptr(), target.data_ptr(), loss.data_ptr(), 0.25, n, V, torch.cuda.current_stream().cuda_stream), "ce")
    live = (target >= 0) & (target < V)
    at = torch.where(live, target, 0)
    want_l = torch.logsumexp(x.double(), -1)
    want = torch.where(live, want_l - x.double().gather(1, at[:, None])[:, 0], 0.0)
    # the row's sum in fp32 and its logarithm: a rounding each of the logits' size, of the log-sum-exp and of 16 additions one after the other
    assert ((loss.double() - want).abs() <= 2.0 ** -23 * (want_l.abs() + 16)).all()
    p = torch.softmax(x.double(), -1)
    hot = torch.nn.functional.one_hot(at, V).bool()
    grad = torch.where(live[:, None], (p - hot.double()) * 0.25, 0.0)
    # half a bf16 step (2^-8 of a value whose eight bits are 10000000), an exponent that is off by fp32's rounding of what it is the difference of, and subnormal results (below 2^-126) that come out as zero
    off = 2.0 ** -8 * grad.abs() + 0.25 * p * 2.0 ** -22 * (x.double().abs().nan_to_num(posinf=0.0) + want_l[:, None].abs() + 2) + 2.0 ** -126
    assert ((y.double() - grad).abs() <= off).all()


FILLS = [torch.finfo(torch.bfloat16).min, -1e30, -1e10]        # what rules a class out, and stays a number


@pytest.mark.parametrize("V", [8, 24, 2048, 2056, 8200, 16392, 32776, 50304])
@pytest.mark.parametrize("fill", FILLS)
def test_ruled_out_classes_of_large_finite_logits(V, fill):
    """A thread may see nothing but ruled-out classes; they get no probability, and the row's other classes share it."""
    from tagseq2tagseq_b200 import _lib
    dev, n = torch.device("cuda"), 5
    g = torch.Generator(device=dev).manual_seed(V)
    x = (torch.randn(n, V, device=dev, generator=g) * 3).bfloat16()
    target = torch.tensor([V - 1, V - 1, V // 2 - 1, V - 1, V - 1], device=dev)
    x[0, :V - 1] = fill                                        # one class left
    x[1, :V // 2] = fill
    x[2, V // 2:] = fill
    x[3, :V - 4] = fill                                        # all vectors but the last
    x[4, :min(8, V - 1)] = fill                                # one vector
    y, loss = x.clone(), torch.empty(n, device=dev)
    _lib.check(_lib.lib().ts2ts_ce_fwd_grad(y.data_ptr(), target.data_ptr(), loss.data_ptr(), 0.25, n, V, torch.cuda.current_stream().cuda_stream), "ce")
    l, p = torch.logsumexp(x.double(), -1), torch.softmax(x.double(), -1)
    assert ((loss.double() - (l - x.double().gather(1, target[:, None])[:, 0])).abs() <= 2.0 ** -23 * (l.abs() + 16)).all()
    grad = (p - torch.nn.functional.one_hot(target, V)) * 0.25
    # as above: half a bf16 step, the exponent's rounding (the ruled out have p = 0 and are to come out as zero), subnormal results
    off = 2.0 ** -8 * grad.abs() + torch.where(p > 0, 0.25 * p * 2.0 ** -22 * (x.double().abs() + l[:, None].abs() + 2), 0.0) + 2.0 ** -126
    assert ((y.double() - grad).abs() <= off).all()


@pytest.mark.parametrize("V", [8, 24, 2048, 2056, 8200, 16392, 32776, 50304])
def test_rows_whose_log_sum_exp_is_large_are_those_of_the_two_kernels(V):
    """From 1e10 on fp32 holds the row's maximum and nothing of the logarithm of the sum: both ways give the same bits."""
    from tagseq2tagseq_b200 import _lib
    dev, L, s = torch.device("cuda"), _lib.lib(), torch.cuda.current_stream().cuda_stream
    x = (torch.randn(2 * len(FILLS) + 2, V, device=dev, generator=torch.Generator(device=dev).manual_seed(V)) * 3).bfloat16()
    n = x.shape[0]
    for i, fill in enumerate(FILLS):
        x[2 * i] = fill                                        # every class ruled out
        x[2 * i + 1] = (x[2 * i + 1].float().clamp(-9, 9) * (-fill / 10)).bfloat16()
        x[2 * i + 1, V // 2] = -fill / 2
    x[n - 2, V // 3] = 3e38
    x[n - 1, ::2], x[n - 1, 1::2] = 3e38, -3e38
    target = torch.tensor([V - 1, 0] * (n // 2), device=dev)
    target[n - 2] = V // 3
    y, z, loss, want, lse, one = x.clone(), x.clone(), torch.empty(n, device=dev), torch.empty(n, device=dev), torch.empty(n, device=dev), torch.ones(1, device=dev)
    _lib.check(L.ts2ts_ce_fwd_grad(y.data_ptr(), target.data_ptr(), loss.data_ptr(), 0.25, n, V, s), "ce")
    _lib.check(L.ts2ts_ce_fwd(z.data_ptr(), target.data_ptr(), lse.data_ptr(), want.data_ptr(), n, V, s), "ce")
    _lib.check(L.ts2ts_ce_bwd(z.data_ptr(), target.data_ptr(), lse.data_ptr(), one.data_ptr(), 0.25, n, V, s), "ce")
    assert lse.isfinite().all() and lse.abs().min() > 1e9
    assert torch.equal(loss, want) and torch.equal(y, z)
