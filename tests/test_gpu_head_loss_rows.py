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
