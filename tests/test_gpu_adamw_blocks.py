"""The native AdamW step over aligned tensors around the elements of one block (2048) and of one of a thread's vectors (1024 a block)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("sizes", [(4, 1023, 1024, 1027, 2045), (2047, 2048, 2049), (3 * 2048 + 1020, 4095, 4100, 1 << 20)])
def test_vectors_and_remainders(sizes):
    from tagseq2tagseq_b200.lm_fused import AdamW
    torch.manual_seed(sum(sizes))
    mine = [torch.randn(n, device=DEV).requires_grad_(True) for n in sizes]
    ref = [p.detach().double().requires_grad_(True) for p in mine]
    kw = dict(lr=3e-3, betas=(0.9, 0.95), weight_decay=0.1)
    a, b = AdamW(mine, **kw), torch.optim.AdamW(ref, foreach=False, **kw)
    for _ in range(2):
        for p, r in zip(mine, ref):
            p.grad = torch.randn_like(p)
            r.grad = p.grad.double()
        a.step(), b.step()
    for p, r in zip(mine, ref):
        for got, want, terms in ((p, r, 1), (a.state[p]["exp_avg"], b.state[r]["exp_avg"], 0.6), (a.state[p]["exp_avg_sq"], b.state[r]["exp_avg_sq"], 1.6)):
            # a step rounds a value eight times at most, by half of 2^-23 of it or of what goes into it: 0.1 of a gradient and 0.05 of its square, gradients up to 5.5
            bound = 2 * 8 * 2.0**-24 * (want.abs() + terms)
            assert ((got.detach().double() - want.detach()).abs() <= bound).all()
