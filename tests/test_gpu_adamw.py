"""The native AdamW step: refused calls, loss scaling, states of other optimizers, and its rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def test_a_refused_step_advances_no_counter():
    from tagseq2tagseq_b200 import _lib
    p, g, m, v = ([torch.ones(8, device=DEV) for _ in range(2)] for _ in range(4))
    steps = [torch.zeros(()) for _ in range(2)]
    g[1] = torch.ones(7, device=DEV)
    with pytest.raises(ValueError, match="adamw"):
        _lib.ops().adamw(p, g, m, v, steps, 1e-3, 0.9, 0.95, 1e-8, 0.1)
    assert [float(s) for s in steps] == [0.0, 0.0] and float(p[0][0]) == 1.0
    _lib.ops().adamw(p[:1], g[:1], m[:1], v[:1], steps[:1], 1e-3, 0.9, 0.95, 1e-8, 0.1)
    assert [float(s) for s in steps] == [1.0, 0.0]


def test_a_gradient_scaler_is_not_passed_by():
    """With fused=True the scaler hands its scale and its inf flag to the optimizer instead of acting on them itself."""
    from tagseq2tagseq_b200.lm_fused import AdamW
    for kw in ({"fused": True}, {}):
        p = torch.nn.Parameter(torch.ones(16, device=DEV))
        plain = torch.nn.Parameter(torch.ones(16, device=DEV))
        opt, ref = AdamW([p], lr=1e-2, eps=1e-3, **kw), torch.optim.AdamW([plain], lr=1e-2, eps=1e-3)
        scaler = torch.amp.GradScaler("cuda", init_scale=1024.0)
        scaler.scale(torch.zeros((), device=DEV))
        p.grad = torch.full_like(p, float("inf"))
        scaler.step(opt)
        scaler.update()
        assert torch.equal(p.detach(), torch.ones_like(p)), kw
        p.grad, plain.grad = torch.full_like(p, 2e-3 * scaler.get_scale()), torch.full_like(p, 2e-3)
        scaler.step(opt)
        ref.step()
        assert (p - plain).abs().max() <= 1e-6, kw


def test_subnormal_moments_are_kept():
    from tagseq2tagseq_b200.lm_fused import AdamW
    p = torch.nn.Parameter(torch.ones(40, device=DEV))
    p.grad = torch.full_like(p, 1e-20)
    opt = AdamW([p], lr=1.0, betas=(0.9, 0.95), eps=1e-25, weight_decay=0.0)
    opt.step()
    v = opt.state[p]["exp_avg_sq"].double()
    assert (v - 0.05e-40).abs().max() <= 2e-45                   # half a unit of the smallest fp32 number, twice
    assert p.detach().abs().max() <= 2e-3                        # m / sqrt(v) is one after the bias corrections; v has 12 bits here


def test_states_of_other_strides_and_counters_are_taken():
    from tagseq2tagseq_b200.lm_fused import AdamW
    torch.manual_seed(0)
    p = torch.nn.Parameter(torch.randn(24, 40, device=DEV))
    ref = torch.nn.Parameter(p.detach().clone())
    a, b = AdamW([p], lr=1e-2), torch.optim.AdamW([ref], lr=1e-2)
    grads = [torch.randn(24, 40, device=DEV) for _ in range(3)]
    for g in grads[:2]:
        p.grad, ref.grad = g.clone(), g.clone()
        a.step(), b.step()
    sd = a.state_dict()
    st = sd["state"][0]
    st["exp_avg"], st["exp_avg_sq"] = (st[k].t().contiguous().t() for k in ("exp_avg", "exp_avg_sq"))
    st["step"] = st["step"].double()
    a = AdamW([p], lr=1e-2)
    a.load_state_dict(sd)
    a.state[p]["step"] = a.state[p]["step"].double()
    p.grad, ref.grad = grads[2].clone(), grads[2].clone()
    a.step(), b.step()
    assert (p - ref).abs().max() <= 1e-6 and float(a.state[p]["step"]) == 3.0
