"""Output head with loss, embedding gradient, AdamW and the norm's weight gradient at the sizes where their kernels change
path or end in a remainder, against PyTorch formulas in fp32 / fp64."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _rel(a, b):
    return ((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("n,k,v", [(1, 64, 8), (33, 72, 1000), (130, 128, 50304), (3, 64, 110592), (5, 64, 120000), (40, 64, 1004)])
@pytest.mark.parametrize("upstream", [1.0, 1.7])
def test_head_loss_matches_torch(n, k, v, upstream):
    from tagseq2tagseq_b200.lm_fused import head_loss
    if v % 8 and upstream != 1.0:
        pytest.skip("refused alike")
    torch.manual_seed(v + n)
    h = torch.randn(n, k, device=DEV).bfloat16().requires_grad_(True)
    w = (torch.randn(v, k, device=DEV) * 0.3).requires_grad_(True)
    t = torch.randint(0, v, (n,), device=DEV)
    if v % 8:  # the loss kernels take rows of whole 16-byte vectors
        with pytest.raises(RuntimeError):
            head_loss(h, w, t)
        return
    loss = head_loss(h, w, t)
    (loss * upstream).backward()
    hr, wr = h.detach().float().requires_grad_(True), w.detach().bfloat16().float().requires_grad_(True)
    logits = (hr @ wr.t())
    ref = F.cross_entropy(logits.detach().bfloat16().float() + (logits - logits.detach()), t)  # the logits' rounding passes the gradient through
    (ref * upstream).backward()
    # fp32 sums of up to 110592 terms of one bf16-rounded row, accumulated per thread and by __expf: 1e-4 relative
    assert abs(loss.item() - ref.item()) <= 1e-4 * max(1.0, abs(ref.item()))
    assert _rel(h.grad, hr.grad) <= 8e-3          # logit gradient and result each rounded to bf16 once (2^-9 each), random signs
    assert _rel(w.grad, wr.grad) <= 4e-3          # one rounding of the logit gradient; the product leaves in fp32


def test_head_loss_ignores_targets_outside_the_vocabulary():
    from tagseq2tagseq_b200.lm_fused import head_loss
    h = torch.randn(6, 64, device=DEV).bfloat16().requires_grad_(True)
    w = torch.randn(512, 64, device=DEV).requires_grad_(True)
    t = torch.tensor([3, -1, 511, 512, 0, -100], device=DEV)
    loss = head_loss(h, w, t)
    loss.backward()
    live = (t >= 0) & (t < 512)
    ref = F.cross_entropy((h.detach().float() @ w.detach().bfloat16().float().t()).bfloat16().float()[live], t[live], reduction="sum") / 6
    assert abs(loss.item() - ref.item()) <= 1e-4 * abs(ref.item())
    assert h.grad[~live].abs().max().item() == 0.0


@pytest.mark.parametrize("n,c,v,same", [(1, 4, 3, False), (9, 100, 50, False), (1000, 768, 300, False), (257, 2048, 50304, False), (515, 256, 10, True)])
def test_embedding_gradient_matches_torch(n, c, v, same):
    from tagseq2tagseq_b200.lm_fused import embedding
    torch.manual_seed(n)
    w = torch.randn(v, c, device=DEV, requires_grad=True)
    idx = torch.full((1, n), 7, device=DEV) if same else torch.randint(0, v, (1, n), device=DEV)
    g = torch.randn(1, n, c, device=DEV)
    out = embedding(w, idx)
    assert torch.equal(out, w.detach()[idx])
    out.backward(g)
    want = torch.zeros(v, c, device=DEV, dtype=torch.float64).index_add_(0, idx[0], g[0].double())
    assert _rel(w.grad, want) <= 2e-6             # fp32 additions of at most 515 terms in any order: sqrt(515) 2^-24
    assert torch.equal(w.grad == 0, want == 0)


def test_adamw_matches_torch_over_steps_shapes_and_alignments():
    from tagseq2tagseq_b200.lm_fused import AdamW
    torch.manual_seed(3)
    base = torch.randn(40001, device=DEV)
    shapes = [(1,), (3,), (4,), (8192,), (8193,), (129, 67), (16384 + 5,)] + [(17,)] * 70    # more tensors than one launch takes
    mine = [torch.randn(s, device=DEV).requires_grad_(True) for s in shapes] + [base[1:].clone().requires_grad_(True)]
    ref = [p.detach().double().requires_grad_(True) for p in mine]
    kw = dict(lr=3e-3, betas=(0.9, 0.95), weight_decay=0.1)
    a, b = AdamW(mine, **kw), torch.optim.AdamW(ref, foreach=False, **kw)
    for step in range(4):
        for i, (p, r) in enumerate(zip(mine, ref)):
            g = torch.randn(p.numel() + 1, device=DEV)[1:].view(p.shape)     # a gradient at an odd address, as bucket views have
            p.grad, r.grad = (None, None) if (step == 2 and i == 1) else (g, g.double())
        a.step()
        b.step()
    for p, r in zip(mine, ref):
        assert _rel(p, r) <= 1e-6                 # a handful of fp32 roundings per step
        assert _rel(a.state[p]["exp_avg_sq"], b.state[r]["exp_avg_sq"]) <= 1e-6
        assert float(a.state[p]["step"]) == float(b.state[r]["step"])
    again = AdamW(mine, **kw)
    again.load_state_dict(a.state_dict())
    assert float(again.state[mine[0]]["step"]) == 4.0


@pytest.mark.parametrize("n,c", [(1, 4), (2, 100), (297, 256), (1185, 768), (4097, 260), (700, 4100), (5, 16384)])
def test_norm_weight_gradient_over_row_and_column_remainders(n, c):
    from tagseq2tagseq_b200.lm_fused import add_rmsnorm
    torch.manual_seed(n + c)
    x = torch.randn(n, c, device=DEV, requires_grad=True)
    w = torch.randn(c, device=DEV, requires_grad=True)
    g, up = torch.randn(n, c, device=DEV).bfloat16(), torch.randn(n, c, device=DEV)
    xo, h = add_rmsnorm(x, None, w, 1e-6)
    torch.autograd.backward([xo, h], [up, g])
    xr, wr = x.detach().double().requires_grad_(True), w.detach().double().requires_grad_(True)
    torch.autograd.backward([xr * 1.0, F.rms_norm(xr, (c,), wr, 1e-6)], [up.double(), g.double()])
    assert _rel(x.grad, xr.grad) <= 2e-6          # fp32 arithmetic, sums of at most 16384 terms
    assert _rel(w.grad, wr.grad) <= 4e-6


def test_optimizer_step_is_refused_during_capture():
    from tagseq2tagseq_b200.lm_fused import AdamW
    p = torch.nn.Parameter(torch.ones(64, device=DEV))
    p.grad = torch.ones_like(p)
    opt = AdamW([p])
    opt.step()
    before = p.detach().clone()
    with torch.cuda.graph(torch.cuda.CUDAGraph()):
        kept = torch.zeros(1, device=DEV)  # a graph of something
        with pytest.raises(RuntimeError, match="capturable"):
            opt.step()
    assert kept is not None and torch.equal(p, before) and float(opt.state[p]["step"]) == 1.0


def test_layer_operators_break_a_compiled_graph_and_run():
    from tagseq2tagseq_b200.lm_fused import add_rmsnorm, swiglu

    def fn(x, w, p):
        _, h = add_rmsnorm(x * 1.5, None, w, 1e-6)
        return (swiglu(h @ p).float() * 2).sum()

    gen = torch.Generator(device=DEV).manual_seed(5)
    leaves = [torch.randn(s, device=DEV, generator=gen).requires_grad_() for s in ((1, 40, 64), (64,))]
    p = torch.randn(64, 128, device=DEV, generator=gen).bfloat16()
    want = torch.autograd.grad(fn(*leaves, p), leaves)
    got = torch.autograd.grad(torch.compile(fn, backend="aot_eager")(*leaves, p), leaves)
    for a, b in zip(got, want):
        assert _rel(a, b) <= 1e-5


def test_head_loss_refuses_a_target_of_another_length():
    from tagseq2tagseq_b200.lm_fused import head_loss
    h = torch.zeros(1, 5, 64, device=DEV, dtype=torch.bfloat16)
    w = torch.zeros(16, 64, device=DEV, requires_grad=True)
    with pytest.raises(ValueError):
        head_loss(h, w, torch.zeros(1, 4, device=DEV, dtype=torch.int64))
