"""The embedding gradient at the sizes where its kernel changes path: ends of a stretch of tokens, a full queue, ids of many
rows, column remainders; every sum repeats bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _ids(kind, n, v):
    g = torch.Generator().manual_seed(n)
    if kind == "uniform":
        return torch.randint(0, v, (n,), generator=g)
    if kind == "zipf":  # a few ids take most tokens
        return (v ** torch.rand(n, generator=g)).long().clamp(0, v - 1)
    if kind == "bucket":  # one block's ids only: the queue fills and is emptied many times
        return torch.randint(0, v // 256, (n,), generator=g) * 256
    if kind == "runs":  # exactly 64 and 65 rows of an id
        return torch.arange(n) // 65 + (torch.arange(n) % 65 == 64).long()
    return torch.full((n,), 3)


@pytest.mark.parametrize("kind,n,c,v", [
    ("uniform", 1, 4, 5), ("uniform", 511, 132, 40), ("uniform", 2048, 512, 4096), ("uniform", 2049, 516, 4096),
    ("zipf", 16384, 768, 50304), ("zipf", 5000, 2052, 3000), ("bucket", 9001, 128, 4096), ("bucket", 3073, 260, 512), ("runs", 3900, 64, 100),
    ("same", 64, 128, 4), ("same", 65, 640, 4), ("same", 9000, 640, 4)])
def test_sums_are_right_and_repeat(kind, n, c, v):
    from tagseq2tagseq_b200.lm_fused import embedding
    idx = _ids(kind, n, v).to(DEV)[None]
    w, g = torch.zeros(v, c, device=DEV, requires_grad=True), torch.randn(1, n, c, device=DEV)
    got = [torch.autograd.grad(embedding(w, idx), w, g)[0] for _ in range(3)]
    assert all(torch.equal(got[0], x) for x in got)
    want = torch.zeros(v, c, device=DEV, dtype=torch.float64).index_add_(0, idx[0], g[0].double())
    most = int(torch.bincount(idx[0]).max())
    # each of at most `most` additions rounds a partial sum of size sqrt(most) by 2^-24, in random directions
    assert (got[0].double() - want).abs().max() <= 8 * most * 2 ** -24
    assert torch.equal(got[0] == 0, want == 0)


def test_no_tokens_give_a_zero_gradient():
    from tagseq2tagseq_b200.lm_fused import embedding
    w = torch.randn(7, 8, device=DEV, requires_grad=True)
    embedding(w, torch.zeros(1, 0, dtype=torch.int64, device=DEV)).sum().backward()
    assert torch.equal(w.grad, torch.zeros_like(w))


def test_gradients_at_odd_addresses_and_transforms_are_taken_as_torch_takes_them():
    from tagseq2tagseq_b200.lm_fused import embedding
    idx = torch.tensor([[3, 1, 3]], device=DEV)
    w, g = torch.randn(7, 8, device=DEV, requires_grad=True), torch.randn(25, device=DEV)[1:].view(1, 3, 8)
    got, = torch.autograd.grad(embedding(w, idx), w, g)
    want, = torch.autograd.grad(torch.nn.functional.embedding(idx, w), w, g)
    assert torch.equal(got, want)
    grad = torch.func.grad(lambda t: (embedding(t, idx) * g).sum())(w.detach())
    assert torch.equal(grad, want)
