"""What autograd is told about the decoder-layer operators, compared with torch's own layers: changed inputs, second
derivatives, transforms."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _linear(n_in=64, n_out=24):
    from tagseq2tagseq_b200.lm_fused import Linear
    torch.manual_seed(n_in)
    return Linear(n_in, n_out).to(DEV)


def _bf16(*shape):
    return torch.randn(*shape, device=DEV).bfloat16()


def test_an_input_written_to_before_the_backward_is_noticed():
    from tagseq2tagseq_b200.lm_fused import head_loss
    lin, w = _linear(), torch.randn(128, 64, device=DEV, requires_grad=True)
    with torch.autocast("cuda", torch.bfloat16):
        x = _bf16(2, 5, 64)
        for y in (lin(x).sum(), head_loss(x, w, torch.zeros(10, dtype=torch.int64, device=DEV))):
            x.add_(1)
            with pytest.raises(RuntimeError, match="inplace"):
                y.backward()


def test_a_weight_changed_before_the_backward_does_not_matter():
    """As under autocast, which multiplies by a copy: the gradient belongs to the weight of the forward."""
    lin, x = _linear(), _bf16(7, 64).requires_grad_(True)
    with torch.autocast("cuda", torch.bfloat16):
        y = lin(x)
    want = lin.weight.detach().bfloat16().float().sum(0)
    with torch.no_grad():
        lin.weight.zero_()
    y.sum().backward()
    assert (x.grad.float() - want).abs().max() <= 2 ** -8 * want.abs().max()


def test_second_derivative_of_a_linear_layer_matches_torch():
    """A gradient penalty reaches the weight through x, dy and the weight itself."""
    lin = _linear(64, 32)
    grads = []
    for layer in (lambda x: lin(x), lambda x: F.linear(x, lin.weight)):
        torch.manual_seed(5)
        x = torch.randn(3, 9, 64, device=DEV).bfloat16().requires_grad_(True)
        lin.weight.grad = None
        with torch.autocast("cuda", torch.bfloat16):
            y = layer(x)
        gx, gw = torch.autograd.grad((y.float() ** 3).sum(), (x, lin.weight), create_graph=True)
        (gx.float().pow(2).sum() + gw.float().pow(2).sum()).backward()
        grads.append((x.grad.double(), lin.weight.grad.double()))
    for a, b in zip(*grads):
        assert (a - b).norm() <= 4 * 2 ** -8 * b.norm()     # bf16 products and results on either side, rounded a few times each
    with torch.autocast("cuda", torch.bfloat16):
        y = lin(x)
    with torch.no_grad():
        lin.weight.add_(1)
    with pytest.raises(RuntimeError, match="inplace"):
        torch.autograd.grad(y.sum(), x, create_graph=True)


def _layer_losses():
    from tagseq2tagseq_b200 import lm_fused as lf
    from tagseq2tagseq_b200.mask_spec import MaskSpec
    x, w = torch.randn(6, 64, device=DEV, requires_grad=True), torch.randn(64, device=DEV, requires_grad=True)
    yield "add_rmsnorm", lf.add_rmsnorm(x, None, w, 1e-6)[1].float().pow(2).sum(), x
    gu = _bf16(6, 128).requires_grad_(True)
    yield "swiglu", lf.swiglu(gu).float().pow(2).sum(), gu
    h, wh = _bf16(6, 64).requires_grad_(True), torch.randn(128, 64, device=DEV, requires_grad=True)
    target = torch.arange(6, device=DEV)
    yield "head_loss", lf.head_loss(h, wh, target), h
    yield "head_loss", lf.head_loss(h, wh, target), wh
    logits = _bf16(6, 128).requires_grad_(True)
    yield "cross_entropy", lf.cross_entropy(logits * 1, target), logits
    qkv = _bf16(1, 6, 3 * 64).requires_grad_(True)
    cos, sin = lf.rope_half_tables(6, 64, 10000.0, DEV)
    mask = MaskSpec(torch.zeros(1, 6, dtype=torch.int32, device=DEV))
    yield "qkv_attention", lf.qkv_attention(qkv * 1, cos, sin, mask, 1, 64).float().pow(2).sum(), qkv


def test_second_derivatives_of_the_layer_kernels_are_refused():
    for name, loss, at in _layer_losses():
        grad, = torch.autograd.grad(loss, at, create_graph=True)
        with pytest.raises(RuntimeError, match="not implemented"):
            grad.float().pow(2).sum().backward()
        assert grad.isfinite().all(), name


def test_second_derivative_of_an_embedding_matches_torch():
    from tagseq2tagseq_b200.lm_fused import embedding
    idx = torch.tensor([[3, 1, 3, 0]], device=DEV)
    got = []
    for f in (embedding, lambda w, i: F.embedding(i, w)):
        torch.manual_seed(1)
        w = torch.randn(5, 8, device=DEV, requires_grad=True)
        g, = torch.autograd.grad(f(w, idx).pow(3).sum(), w, create_graph=True)
        got.append(torch.autograd.grad(g.pow(2).sum(), w)[0])
    assert (got[0] - got[1]).norm() <= 1e-6 * got[1].norm()


def test_linear_outside_bf16_autocast_is_torchs_layer():
    lin, x = _linear(), _bf16(4, 64)
    with pytest.raises(RuntimeError, match="dtype"):
        lin(x)                                                       # bf16 against an fp32 weight
    with torch.autocast("cuda", torch.float16):
        assert torch.equal(lin(x), F.linear(x, lin.weight)) and lin(x).dtype == torch.float16
    with torch.autocast("cuda", torch.bfloat16):
        ref = torch.func.grad(lambda t: F.linear(t, lin.weight).float().pow(2).sum())(x)
        assert torch.equal(torch.func.grad(lambda t: lin(t).float().pow(2).sum())(x), ref)
        with torch.autograd.forward_ad.dual_level():
            dual = torch.autograd.forward_ad.make_dual(x, torch.ones_like(x))
            assert torch.autograd.forward_ad.unpack_dual(lin(dual)).tangent is not None
