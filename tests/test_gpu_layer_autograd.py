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
