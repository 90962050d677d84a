"""What autograd is told about the torch operators, with stand-ins for the kernels on the CPU: results that have no
derivative refuse to be differentiated instead of leaving a gradient out."""
import pytest
import torch


@pytest.fixture
def ops():
    from tagseq2tagseq_b200 import attention  # noqa: F401  loads the operators
    with torch.library._scoped_library("ts2ts", "IMPL") as lib:
        lib.impl("masked_attn_fwd", lambda q, k, v, *rest: (q * k * v, q.float().sum(-1)), "CPU")
        lib.impl("masked_attn_bwd", lambda q, k, v, out, dout, *rest: (dout * k * v, dout * q * v, dout * q * k), "CPU")
        lib.impl("masked_attn_decode", lambda q, k, v, *rest: (q * 2, q.float().sum(-1)), "CPU")
        yield torch.ops.ts2ts


def _args(requires_grad=True):
    q, k, v = (torch.randn(1, 2, 4, 64, requires_grad=requires_grad) for _ in range(3))
    return q, k, v, torch.zeros(1, 4, dtype=torch.int32), None, None, None


def test_first_derivative_passes_and_second_is_refused(ops):
    args = _args()
    plan = torch.zeros(4, dtype=torch.uint8)
    out, lse = ops.masked_attn_fwd(*args, plan, 1.0)
    assert not lse.requires_grad
    dq, = torch.autograd.grad(out.sum(), args[0], retain_graph=True)
    assert torch.equal(dq, (args[1] * args[2]).detach()) and not dq.requires_grad
    dq, = torch.autograd.grad(out.sum(), args[0], create_graph=True)
    with pytest.raises(RuntimeError, match="not implemented"):
        dq.sum().backward()


def test_decoding_step_refuses_a_gradient(ops):
    out, _ = ops.masked_attn_decode(*_args(), None, 1.0)
    with pytest.raises(RuntimeError, match="not implemented"):
        out.sum().backward()
    out, _ = ops.masked_attn_decode(*_args(False), None, 1.0)
    assert not out.requires_grad
    with torch.no_grad():
        assert not ops.masked_attn_decode(*_args(), None, 1.0)[0].requires_grad
