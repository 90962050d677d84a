"""Replayed steps look at their inputs and at their caller as launched ones do."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def _make():
    from tagseq2tagseq_b200.train_step import LMConfig, TrainStep
    return TrainStep(LMConfig(n_layers=1, d_model=128, n_heads=2, head_dim=64, mlp_hidden=256, vocab=512), DEV)


def _batch(t=200, b=2, links=True):
    from tagseq2tagseq_b200.mask_spec import MaskSpec
    doc = (torch.arange(t, device=DEV, dtype=torch.int32) // 50).expand(b, t).contiguous()
    link = torch.full((b, 4, 1), 1, dtype=torch.int64, device=DEV) if links else None
    return torch.randint(0, 512, (b, t + 1), generator=torch.Generator().manual_seed(1)).to(DEV), MaskSpec(doc, link, doc.clone(), doc.clone())


def _replaying():
    ts = _make()
    for _ in range(3):
        ts.forward_backward(*_batch())
    assert any(g is not None for g in ts._graphs.values())
    return ts


@pytest.mark.parametrize("field,wrong", [
    ("doc_ids", lambda t: t.long()), ("q_row_ids", lambda t: t[:1]), ("kv_col_ids", lambda t: t.long()),
    ("link_bits", lambda t: t[:1]), ("link_bits", lambda t: t.cpu()), ("link_bits", lambda t: t.int())])
def test_inputs_a_launched_step_refuses_are_refused(field, wrong):
    ts = _replaying()
    tokens, mask = _batch()
    setattr(mask, field, wrong(getattr(mask, field)))
    with pytest.raises((ValueError, RuntimeError)):
        ts.forward_backward(tokens, mask)


def test_hooks_modes_and_anomaly_detection_see_a_launched_step():
    ts, seen = _replaying(), []

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(func)
            return func(*args, **(kwargs or {}))

    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(t) or t, lambda t: t):
        ts.forward_backward(*_batch())
    saved = len(seen)
    with Mode():
        ts.forward_backward(*_batch())
    assert saved > 10 and len(seen) > saved + 10
    ts.model.embed.weight.data.fill_(float("nan"))
    with torch.autograd.detect_anomaly(), pytest.raises(RuntimeError, match="nan"):
        ts.forward_backward(*_batch())
