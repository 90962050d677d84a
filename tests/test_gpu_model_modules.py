"""The model's embedding and head are used as modules: what a program hangs on them or puts in their place takes effect."""
import pytest
import torch
import torch.nn as nn
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def _step(**kw):
    from tagseq2tagseq_b200.train_step import LMConfig, TrainStep
    ts = TrainStep(LMConfig(n_layers=1, d_model=128, n_heads=2, head_dim=64, mlp_hidden=256, vocab=512), DEV, **kw)
    ts.use_graphs = False
    return ts


def _batch(t=200):
    from tagseq2tagseq_b200.mask_spec import MaskSpec
    doc = (torch.arange(t, device=DEV, dtype=torch.int32) // 50)[None]
    return torch.randint(0, 512, (1, t + 1), generator=torch.Generator().manual_seed(1)).to(DEV), MaskSpec(doc)


def test_hooks_on_embedding_and_head_are_called():
    ts, seen = _step(), []
    loss = float(ts.forward_backward(*_batch()))
    for m in (ts.model.embed, ts.model.head):
        m.register_forward_hook(lambda m, i, o: seen.append(tuple(o.shape)))
        m.register_forward_pre_hook(lambda m, i: seen.append("pre"))
        m.register_full_backward_hook(lambda m, gi, go: seen.append("grad"))
    again = float(ts.forward_backward(*_batch()))
    assert seen == ["pre", (1, 200, 128), "pre", (1, 200, 512), "grad", "grad"]
    assert abs(again - loss) <= 2e-3 * abs(loss)
    ts.model.head.register_forward_hook(lambda m, i, o: o * 0)             # logits 0: loss ln 512
    assert abs(float(ts.forward_backward(*_batch())) - 6.2383) <= 1e-3


def test_other_modules_in_their_place_are_used():
    ts = _step()
    old = ts.model.head.weight.detach().clone()
    ts.model.head = nn.Linear(128, 512).to(DEV)
    with torch.no_grad():
        ts.model.head.weight.zero_()
        ts.model.head.bias.fill_(0.0)
        ts.model.head.bias[0] = 20.0
    tokens, mask = _batch()
    want = F.cross_entropy(ts.model.head.bias.detach().expand(200, 512), tokens[0, 1:])
    assert abs(float(ts.forward_backward(tokens, mask)) - float(want)) <= 1e-2 * float(want)
    assert ts.model.head.bias.grad.abs().max() > 0 and not torch.equal(ts.model.head.weight, old)
    ts = _step()
    ts.model.embed.padding_idx = 3
    ts.forward_backward(tokens.fill_(3), mask)
    assert ts.model.embed.weight.grad.abs().max() == 0                      # a padding row takes no gradient
