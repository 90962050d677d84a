"""Capturing a training step: what must not be in its way, and what happens when it fails."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def _make(seed=7):
    from tagseq2tagseq_b200.train_step import LMConfig, TrainStep
    return TrainStep(LMConfig(n_layers=1, d_model=128, n_heads=2, head_dim=64, mlp_hidden=256, vocab=512), DEV, seed=seed)


def _batch(t=200, seed=1):
    from tagseq2tagseq_b200.mask_spec import MaskSpec
    doc = (torch.arange(t, device=DEV, dtype=torch.int32) // 50)[None]
    return torch.randint(0, 512, (1, t + 1), generator=torch.Generator().manual_seed(seed)).to(DEV), MaskSpec(doc)


def test_a_live_autograd_graph_of_the_same_parameters_is_not_in_the_way():
    ts = _make()
    with torch.autocast("cuda", torch.bfloat16):
        kept = ts.model(*_batch(seed=2))                                    # its backward comes later
    want = _make()
    want.use_graphs = False
    for i in range(4):
        a, b = ts.forward_backward(*_batch(seed=i)), want.forward_backward(*_batch(seed=i))
        assert torch.equal(a, b)
        assert all(torch.equal(p.grad, r.grad) for p, r in zip(ts.model.parameters(), want.model.parameters()))
    assert any(g is not None for g in ts._graphs.values())
    kept.backward()


def test_a_step_that_cannot_be_captured_runs_launched(monkeypatch):
    from tagseq2tagseq_b200 import train_step

    def fails(*a):
        raise RuntimeError("operation not permitted when stream is capturing")
    ts = _make()
    monkeypatch.setattr(train_step, "_StepGraph", fails)
    want = _make()
    want.use_graphs = False
    with pytest.warns(UserWarning, match="could not be captured"):
        for i in range(4):
            assert torch.equal(ts.step(*_batch(seed=i)), want.step(*_batch(seed=i)))


def test_replays_on_two_streams_do_not_share_their_inputs():
    ts, want = _make(), _make()
    want.use_graphs = False
    expect = [float(want.forward_backward(*_batch(seed=i))) for i in range(6)]
    assert len(set(expect)) == 6
    for _ in range(2):
        ts.forward_backward(*_batch(seed=0))
    batches = [_batch(seed=i) for i in range(6)]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream() for _ in range(2)], []
    for i, batch in enumerate(batches):
        with torch.cuda.stream(streams[i % 2]):
            if i % 2 == 0:
                torch.cuda._sleep(20_000_000)                               # some ten milliseconds: the other stream is ahead
            got.append(ts.forward_backward(*batch))
    torch.cuda.synchronize()
    assert [float(x) for x in got] == expect
