"""Which shapes of a training step keep a graph, with stand-ins for graph and step: captures are counted, no kernel runs."""
import pytest
import torch

from tagseq2tagseq_b200 import train_step
from tagseq2tagseq_b200.train_step import LMConfig, TrainStep


class _Graph:
    made = []

    def __init__(self, owner, tokens, mask, key):
        _Graph.made.append(key)

    def run(self, tokens, mask):
        return "replayed"


@pytest.fixture
def step(monkeypatch):
    _Graph.made = []
    monkeypatch.setattr(train_step, "_StepGraph", _Graph)
    ts = TrainStep(LMConfig(n_layers=1, d_model=8, n_heads=1, head_dim=4, mlp_hidden=8, vocab=16), torch.device("cpu"))
    monkeypatch.setattr(ts, "_eager", lambda *a: "launched")
    return ts


def test_shapes_that_take_turns_are_not_captured_again_and_again(step):
    ran = [step._graphed((i % 5,), torch.zeros(1), None) for i in range(1000)]
    assert len(_Graph.made) == step.MAX_GRAPHS and ran.count("replayed") > 390
    assert len(step._graphs) == step.MAX_GRAPHS


def test_an_idle_graph_makes_room(step):
    for key in ("a", "b"):
        step._graphed(key, None, None), step._graphed(key, None, None)
    for _ in range(step.IDLE_STEPS + 2):
        step._graphed("c", torch.zeros(1), None)
    assert _Graph.made == ["a", "b", "c"] and list(step._graphs) == ["b", "c"]


def test_graphs_are_given_back_when_they_are_turned_off(step):
    step._graphed("a", None, None), step._graphed("a", None, None)
    step.use_graphs = False
    assert step.forward_backward(None, None) == "launched" and not step._graphs


def test_memory_of_a_thin_model_bounds_its_graphs(monkeypatch):
    props = type("Props", (), {"total_memory": 183 << 30})
    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d: props)
    thin = TrainStep(LMConfig(n_layers=2, d_model=64, n_heads=1, head_dim=64, mlp_hidden=128, vocab=50304), torch.device("cpu"))
    assert thin._use_graph(4096) and not thin._use_graph(65536)              # 6.8 GB of logits; by its FLOPs alone it would be small
    assert 6.0 * thin.cfg.matmul_params * 65536 / 1.2e12 < 0.5 * 3
