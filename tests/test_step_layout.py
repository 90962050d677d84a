"""When a training step may be replayed as a graph: anything that makes the model another one, or hangs something on it, is
noticed.  No kernel runs: the question is asked of a model on the CPU."""
import pytest
import torch
import torch.nn as nn

from tagseq2tagseq_b200.train_step import DecoderLM, LMConfig, TrainStep

CFG = dict(n_layers=1, d_model=8, n_heads=1, head_dim=4, mlp_hidden=8, vocab=16)


@pytest.fixture
def step():
    ts = TrainStep(LMConfig(**CFG), torch.device("cpu"))
    assert ts._as_built() and ts._as_built()
    ts._graphs["a shape"] = "its graph"
    return ts


def test_a_replaced_model_drops_the_old_ones_graphs(step):
    step.model = DecoderLM(LMConfig(**CFG))
    assert step._as_built() and not step._graphs


@pytest.mark.parametrize("change", [
    lambda m: setattr(m, "head", nn.Linear(8, 16)), lambda m: setattr(m.blocks[0], "down", nn.Sequential(m.blocks[0].down, nn.Dropout(0.5))),
    lambda m: m.blocks.append(nn.Identity()), lambda m: nn.utils.parametrize.register_parametrization(m.head, "weight", nn.Identity())])
def test_a_model_with_foreign_modules_is_not_replayed(step, change):
    change(step.model)
    assert not step._as_built() and not step._graphs


@pytest.mark.parametrize("change", [
    lambda m: setattr(m.head, "weight", nn.Parameter(m.head.weight.detach().clone())), lambda m: setattr(m.head.weight, "data", m.head.weight.detach().clone()),
    lambda m: setattr(m.head, "bias", nn.Parameter(torch.zeros(16))), lambda m: setattr(m.cfg, "rope_base", 500.0),
    lambda m: setattr(m.embed, "padding_idx", 3), lambda m: setattr(m.blocks[0], "cfg", LMConfig(**dict(CFG, n_heads=2, head_dim=2)))])
def test_a_changed_model_is_captured_anew(step, change):
    change(step.model)
    step._as_built()
    assert not step._graphs


@pytest.mark.parametrize("change", [
    lambda m: m.blocks[0].register_forward_hook(lambda *a: None), lambda m: m.head.register_forward_pre_hook(lambda *a: None),
    lambda m: m.embed.register_full_backward_hook(lambda *a: None), lambda m: m.head.weight.register_hook(lambda g: g),
    lambda m: m.head.weight.requires_grad_(False), lambda m: setattr(m.blocks[0], "forward", lambda *a: a)])
def test_hooks_and_replaced_forwards_are_not_replayed_over(step, change):
    change(step.model)
    assert not step._as_built() and step._graphs  # kept for when it is gone again


def test_a_class_whose_forward_was_replaced_is_noticed(step, monkeypatch):
    monkeypatch.setattr(DecoderLM, "forward", lambda self, *a: 0)
    assert not step._as_built()


def test_a_step_on_the_cpu_is_refused_as_the_kernels_refuse_it():
    from tagseq2tagseq_b200 import MaskSpec
    ts = TrainStep(LMConfig(**CFG), torch.device("cpu"))
    with pytest.raises(RuntimeError, match="CUDA"):
        ts.forward_backward(torch.zeros(1, 5, dtype=torch.int64), MaskSpec(torch.zeros(1, 4, dtype=torch.int32)))
