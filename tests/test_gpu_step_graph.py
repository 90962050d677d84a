"""The training step as a CUDA graph against the same step launched kernel by kernel: packs of different document counts,
sequence lengths that come and go, and the conditions under which a graph must not be replayed."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda", 0)


def _make(seed=7):
    from tagseq2tagseq_b200.train_step import LMConfig, TrainStep
    return TrainStep(LMConfig(n_layers=2, d_model=128, n_heads=2, head_dim=64, mlp_hidden=256, vocab=512), DEV, seed=seed)


def _batch(i, t, p_link=0.3, median=20):
    from tagseq2tagseq_b200 import synth
    from tagseq2tagseq_b200.mask_spec import MaskSpec
    pack = synth.make_pack(500 + i, t, median, 4, 200, p_link=p_link)
    doc = torch.from_numpy(pack.doc_ids)[None].to(DEV)
    spec = MaskSpec(doc, None if pack.link_bits is None else torch.from_numpy(pack.link_bits)[None].to(DEV))
    return torch.randint(0, 512, (1, t + 1), generator=torch.Generator().manual_seed(i)).to(DEV), spec


def test_replayed_steps_equal_launched_steps():
    a, b = _make(), _make()
    b.use_graphs = False
    # 25 to 40 documents (one padded shape of the link bits), a second length, no links, then the first length again
    plan = [(i, 600, 0.3) for i in range(5)] + [(5, 333, 0.3), (6, 333, 0.3), (7, 600, 0.0), (8, 600, 0.0), (9, 129, 0.2), (10, 129, 0.2), (11, 600, 0.3)]
    kept = []
    for i, t, p in plan:
        la, lb = a.step(*_batch(i, t, p)), b.step(*_batch(i, t, p))
        kept.append((la, float(la)))
        # same kernels on the same values: dq's order of fp32 additions differs from run to run, and Adam's first steps pass
        # a changed sign of a tiny gradient on as a whole step of 3e-4
        assert abs(float(la) - float(lb)) <= 2e-3 * abs(float(lb)), i
        for x, y in zip(a.model.parameters(), b.model.parameters()):
            assert (x.grad - y.grad).norm() <= 2e-2 * y.grad.norm() + 1e-6
    assert sum(g is not None for g in a._graphs.values()) == a.MAX_GRAPHS
    assert not b._graphs
    assert all(float(l) == v for l, v in kept)      # a returned loss does not change with later steps


def test_hooks_and_replaced_parameters_are_not_replayed_over():
    ts = _make()
    for i in range(3):
        ts.step(*_batch(i, 300))
    assert any(g is not None for g in ts._graphs.values())
    calls = []
    handle = ts.model.blocks[0].register_forward_hook(lambda m, i, o: calls.append(1))
    ts.step(*_batch(3, 300))
    assert calls == [1]
    handle.remove()
    ts.model.head.weight.data = torch.zeros_like(ts.model.head.weight)      # another address: logits 0, loss ln 512
    loss = ts.forward_backward(*_batch(4, 300))
    assert abs(float(loss) - 6.2383) <= 1e-3
    for i in range(3):
        assert abs(float(ts.forward_backward(*_batch(5, 300))) - 6.2383) <= 1e-3
    assert any(g is not None for g in ts._graphs.values())                   # captured again at the new address


def test_gradients_of_a_step_outlive_the_next_one():
    ts = _make()
    for i in range(2):
        ts.forward_backward(*_batch(i, 300))
    held = [p.grad for p in ts.model.parameters()]
    before = [g.clone() for g in held]
    ts.forward_backward(*_batch(2, 300))
    assert all(torch.equal(g, b) for g, b in zip(held, before))
    assert any(not torch.equal(p.grad, b) for p, b in zip(ts.model.parameters(), before))


def test_graph_keeps_the_rotation_tables_it_reads():
    ts = _make()
    for i in range(2):
        ts.forward_backward(*_batch(i, 300))
    graph, = [g for g in ts._graphs.values() if g is not None]
    tables = ts.model._rope[1]
    ts.forward_backward(*_batch(2, 200))                    # the model now holds another length's tables
    assert ts.model._rope[1] is not tables
    assert all(a is b for a, b in zip(graph.tables, tables))
