"""The rotation tables a model keeps: what they are kept by, and who may use them."""
import copy
import pickle

import torch

from tagseq2tagseq_b200.train_step import DecoderLM, LMConfig

CPU = torch.device("cpu")


def _model(cls=DecoderLM, **kw):
    return cls(LMConfig(n_layers=1, d_model=8, n_heads=1, head_dim=4, mlp_hidden=8, vocab=16, **kw))


def test_tables_follow_length_and_base():
    m = _model()
    a = m._rope_tables(5, CPU)
    assert m._rope_tables(5, CPU) is a and m._rope_tables(7, CPU)[0].shape == (7, 2)
    b = m._rope_tables(5, CPU)
    m.cfg.rope_base = 500.0
    assert torch.equal(a[0], b[0]) and not torch.equal(m._rope_tables(5, CPU)[0], a[0])


def test_another_threads_length_is_not_handed_out():
    class Raced(DecoderLM):
        def __setattr__(self, name, value):  # another thread's tables take the place at once
            super().__setattr__(name, value)
            if name == "_rope" and value is not None and value[1][0].shape[0] == 5:
                self._rope_tables(3, CPU)
    assert _model(Raced)._rope_tables(5, CPU)[0].shape == (5, 2)


def test_tables_made_in_inference_mode_can_be_saved_for_a_backward():
    m = _model()
    with torch.inference_mode():
        m._rope_tables(5, CPU)
    assert not any(t.is_inference() for t in m._rope_tables(5, CPU))


def test_a_model_is_copied_and_saved_without_them():
    m = _model()
    m._rope_tables(5, CPU)
    for other in (copy.deepcopy(m), pickle.loads(pickle.dumps(m))):
        assert other._rope is None and torch.equal(other._rope_tables(5, CPU)[1], m._rope_tables(5, CPU)[1])
