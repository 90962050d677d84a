"""Branches of the pre-pass that sizes choose."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _two_packs(t):
    """Two sequences of documents of different lengths, so that the batch elements' lists and orders differ."""
    return torch.from_numpy(np.stack([np.arange(t) // 700, np.sqrt(np.arange(t) * 40).astype(np.int64) // 50]).astype(np.int32)).cuda()


@pytest.mark.parametrize("t", [128 * 32 + 1, 128 * 257])
def test_lists_of_more_tiles_than_one_sweep(t):
    """Fewer and more than 256 tiles (a sweep of the lists), the last tile ragged or not: every list is what the states say."""
    from tagseq2tagseq_b200 import build_block_map
    nb = -(-t // 128)
    bm = build_block_map(_two_packs(t), with_lists=True)
    for b in range(2):
        state = bm.state[b].cpu().numpy()
        outs = [x[b].cpu().numpy() for x in (bm.kv_cnt, bm.kv_idx, bm.full_cnt, bm.full_idx, bm.q_cnt, bm.q_idx, bm.full_q_cnt, bm.full_q_idx)]
        for (cnt, idx), s in zip(zip(outs[0::2], outs[1::2]), (state == 1, state == 2, (state == 1).T, (state == 2).T)):
            for line in range(nb):
                want = np.flatnonzero(s[line])
                assert cnt[line] == want.size and np.array_equal(idx[line, :want.size], want) and (idx[line, want.size:] == -1).all()


@pytest.mark.parametrize("nb", [1, 2, 31, 32, 33, 64, 65, 257, 1026])
def test_launch_orders_are_permutations_by_descending_count(nb):
    """The orders of q tiles, kv tiles and q-tile pairs, around the 32 tiles that a block ranks and the 1024 counts that it reads at a
    time: heaviest first, ties by index.  A missing or doubled rank would leave rows of the result unwritten."""
    from tagseq2tagseq_b200 import build_block_map
    doc = _two_packs(128 * nb - 5)
    bm = build_block_map(doc, with_lists=True)
    words, at, part = bm.plan.cpu().view(torch.int32).numpy(), 256, {}
    pairs = (nb + 1) // 2
    for name, count, size in (("run_cnt", nb, 4), ("runs", nb * 128, 16), ("state", nb * nb, 1), ("fwd_cnt", nb, 4), ("fwd_idx", nb * nb, 4),  # csrc/plan.h
                              ("bwd_cnt", nb, 4), ("bwd_idx", nb * nb, 4), ("fwd_order", nb, 4), ("bwd_order", nb, 4), ("pair_cnt", pairs, 4), ("pair_order", pairs, 4)):
        part[name] = words[at // 4:at // 4 + 2 * count].reshape(2, count) if size == 4 else None
        at = -(-(at + 2 * count * size) // 256) * 256
    for b in range(2):
        live = bm.state[b].cpu().numpy() != 0
        both = np.pad(live, ((0, nb % 2), (0, 0))).reshape(pairs, 2, nb).any(axis=1)
        for name, cnt in (("fwd", live.sum(axis=1)), ("bwd", live.sum(axis=0)), ("pair", both.sum(axis=1))):
            assert np.array_equal(part[name + "_cnt"][b], cnt), name
            assert np.array_equal(part[name + "_order"][b], np.argsort(-cnt, kind="stable")), name
