"""Branches of the pre-pass that sizes choose."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [128 * 32 + 1, 128 * 257])
def test_lists_of_more_tiles_than_one_sweep(t):
    """More than 32 tiles (a block of the ordering) and more than 256 (a sweep of the lists): every list is what the states say."""
    from tagseq2tagseq_b200 import build_block_map
    nb = -(-t // 128)
    doc = torch.from_numpy((np.arange(t) // 700).astype(np.int32))[None].cuda()
    bm = build_block_map(doc, with_lists=True)
    state = bm.state[0].cpu().numpy()
    outs = [x[0].cpu().numpy() for x in (bm.kv_cnt, bm.kv_idx, bm.full_cnt, bm.full_idx, bm.q_cnt, bm.q_idx, bm.full_q_cnt, bm.full_q_idx)]
    for (cnt, idx), s in zip(zip(outs[0::2], outs[1::2]), (state == 1, state == 2, (state == 1).T, (state == 2).T)):
        for line in range(nb):
            want = np.flatnonzero(s[line])
            assert cnt[line] == want.size and np.array_equal(idx[line, :want.size], want) and (idx[line, want.size:] == -1).all()
