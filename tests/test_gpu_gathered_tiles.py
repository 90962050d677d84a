"""The query tiles that the backward walks: stretches of 32 rows gathered by the pre-pass, against the dense mask."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _plan_part(plan, B, nb, name):
    """A table of the block plan by the layout of csrc/plan.h."""
    pairs, tri, at = (nb + 1) // 2, nb * (nb + 1) // 2, 256
    for part, size in (("run_cnt", nb * 4), ("runs", nb * 128 * 16), ("state", nb * nb), ("fwd_cnt", nb * 4), ("fwd_idx", nb * nb * 4), ("bwd_cnt", nb * 4),
                       ("bwd_idx", nb * nb * 4), ("fwd_order", nb * 4), ("bwd_order", nb * 4), ("pair_cnt", pairs * 4), ("pair_order", pairs * 4),
                       ("link_t", 1024 * 16 * 8), ("run_mask", nb * 8 * 16), ("q_mask", tri * 8 * 16), ("kv_mask", tri * 4 * 8 * 4), ("bwd_sub", tri * 4 * 2),
                       ("bwd_tiles", nb * 4)):
        if part == name:
            return plan[at:at + B * size].cpu().numpy().reshape(B, size)
        at = -(-(at + B * size) // 256) * 256
    raise KeyError(name)


def _check_lines(plan, b, B, nb, live, full):
    """live: bool [4 nb, nb], stretch against kv tile; full: bool [nb, nb].  Full q tiles, then partial ones with four live stretches, then the
    live stretches of the others."""
    sub = _plan_part(plan, B, nb, "bwd_sub").view(np.uint16)[b].reshape(-1, 4)
    tiles = _plan_part(plan, B, nb, "bwd_tiles").view(np.int32)[b]
    at = 0
    for kb in range(nb):
        four = live[:, kb].reshape(nb, 4).all(axis=1)
        assert not (full[:, kb] & ~four).any()
        whole, four = full[:, kb].repeat(4), (four & ~full[:, kb]).repeat(4)
        want = np.concatenate([np.flatnonzero(whole) | 0x8000, np.flatnonzero(four), np.flatnonzero(live[:, kb] & ~whole & ~four)])
        want = np.concatenate([want, np.full(-want.size % 4, 4 * nb)]).reshape(-1, 4)
        assert tiles[kb] == len(want) and np.array_equal(sub[at:at + len(want)], want), kb
        at += nb - kb
    order = _plan_part(plan, B, nb, "bwd_order").view(np.int32)[b]
    assert np.array_equal(order, np.argsort(-tiles, kind="stable"))       # most of these tiles first, ties by number


@pytest.mark.parametrize("t", [1, 31, 32, 33, 96, 97, 128, 129, 700, 2047])
@pytest.mark.parametrize("median,lo", [(40, 1), (300, 40)])
def test_stretches_against_the_dense_mask(t, median, lo):
    from oracle import masks as om
    from tagseq2tagseq_b200 import build_block_map, synth
    packs = [synth.make_pack(s, t, median, min(lo, t), max(4 * median, lo), p_link=0.2) for s in (1, 2)]
    doc, link = (torch.from_numpy(x).cuda() for x in synth.stack_packs(packs))
    plan, nb = build_block_map(doc, link).plan, (t + 127) // 128
    for b, pack in enumerate(packs):
        ok = np.zeros((128 * nb, 128 * nb), bool)
        ok[:t, :t] = om.class_mask_dense(pack.doc_ids, None, None, pack.link_bits)
        cells = ok.reshape(4 * nb, 32, nb, 128)
        live, full = cells.any(axis=(1, 3)), ok.reshape(nb, 128, nb, 128).all(axis=(1, 3))
        runs = _plan_part(plan, 2, nb, "run_cnt").view(np.int32)[b]
        for kb in np.flatnonzero(runs > 8):  # tiles of more than eight runs: every stretch of a partial tile counts as live
            live[:, kb] = live[:, kb].reshape(nb, 4).any(axis=1).repeat(4) & (np.arange(4 * nb) * 32 < t)
        _check_lines(plan, b, 2, nb, live, full)


@pytest.mark.parametrize("nb", [31, 32, 33, 64, 65, 128, 129, 255, 511, 512])
def test_stretches_of_long_sequences(nb):
    """Around the tiles of a warp's sweep, where one warp a line becomes four, and at the most that the table covers, documents alone."""
    from tagseq2tagseq_b200 import build_block_map
    t = 128 * nb - 70
    doc = torch.arange(t, device="cuda", dtype=torch.int32) // 1111
    plan = build_block_map(doc[None]).plan
    d = np.concatenate([np.arange(t) // 1111, np.full(70, 1 << 30)])
    lo, hi = d.reshape(-1, 32).min(axis=1), np.where(d < 1 << 30, d, -1).reshape(-1, 32).max(axis=1)
    whole = d.reshape(-1, 32).max(axis=1) < 1 << 30
    klo, khi = lo.reshape(nb, 4).min(axis=1), hi.reshape(nb, 4).max(axis=1)
    q_tile = np.arange(4 * nb)[:, None] // 4
    live = (lo[:, None] <= khi[None]) & (q_tile >= np.arange(nb)) & (hi[:, None] >= 0)
    full = (hi[:, None] == klo[None]) & (lo == hi)[:, None] & (klo == khi)[None] & whole[:, None] & (q_tile > np.arange(nb))
    full = full.reshape(nb, 4, nb).all(axis=1)
    _check_lines(plan, 0, 1, nb, live, full)
