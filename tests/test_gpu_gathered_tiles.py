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


@pytest.mark.parametrize("t", [97, 128, 700, 1500, 2047])
@pytest.mark.parametrize("classes", [5, 40, 300])
def test_stretches_of_classes_that_change_inside_documents(t, classes):
    """Row and column classes with borders of their own, some of them no class, and few documents: the stretches that count are those of the
    row class; the backward over them agrees with the dense mask in 64 bits (gradients are bf16, their sums of bf16 products)."""
    from oracle import masks as om
    from tagseq2tagseq_b200 import build_block_map, read_status
    from tagseq2tagseq_b200.attention import masked_attn
    rng = np.random.default_rng(t + classes)
    def ids(n):
        cuts = np.sort(rng.choice(np.arange(1, t), min(n, t) - 1, replace=False))
        return np.repeat(rng.permutation(min(n, t)), np.diff(np.concatenate([[0], cuts, [t]]))).astype(np.int32)
    doc, row, col = ids(max(2, classes // 8)), ids(classes), ids(classes)
    row[row % 7 == 3] = -1
    col[col % 5 == 2] = -1
    r, w = max(1, classes), -(-max(1, classes) // 64)
    bits = rng.random((r, 64 * w)) < 0.1
    link = np.array([[int(np.packbits(bits[i, 64 * j:64 * j + 64], bitorder="little").view(np.int64)[0]) for j in range(w)] for i in range(r)], np.int64)
    dense = om.class_mask_dense(doc, row, col, link)
    dev = [torch.from_numpy(x)[None].cuda() for x in (doc, link, row, col)]
    plan, nb = build_block_map(*dev).plan, (t + 127) // 128
    ok = np.zeros((128 * nb, 128 * nb), bool)
    ok[:t, :t] = _before_causality(doc, row, col, link)
    low = np.tril(np.ones((nb, nb), bool))
    live, full = ok.reshape(4 * nb, 32, nb, 128).any(axis=(1, 3)) & low.repeat(4, axis=0), ok.reshape(nb, 128, nb, 128).all(axis=(1, 3)) & np.tril(low, -1)
    runs = _plan_part(plan, 1, nb, "run_cnt").view(np.int32)[0]
    for kb in np.flatnonzero(runs > 8):
        live[:, kb] = live[:, kb].reshape(nb, 4).any(axis=1).repeat(4) & (np.arange(4 * nb) * 32 < t)
    _check_lines(plan, 0, 1, nb, live, full)
    g = torch.Generator(device="cuda").manual_seed(t)
    q, k, v, do = (torch.randn(1, 2, t, 64, device="cuda", generator=g).bfloat16() for _ in range(4))
    qd, kd, vd = (x.clone().requires_grad_(True) for x in (q, k, v))
    out, _ = masked_attn(qd, kd, vd, dev[0], dev[1], q_row_ids=dev[2], kv_col_ids=dev[3], plan=plan)
    out.backward(do)
    assert read_status(plan) == 0
    q6, k6, v6 = (x.double().requires_grad_(True) for x in (q, k, v))
    s = (q6 @ k6.transpose(-1, -2) / 8).masked_fill(~torch.from_numpy(dense).cuda(), float("-inf"))
    (torch.softmax(s, -1) @ v6).backward(do.double())
    for got, want in ((qd.grad, q6.grad), (kd.grad, k6.grad), (vd.grad, v6.grad)):
        assert (got.double() - want).norm() <= 1e-2 * want.norm()


def _before_causality(doc, row, col, link):
    """[T, T] of who may read whom, above the diagonal as well: the pre-pass leaves causality inside the diagonal tile to its readers."""
    table = np.zeros((link.shape[0] + 1, 64 * link.shape[1] + 1), bool)
    table[:-1, :-1] = np.unpackbits(link.view(np.uint8), axis=1, bitorder="little").astype(bool)
    return (doc[:, None] == doc[None]) | table[row][:, col]


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
