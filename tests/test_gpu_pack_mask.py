"""Native mask construction against the host functions it restates, and the link scan on both sides of the length up to
which the tokens come back together with the candidates."""
import numpy as np
import pytest
import torch

import _synthvocab as sv
from oracle import link_detect as old

pytestmark = pytest.mark.gpu


def _spread(bounds, ids, t):
    out = np.full(t, -1, dtype=np.int32)
    for j in range(len(ids)):
        out[max(0, bounds[j]):max(0, bounds[j + 1])] = ids[j]  # positions before the sequence grant nothing of their own
    return out


@pytest.mark.parametrize("seed", range(16))
def test_pack_mask_equals_the_host_functions(seed):
    from tagseq2tagseq_b200 import DocSpan, from_reference
    from tagseq2tagseq_b200 import mask_spec as ms
    rng = np.random.default_rng(seed)
    t = int(rng.integers(1, 900))
    n = int(rng.integers(0, 70))
    cuts = np.sort(rng.integers(-20, t + 40, n + 1))
    spans = [DocSpan(int(rng.integers(0, max(1, n // 2))) if seed % 4 == 3 else i, "", int(cuts[i]), int(cuts[i + 1])) for i in range(n)]
    if seed % 2:
        rng.shuffle(spans)                                                 # out of order, ids repeated: the first span of an id is the target
    if seed % 5 == 4:
        spans.append(DocSpan(99, "", t // 3, t // 2))                      # overlaps: the last span owns the token
    links = {int(p): [int(x) for x in rng.integers(0, n + 3, rng.integers(1, 4))] for p in rng.integers(-5, t + 10, int(rng.integers(0, 200)))}
    for cap in (0, 1, 65, 500):
        got = from_reference(spans, links, t, max_grants_cap=cap, device=torch.device("cuda"))
        assert np.array_equal(got.doc_ids[0].cpu().numpy(), ms.build_document_ids(t, spans))
        grants = ms.ordered_grants(t, spans, links, cap)
        if not grants:
            assert got.link_bits is None and got.q_row_ids is None and got.kv_col_ids is None
            continue
        (qb, qi), (kb, ki), link = ms.grant_segments(grants)
        assert np.array_equal(got.link_bits[0].cpu().numpy(), link)
        assert np.array_equal(got.q_row_ids[0].cpu().numpy(), _spread(qb, qi, t))
        assert np.array_equal(got.kv_col_ids[0].cpu().numpy(), _spread(kb, ki, t))


@pytest.mark.parametrize("t,dtype", [(65536, torch.int64), (65537, torch.int64), (65537, torch.int32)])
def test_link_scan_around_the_length_whose_tokens_come_along(t, dtype):
    import random
    from tagseq2tagseq_b200.link_detect import MarkdownLinkDetector
    toks = sv.random_stream(random.Random(t), t, 50)
    det = MarkdownLinkDetector(sv.decode, window_tokens=50, link_start_token_ids=sv.STARTS, link_mid_token_id=sv.MID, vocab_size=len(sv.VOCAB))
    ids = torch.tensor(toks, dtype=dtype, device="cuda")
    assert det.candidates(ids) == old.candidates(toks, sv.decode, mid_id=sv.MID, start_ids=sv.STARTS, window=50)
    assert [tuple(x) for x in det.detect_links(ids)] == [tuple(x) for x in old.detect_links(toks, sv.decode, sv.MID, sv.STARTS, 50)]


@pytest.mark.parametrize("tiles", [1, 255, 257, 1026])
def test_plan_orders_are_heaviest_first_over_many_tiles(tiles):
    """The launch orders, whose ranks are counted 1024 tiles at a time: permutations by descending count."""
    from tagseq2tagseq_b200 import build_block_map
    doc = (torch.arange(tiles * 128 - 5, device="cuda", dtype=torch.int32) // 333)[None]
    bm = build_block_map(doc, with_lists=True)
    cnt = (bm.kv_cnt + bm.full_cnt)[0]
    plan, nb = bm.plan, tiles
    align = lambda x: (x + 255) // 256 * 256
    off = align(256)
    for size in (nb * 4, nb * 128 * 16, nb * nb, nb * 4, nb * nb * 4, nb * 4, nb * nb * 4):
        off = align(off + size)
    order = plan[off:off + 4 * nb].view(torch.int32)
    assert torch.equal(order.sort().values, torch.arange(nb, device="cuda", dtype=torch.int32))
    ranked = cnt[order.long()]
    assert bool((ranked[:-1] >= ranked[1:]).all())


@pytest.mark.parametrize("t,d,median,lo", [(640, 64, 16, 12), (1300, 128, 9, 1), (65664, 64, 300, 40)])
def test_attention_where_tiles_leave_the_mask_table(t, d, median, lo):
    """Tiles of exactly eight, nine and many runs, and a sequence of more tiles than the table covers (513), forward and
    backward, against fp64 rows computed for a sample of the queries and, through V = dO = one-hot sums, all keys."""
    from tagseq2tagseq_b200 import build_block_map, read_status, synth
    from tagseq2tagseq_b200.attention import masked_attn
    dev = torch.device("cuda")
    pack = synth.make_pack(t, t, median, lo, max(4 * median, lo), p_link=0.3)
    doc = torch.from_numpy(pack.doc_ids).to(dev)
    link = torch.from_numpy(pack.link_bits).to(dev)
    g = torch.Generator(device=dev).manual_seed(1)
    q, k, v, do = (torch.randn(1, 1, t, d, device=dev, generator=g).bfloat16() for _ in range(4))
    rows = torch.randperm(t, device=dev, generator=g)[:200]
    keep = torch.zeros(t, dtype=torch.bool, device=dev)
    keep[rows] = True
    do[:, :, ~keep] = 0                                    # only the sampled rows send a gradient back
    qd, kd, vd = (x.clone().requires_grad_(True) for x in (q, k, v))
    bm = build_block_map(doc[None], link[None])
    out, lse = masked_attn(qd, kd, vd, doc[None], link[None], plan=bm.plan)
    out.backward(do)
    assert read_status(bm.plan) == 0
    words = link[doc[rows].long()]
    bits = (torch.gather(words, 1, (doc >> 6).long()[None].expand(rows.numel(), -1)) >> (doc & 63).long()[None]) & 1
    ok = ((doc[rows][:, None] == doc[None]) | bits.bool()) & (torch.arange(t, device=dev)[None] <= rows[:, None])
    s = ((q[0, 0, rows].double() @ k[0, 0].double().T) * d ** -0.5).masked_fill(~ok, float("-inf"))
    p = torch.softmax(s, -1)
    ref = p @ v[0, 0].double()
    dor = do[0, 0, rows].double()
    ds = p * (dor @ v[0, 0].double().T - (dor * ref).sum(-1, keepdim=True)) * d ** -0.5
    # the operator's tolerances: out 2e-2, lse 1e-2, gradients 1e-2 relative
    assert (out[0, 0, rows].double() - ref).abs().max().item() <= 2e-2
    assert (lse[0, 0, rows].double() - torch.logsumexp(s, -1)).abs().max().item() <= 1e-2
    for got, want in ((qd.grad[0, 0, rows], ds @ k[0, 0].double()), (kd.grad[0, 0], ds.T @ q[0, 0, rows].double()), (vd.grad[0, 0], p.T @ dor)):
        assert ((got.double() - want).norm() / want.norm()).item() <= 1e-2
