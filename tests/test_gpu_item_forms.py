"""The forward's choice between pairs of query tiles and shared ones where blocks compute several items, on either side of its lines, against
the dense mask in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _mask(kind, b, t, dev):
    from tagseq2tagseq_b200 import synth
    if kind == "causal":
        return torch.zeros((b, t), dtype=torch.int32, device=dev), None
    doc, link = synth.stack_packs([synth.make_pack(s + 1, t, 100, min(16, t), 300, p_link=0.3 if kind == "linked" else 0.0) for s in range(b)])
    return torch.from_numpy(doc).to(dev), None if link is None else torch.from_numpy(link).to(dev)


def _allowed(doc, link):
    t = doc.numel()
    ok = doc[:, None] == doc[None]
    if link is not None:
        words = link[doc.long()]
        ok |= ((torch.gather(words, 1, (doc >> 6).long()[None].expand(t, -1)) >> (doc & 63).long()[None]) & 1).bool()
    return ok & torch.ones(t, t, dtype=torch.bool, device=doc.device).tril()


# two or three shared tiles a block; pairs as the lists call for; the last launch that asks the lists (four pairs an SM of 148) and the first that does not; lists of one to three tiles
@pytest.mark.parametrize("b,h,t", [(1, 30, 1280), (3, 23, 1279), (1, 60, 1281), (4, 37, 1024), (4, 38, 1024), (2, 100, 384), (2, 100, 129)])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("kind", ["causal", "documents", "linked"])
def test_forward_of_blocks_with_several_items(b, h, t, d, kind):
    """Bounds of the arithmetic, per row: fp32 scores and sums (2^-24 a term), P and the result rounded to bf16 (2^-8 of their size at most, P's error
    weighted by |V|)."""
    from tagseq2tagseq_b200 import build_block_map, read_status
    from tagseq2tagseq_b200.attention import masked_attn
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(t + d)
    doc, link = _mask(kind, b, t, dev)
    q, k, v = (torch.randn(b, h, t, d, device=dev, generator=g).bfloat16() for _ in range(3))
    plan = build_block_map(doc, link).plan
    for _ in range(2):                                         # the counters that items are drawn from start again
        out, lse = masked_attn(q, k, v, doc, link, plan=plan)
        assert read_status(plan) == 0 and plan.view(torch.int32)[8:10].tolist() == [0, 0]
        for i in range(b):
            ok = _allowed(doc[i], None if link is None else link[i])
            for j in range(h):                                 # every item of the launch
                s = ((q[i, j].double() @ k[i, j].double().T) * d ** -0.5).masked_fill(~ok, float("-inf"))
                want, p = torch.logsumexp(s, -1), torch.softmax(s, -1)
                off = 2.0 ** -23 * (ok.sum(-1) + 8 * d + want.abs())
                assert ((lse[i, j].double() - want).abs() <= off).all(), (i, j)
                size, want = p @ v[i, j].double().abs(), p @ v[i, j].double()
                assert ((out[i, j].double() - want).abs() <= 2.0 ** -8 * (size + want.abs()) + 2 * off[:, None] * size).all(), (i, j)


@pytest.mark.parametrize("t,few,many", [(506, 2, 300), (1024, 4, 150), (2048, 8, 76)])
@pytest.mark.parametrize("d", [64, 128])
def test_shared_tiles_cost_no_precision_against_pairs(t, few, many, d):
    """The same heads in a launch that shares query tiles and in one that has too many pairs for that, against 64 bits: five seeds together,
    as what one rounding more or less decides averages out."""
    from tagseq2tagseq_b200 import build_block_map
    from tagseq2tagseq_b200.attention import masked_attn
    dev = torch.device("cuda")
    doc = torch.zeros((1, t), dtype=torch.int32, device=dev)
    plan, ok, off = build_block_map(doc).plan, _allowed(doc[0], None), torch.zeros(2, 2, dtype=torch.float64, device=dev)
    for seed in range(5):
        g = torch.Generator(device=dev).manual_seed(seed)
        q, k, v = (torch.randn(1, many, t, d, device=dev, generator=g).bfloat16() for _ in range(3))
        for form, n in enumerate((few, many)):
            out, lse = masked_attn(*(x[:, :n].contiguous() for x in (q, k, v)), doc, plan=plan)
            for j in range(few):
                s = ((q[0, j].double() @ k[0, j].double().T) * d ** -0.5).masked_fill(~ok, float("-inf"))
                off[form, 0] += (out[0, j].double() - torch.softmax(s, -1) @ v[0, j].double()).square().sum()
                off[form, 1] += (lse[0, j].double() - torch.logsumexp(s, -1)).square().sum()
    assert (off[0].sqrt() <= 1.05 * off[1].sqrt()).all(), off.sqrt()
