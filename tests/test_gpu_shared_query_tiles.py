"""Short launches of the forward, where the two teams of a block share a query tile, against the dense mask in fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# tiles of one list (none shared, one each, one and two ...); all items at once and one more; pairs at once from 32 tiles on, and one fewer
@pytest.mark.parametrize("b,h,t", [(1, 1, 1), (2, 2, 127), (1, 3, 200), (2, 3, 385), (1, 4, 1024), (1, 9, 2048), (2, 37, 256), (2, 37, 257), (4, 8, 600),
                                   (1, 2, 9472), (1, 2, 9473), (1, 9, 4096), (1, 9, 3968), (1, 9, 4097)])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("kind", ["causal", "documents", "linked", "linked, packed"])
def test_forward_of_short_launches(b, h, t, d, kind):
    """Both parts of a shared tile have to come in with their own weight.  The bounds are those of the arithmetic, per row: a score is a sum of D
    products of about 0.64 in fp32 and its scaled size adds up to less than 8 D units of 2^-24, the row's sum adds its keys one by one
    in fp32; P and the result are rounded to bf16's eight bits (by 2^-8 of their size at most, P's error weighted by |V|)."""
    from tagseq2tagseq_b200 import build_block_map, read_status, synth
    from tagseq2tagseq_b200.attention import masked_attn
    dev = torch.device("cuda")
    g = torch.Generator(device=dev).manual_seed(t + d)
    doc, link = torch.zeros((b, t), dtype=torch.int32, device=dev), None
    if kind != "causal":
        doc, link = synth.stack_packs([synth.make_pack(s + 1, t, 150, min(16, t), max(600, t // 8), p_link=0.3 if "linked" in kind else 0.0) for s in range(b)])
        doc, link = torch.from_numpy(doc).to(dev), None if link is None else torch.from_numpy(link).to(dev)
    q, k, v = (torch.randn(b, h, t, d, device=dev, generator=g).bfloat16() for _ in range(3))
    if "packed" in kind:                                       # views of one [B, T, 3, H, D] projection
        q, k, v = torch.stack([x.transpose(1, 2) for x in (q, k, v)], dim=2).transpose(1, 3).unbind(2)
    plan = build_block_map(doc, link).plan
    out, lse = masked_attn(q, k, v, doc, link, plan=plan)
    assert read_status(plan) == 0
    for i in range(b):
        ok = doc[i][:, None] == doc[i][None]
        if link is not None:
            words = link[i][doc[i].long()]                                     # [t, W]: what row t's document may read
            ok |= ((torch.gather(words, 1, (doc[i] >> 6).long()[None].expand(t, -1)) >> (doc[i] & 63).long()[None]) & 1).bool()
        ok &= torch.ones(t, t, dtype=torch.bool, device=dev).tril()
        for j in sorted({0, h // 2, h - 1}):
            s = ((q[i, j].double() @ k[i, j].double().T) * d ** -0.5).masked_fill(~ok, float("-inf"))
            want, p = torch.logsumexp(s, -1), torch.softmax(s, -1)
            off = 2.0 ** -23 * (ok.sum(-1) + 8 * d + want.abs())
            assert ((lse[i, j].double() - want).abs() <= off).all()
            size, want = p @ v[i, j].double().abs(), p @ v[i, j].double()
            assert ((out[i, j].double() - want).abs() <= 2.0 ** -8 * (size + want.abs()) + 2 * off[:, None] * size).all()
    again, _ = masked_attn(q, k, v, doc, link, plan=plan)
    assert torch.equal(out, again)


@pytest.mark.parametrize("t,few,many", [(506, 2, 75), (1024, 4, 38), (2048, 8, 20)])
@pytest.mark.parametrize("d", [64, 128])
def test_sharing_a_query_tile_costs_no_precision(t, few, many, d):
    """The same heads in a launch that shares query tiles and in one that has a team add up a row alone, against 64 bits: the split is no
    further off, neither in the row sums nor in the result (five seeds together: what one rounding more or less decides averages out)."""
    from tagseq2tagseq_b200 import build_block_map
    from tagseq2tagseq_b200.attention import masked_attn
    dev = torch.device("cuda")
    doc = torch.zeros((1, t), dtype=torch.int32, device=dev)
    plan, off = build_block_map(doc).plan, torch.zeros(2, 2, dtype=torch.float64, device=dev)
    for seed in range(5):
        g = torch.Generator(device=dev).manual_seed(seed)
        q, k, v = (torch.randn(1, many, t, d, device=dev, generator=g).bfloat16() for _ in range(3))
        s = ((q[:, :few].double() @ k[:, :few].double().transpose(-1, -2)) * d ** -0.5).masked_fill(~torch.ones(t, t, dtype=torch.bool, device=dev).tril(), float("-inf"))
        want, want_lse = torch.softmax(s, -1) @ v[:, :few].double(), torch.logsumexp(s, -1)
        for i, n in enumerate((few, many)):
            out, lse = masked_attn(q[:, :n], k[:, :n], v[:, :n], doc, plan=plan)
            off[i] += torch.stack([(lse[:, :few].double() - want_lse).square().sum(), (out[:, :few].double() - want).square().sum()])
    assert (off[0] <= off[1]).all(), (off[0] / off[1]).sqrt().tolist()


# around 32 tiles and the most pairs and tiles that run at once (148 SMs): one and several elements, one head (whose tiles never all run at
# once at that length, so that only the pairs' bits are to be had) and several
@pytest.mark.parametrize("kind,b,h,t", [(k, *s) for k in ("short", "long") for s in ((1, 9, 4096), (1, 9, 3969), (3, 3, 4096), (1, 2, 18900))] + [("short", 1, 1, 37800)])
@pytest.mark.parametrize("d", [64, 128])
def test_the_form_of_middle_launches_follows_the_lists(b, h, t, d, kind):
    """All pairs run at once but not all tiles: short lists keep pairs of query tiles, which they are faster with, long ones share tiles.  The
    two forms round differently, so the bits tell which ran: those of the same heads among more than run at once as pairs, or among as few
    as run at once as tiles."""
    from tagseq2tagseq_b200 import build_block_map, read_status, synth
    from tagseq2tagseq_b200.attention import masked_attn
    dev = torch.device("cuda")
    tiles, pairs, sms = -(-t // 128), -(-t // 256), torch.cuda.get_device_properties(0).multi_processor_count
    assert b * h * pairs <= sms < b * h * tiles
    other = sms // (b * tiles) if kind == "long" else sms // (b * pairs) + 1
    doc = torch.zeros((b, t), dtype=torch.int32, device=dev)
    if kind == "short":
        doc = torch.from_numpy(synth.stack_packs([synth.make_pack(s + 1, t, 60, 16, 200) for s in range(b)])[0]).to(dev)
    g = torch.Generator(device=dev).manual_seed(t)
    q, k, v = (torch.randn(b, max(h, other), t, d, device=dev, generator=g).bfloat16() for _ in range(3))
    plan, n = build_block_map(doc).plan, min(h, other)
    out, lse = masked_attn(q[:, :h], k[:, :h], v[:, :h], doc, plan=plan)
    want, want_lse = masked_attn(q[:, :other], k[:, :other], v[:, :other], doc, plan=plan)
    assert read_status(plan) == 0
    assert torch.equal(out[:, :n], want[:, :n]) and torch.equal(lse[:, :n], want_lse[:, :n])
    again, _ = masked_attn(q[:, :h], k[:, :h], v[:, :h], doc, plan=plan)
    assert torch.equal(out, again)


@pytest.mark.parametrize("kind", ["short", "long"])
def test_a_refused_plan_serves_its_own_call_afterwards(kind):
    """Blocks of a middle launch that have no item leave early: not before the plan's stamp is looked at, or a plan of another call would keep
    a part of their count and start its own next launch with it."""
    from tagseq2tagseq_b200 import build_block_map, read_status, synth
    from tagseq2tagseq_b200.attention import masked_attn
    dev, h = torch.device("cuda"), 8
    doc = torch.zeros((1, 4224), dtype=torch.int32, device=dev)
    if kind == "short":
        doc = torch.from_numpy(synth.stack_packs([synth.make_pack(1, 4224, 60, 16, 200)])[0]).to(dev)
    g = torch.Generator(device=dev).manual_seed(1)
    q, k, v = (torch.randn(1, h, 4224, 64, device=dev, generator=g).bfloat16() for _ in range(3))
    plan = build_block_map(doc).plan
    want, _ = masked_attn(q, k, v, doc, plan=plan)
    masked_attn(*(x[:, :, :4096] for x in (q, k, v)), doc[:, :4096].contiguous(), plan=plan)
    assert read_status(plan) == 1900 and plan.view(torch.int32)[8:10].tolist() == [0, 0]
    for _ in range(3):
        out, _ = masked_attn(q, k, v, doc, plan=plan)
        assert torch.equal(out, want) and plan.view(torch.int32)[8:10].tolist() == [0, 0]
