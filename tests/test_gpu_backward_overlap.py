"""The backward's three launches overlap in short calls: repeated calls over one workspace's worth of reused memory, around the size from
which they run one after the other, give what a call alone gives."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,t,d", [(1, 1, 64), (2, 129, 128), (8, 600, 64), (12, 4096, 128), (12, 4097, 128), (12, 8192, 64), (12, 8193, 64)])
def test_back_to_back_calls_agree(h, t, d):
    """dk and dv are the same bits every time.  dq, added up in an order that varies, stays within the rounding of its fp32 sums and
    one step of bf16; a call that read statistics or zeros of the one before would be off by as much as the gradients differ."""
    from tagseq2tagseq_b200 import build_block_map, read_status, synth
    from tagseq2tagseq_b200.attention import _attn_bwd, _attn_fwd
    dev = torch.device("cuda")
    doc, link = synth.stack_packs([synth.make_pack(5, t, 150, min(16, t), 600, p_link=0.2)])
    doc, link = torch.from_numpy(doc).to(dev), torch.from_numpy(link).to(dev)
    plan = build_block_map(doc, link).plan
    g = torch.Generator(device=dev).manual_seed(t)
    calls = []
    for _ in range(2):                                        # two sets of inputs in turn: nothing of one call fits the next
        q, k, v, do = (torch.randn(1, h, t, d, device=dev, generator=g).bfloat16() for _ in range(4))
        out, lse = _attn_fwd(q, k, v, doc, link, None, None, plan, d ** -0.5)
        calls.append((q, k, v, out, do, lse, doc, link, None, None, plan, d ** -0.5))
    alone = []
    for c in calls:
        alone.append(_attn_bwd(*c))
        torch.cuda.synchronize()
    rest = [_attn_bwd(*calls[i % 2]) for i in range(12)]
    assert read_status(plan) == 0
    for i, (dq, dk, dv) in enumerate(rest):
        want = alone[i % 2]
        assert torch.equal(dk, want[1]) and torch.equal(dv, want[2])
        assert ((dq.float() - want[0].float()).abs() / want[0].float().abs().clamp_min(1e-2)).max().item() <= 2 ** -6


def test_calls_on_two_streams_agree():
    """Short backwards on two streams at once, each with a plan and inputs of its own: what either overlaps with is its own stream's launch."""
    from tagseq2tagseq_b200 import build_block_map, read_status, synth
    from tagseq2tagseq_b200.attention import _attn_bwd, _attn_fwd
    dev, calls = torch.device("cuda"), []
    for seed, (h, t, d) in enumerate([(4, 900, 64), (2, 1500, 128)]):
        doc, link = synth.stack_packs([synth.make_pack(seed + 1, t, 150, 16, 600, p_link=0.2)])
        doc, link = torch.from_numpy(doc).to(dev), torch.from_numpy(link).to(dev)
        plan = build_block_map(doc, link).plan
        g = torch.Generator(device=dev).manual_seed(seed)
        q, k, v, do = (torch.randn(1, h, t, d, device=dev, generator=g).bfloat16() for _ in range(4))
        out, lse = _attn_fwd(q, k, v, doc, link, None, None, plan, d ** -0.5)
        calls.append((q, k, v, out, do, lse, doc, link, None, None, plan, d ** -0.5))
    alone = [_attn_bwd(*c) for c in calls]
    torch.cuda.synchronize()
    streams, got = [torch.cuda.Stream() for _ in calls], [[], []]
    for _ in range(20):
        for i, c in enumerate(calls):
            with torch.cuda.stream(streams[i]):
                got[i].append(_attn_bwd(*c))
    torch.cuda.synchronize()
    for i, c in enumerate(calls):
        assert read_status(c[10]) == 0
        for dq, dk, dv in got[i]:
            assert torch.equal(dk, alone[i][1]) and torch.equal(dv, alone[i][2])
            assert ((dq.float() - alone[i][0].float()).abs() / alone[i][0].float().abs().clamp_min(1e-2)).max().item() <= 2 ** -6
