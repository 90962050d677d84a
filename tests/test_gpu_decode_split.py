"""The decoding step where its split over warps, blocks and clusters changes: cache lengths around a group of 32 keys, around
the lengths at which a cluster grows, many and few (batch, head) pairs, queues that end in a remainder, q_pos per sequence."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,h,tk,d,p,median", [(1, 1, 1, 64, 0.0, 1), (1, 2, 31, 128, 0.0, 9), (2, 1, 33, 64, 0.5, 3), (3, 2, 1100, 128, 0.3, 40),
                                               (1, 1, 2047, 64, 0.3, 30), (1, 2, 2049, 128, 0.0, 1500), (1, 1, 4097, 128, 0.4, 60),
                                               (1, 1, 16385, 64, 0.2, 200), (16, 20, 70, 64, 0.3, 10), (2, 8, 9001, 128, 0.05, 2)])
def test_decode_matches_the_masked_row_in_fp64(b, h, tk, d, p, median):
    from tagseq2tagseq_b200 import synth
    from tagseq2tagseq_b200.attention import masked_attn_decode
    dev = torch.device("cuda")
    packs = [synth.make_pack(40 + i, tk, median, 1, max(2, tk), p_link=p) for i in range(b)] if tk < 5000 or median > 2 else \
        [synth.make_pack(40 + i, tk, 400, 1, tk, p_link=p) for i in range(b)]
    doc_np, link_np = synth.stack_packs(packs)
    doc = torch.from_numpy(doc_np).to(dev)
    link = None if link_np is None else torch.from_numpy(link_np).to(dev)
    g = torch.Generator(device=dev).manual_seed(tk)
    q = torch.randn(b, h, 1, d, device=dev, generator=g).bfloat16()
    k, v = (torch.randn(b, h, tk, d, device=dev, generator=g).bfloat16() for _ in range(2))
    pos = torch.randint(0, tk, (b,), device=dev, generator=g, dtype=torch.int32)
    for q_pos in (None, pos):
        out, lse = masked_attn_decode(q, k, v, doc, link, q_pos=q_pos)
        for i in range(b):
            at = tk - 1 if q_pos is None else int(pos[i])
            ok = doc[i] == doc[i, at]
            if link is not None:
                words = link[i][doc[i, at].long()]
                ok |= ((words[(doc[i] >> 6).long()] >> (doc[i] & 63).long()) & 1).bool()
            ok &= torch.arange(tk, device=dev) <= at
            s = (k[i].double() @ q[i].double().transpose(1, 2))[..., 0] * d ** -0.5
            s = s.masked_fill(~ok, float("-inf"))
            ref = torch.softmax(s, -1)[:, None] @ v[i].double()
            # one bf16 rounding of a mean of unit normals, fp32 sums of at most 16385 products
            assert (out[i].double() - ref).abs().max().item() <= 2 ** -8 * max(1.0, ref.abs().max().item())
            assert (lse[i].double() - torch.logsumexp(s, -1)).abs().max().item() <= 1e-4
