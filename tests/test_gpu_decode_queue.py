"""The decoding step where a block's warps share one queue of keys: around the cache length at which they begin to (64 groups of 32 keys a block), one
round and several, and keys without weight whose values are infinite."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(q, k, v, ok, d):
    s = ((k.double() @ q.double().transpose(1, 2))[..., 0] * d ** -0.5).masked_fill(~ok, float("-inf"))
    p = torch.softmax(s, -1)
    return (p[..., None] * torch.where(p[..., None] > 0, v.double(), 0.0)).sum(1, keepdim=True), torch.logsumexp(s, -1)


# blocks of one per head (320 heads): 64, 65, 128 and 129 groups; clusters of eight: one round and two, three with a remainder
@pytest.mark.parametrize("b,h,tk", [(16, 20, 2048), (16, 20, 2049), (16, 20, 4096), (16, 20, 4097), (1, 1, 32768), (1, 2, 32769), (1, 1, 70001)])
@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("p_link", [0.0, 0.3])
def test_shared_queue_matches_the_masked_row(b, h, tk, d, p_link):
    from tagseq2tagseq_b200 import synth
    from tagseq2tagseq_b200.attention import masked_attn_decode
    dev = torch.device("cuda")
    doc, link = synth.stack_packs([synth.make_pack(60 + i, tk, 300, 16, tk // 2, p_link=p_link) for i in range(b)])
    doc, link = torch.from_numpy(doc).to(dev), None if link is None else torch.from_numpy(link).to(dev)
    g = torch.Generator(device=dev).manual_seed(tk + d)
    q = torch.randn(b, h, 1, d, device=dev, generator=g).bfloat16()
    k, v = (torch.randn(b, h, tk, d, device=dev, generator=g).bfloat16() for _ in range(2))
    pos = torch.randint(0, tk, (b,), device=dev, generator=g, dtype=torch.int32)
    pos[0] = 0                                                 # blocks without a group of their own
    for q_pos in (None, pos):
        out, lse = masked_attn_decode(q, k, v, doc, link, q_pos=q_pos)
        again, _ = masked_attn_decode(q, k, v, doc, link, q_pos=q_pos)
        assert torch.equal(out, again)
        for i in range(b):
            at = tk - 1 if q_pos is None else int(pos[i])
            ok = doc[i] == doc[i, at]
            if link is not None:
                ok |= ((link[i][doc[i, at].long()][(doc[i] >> 6).long()] >> (doc[i] & 63).long()) & 1).bool()
            ok &= torch.arange(tk, device=dev) <= at
            want, want_lse = _reference(q[i], k[i], v[i], ok, d)
            # one bf16 rounding of a mean of unit normals, fp32 sums of at most 70001 products
            assert (out[i].double() - want).abs().max().item() <= 2 ** -8 * max(1.0, want.abs().max().item())
            assert (lse[i].double() - want_lse).abs().max().item() <= 1e-4


@pytest.mark.parametrize("tk", [2048, 4097, 9000])
def test_keys_without_weight_add_nothing_whatever_their_values(tk):
    from tagseq2tagseq_b200.attention import masked_attn_decode
    dev, d, b, h = torch.device("cuda"), 64, 16, 20
    g = torch.Generator(device=dev).manual_seed(tk)
    q = torch.randn(b, h, 1, d, device=dev, generator=g).bfloat16()
    k, v = (torch.randn(b, h, tk, d, device=dev, generator=g).bfloat16() for _ in range(2))
    far = torch.randint(0, tk, (64,), device=dev, generator=g)
    k[:, :, far] = (-q * 2.0 ** 12).to(torch.bfloat16)         # scores of -2^12 |q|^2 / 8: their weights are zeros
    v[:, :, far] = float("inf")
    doc = torch.zeros((b, tk), dtype=torch.int32, device=dev)
    out, lse = masked_attn_decode(q, k, v, doc)
    for i in (0, b - 1):
        want, want_lse = _reference(q[i], k[i], v[i], torch.ones(tk, dtype=torch.bool, device=dev), d)
        assert (out[i].double() - want).abs().max().item() <= 2 ** -8 * max(1.0, want.abs().max().item())
        assert (lse[i].double() - want_lse).abs().max().item() <= 1e-4


# one block an SM or two: 148 blocks and 149, 128 in clusters of two and of four and a few more, 96 and 104 in clusters of eight; own keys and a shared queue
@pytest.mark.parametrize("b,h,tk", [(4, 37, 1000), (1, 149, 1000), (4, 37, 2100), (1, 149, 2100), (4, 16, 3000), (5, 13, 3000), (2, 16, 7000), (3, 11, 7000), (1, 12, 17000), (1, 13, 17000), (1, 12, 33000), (1, 13, 33000)])
@pytest.mark.parametrize("d", [64, 128])
def test_one_or_two_blocks_an_sm_give_the_same(b, h, tk, d):
    from tagseq2tagseq_b200 import synth
    from tagseq2tagseq_b200.attention import masked_attn_decode
    dev = torch.device("cuda")
    doc, link = synth.stack_packs([synth.make_pack(7 + i, tk, 300, 16, tk // 2, p_link=0.3) for i in range(b)])
    doc, link = torch.from_numpy(doc).to(dev), torch.from_numpy(link).to(dev)
    g = torch.Generator(device=dev).manual_seed(tk + d)
    q = torch.randn(b, h, 1, d, device=dev, generator=g).bfloat16()
    k, v = (torch.randn(b, h, tk, d, device=dev, generator=g).bfloat16() for _ in range(2))
    out, lse = masked_attn_decode(q, k, v, doc, link)
    for i in range(b):
        ok = (doc[i] == doc[i, -1]) | ((link[i][doc[i, -1].long()][(doc[i] >> 6).long()] >> (doc[i] & 63).long()) & 1).bool()
        want, want_lse = _reference(q[i], k[i], v[i], ok, d)
        # one bf16 rounding of a mean of unit normals, fp32 sums of at most 33000 products
        assert (out[i].double() - want).abs().max().item() <= 2 ** -8 * max(1.0, want.abs().max().item())
        assert (lse[i].double() - want_lse).abs().max().item() <= 1e-4
