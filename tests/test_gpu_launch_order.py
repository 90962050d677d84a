"""Every kernel may start before the writes of the one before it are visible, and waits for them: chains of dependent calls on buffers that
are used again at once give what the same calls give with the device idle between them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(inputs, wait):
    from tagseq2tagseq_b200 import MaskSpec
    from tagseq2tagseq_b200.attention import masked_attn, masked_attn_decode
    from tagseq2tagseq_b200.lm_fused import add_rmsnorm, cross_entropy, embedding, qkv_attention, rope_half_tables, swiglu
    table, tokens, w, doc, link, target = inputs
    table = table.detach().requires_grad_(True)
    n, c = tokens.numel(), table.shape[1]
    out = []

    def done(*ts):
        if wait:
            torch.cuda.synchronize()
        out.extend(t.detach().clone() for t in ts)
        return ts[0] if len(ts) == 1 else ts

    spec = MaskSpec(doc, link)
    x = done(embedding(table, tokens))
    x2, h = done(*add_rmsnorm(x, None, w, 1e-6))
    qkv = h.view(1, n, c)[..., :192].clone(memory_format=torch.contiguous_format)
    cos, sin = rope_half_tables(n, 64, 1e4, x.device)
    a = done(qkv_attention(qkv, cos, sin, spec, 1, 64)).view(n, 64)
    q = a.detach().view(1, n, 1, 64).permute(0, 2, 1, 3)
    done(*masked_attn_decode(q[:, :, -1:].contiguous(), q, q, doc, link))
    done(*masked_attn(q, q, q, doc, link, plan=spec.plan))
    act = done(swiglu(h))
    x3, h3 = done(*add_rmsnorm(x2, torch.cat([act, act], -1) + a.repeat(1, c // 64), w, 1e-6))
    loss = done(cross_entropy(h3.clone(), target))
    done(torch.autograd.grad(loss + x3.square().mean(), table)[0])
    return out


@pytest.mark.parametrize("n,c", [(1, 256), (257, 256), (1000, 768), (700, 4352)])
def test_dependent_calls_back_to_back(n, c):
    from tagseq2tagseq_b200 import synth
    dev, sets = torch.device("cuda"), []
    for seed in range(2):                                     # two sets of inputs in turn: nothing of one fits the other
        g = torch.Generator(device=dev).manual_seed(seed)
        doc, link = synth.stack_packs([synth.make_pack(seed, n, 100, min(8, n), 300, p_link=0.3)])
        sets.append((torch.randn(300, c, device=dev, generator=g), torch.randint(0, 300, (n,), device=dev, generator=g), torch.rand(c, device=dev, generator=g) + 0.5,
                     torch.from_numpy(doc).to(dev), None if link is None else torch.from_numpy(link).to(dev), torch.randint(0, c, (n,), device=dev, generator=g)))
    want = [_chain(s, True) for s in sets]
    torch.cuda.synchronize()
    got = [_chain(sets[i % 2], False) for i in range(8)]
    for i, outs in enumerate(got):
        for k, (a, b) in enumerate(zip(outs, want[i % 2])):
            if k < len(outs) - 1:
                assert torch.equal(a, b), (i, k)
            else:                                             # dq of the attention is added up in the order of arrival, in fp32, and rounded to bf16
                assert (a - b).norm() <= 2 ** -9 * b.norm()
