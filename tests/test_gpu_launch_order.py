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


def _step(inputs, wait):
    """What a training loop has follow one another: tokens and targets written on the device, the mask from them, a head with a scaled loss, its gradients copied, an optimizer
    step on them and the weights' copies for the next."""
    from tagseq2tagseq_b200 import CrossDocLinkMaskCreator, DocSpan
    from tagseq2tagseq_b200.link_detect import MarkdownLinkDetector
    from tagseq2tagseq_b200.lm_fused import AdamW, Linear, cast_weights, copy_tensors, embedding, head_loss
    plain, link_at, h, weight = inputs
    n, v = plain.numel(), weight.shape[0]
    text = {1: "[", 2: "](", 3: ")"}
    detector = MarkdownLinkDetector(lambda ids: "".join(text.get(i, "w%d" % i) for i in ids), window_tokens=8, link_start_token_ids=(1,), link_mid_token_id=2, vocab_size=64)
    spans = [DocSpan(i, "", i * n // 4, (i + 1) * n // 4, False, [], "w%d" % (10 + i)) for i in range(4)]
    creator = CrossDocLinkMaskCreator(detector)
    with torch.device(plain.device):
        head = Linear(h.shape[1], v)
        table = torch.nn.Parameter(weight[:64].clone())
    with torch.no_grad():
        head.weight.copy_(weight)
    opt = AdamW([head.weight, table], lr=0.1)
    copies, out = [c for c in cast_weights([head.weight, table])], []

    def done(*ts):
        if wait:
            torch.cuda.synchronize()
        out.extend(t.detach().clone() for t in ts)

    for step in range(3):
        tokens = plain.clone()
        for k, tok in enumerate((1, 20, 2, 10 + step % 3, 3)):   # a link in the last document, written just before the scan
            tokens[link_at + k] = tok
        spec = creator(tokens[None], spans)
        done(spec.doc_ids, *(t for t in (spec.link_bits, spec.q_row_ids, spec.kv_col_ids) if t is not None), spec.block_map(with_lists=True).state)
        x = (h + embedding(table, tokens).repeat(1, h.shape[1] // table.shape[1])).bfloat16()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = head_loss(x, head.weight, tokens, copies[0])
        done(loss)
        grads = torch.autograd.grad(3.0 * loss, (head.weight, table))
        kept = [torch.empty_like(g) for g in grads]
        copy_tensors(kept, grads)
        del grads                                                # their memory is the next allocation's
        head.weight.grad, table.grad = kept
        opt.step()
        copies = cast_weights([head.weight, table])
        done(*kept, head.weight, table, *copies)
    return out


@pytest.mark.parametrize("n,c,v", [(64, 64, 64), (1000, 256, 4096), (5000, 128, 1024)])
def test_a_loop_of_steps_back_to_back(n, c, v):
    dev, sets = torch.device("cuda"), []
    for seed in range(2):
        g = torch.Generator(device=dev).manual_seed(10 + seed)
        weight = torch.randn(v, c, device=dev, generator=g) * 0.05
        sets.append((torch.randint(20, 60, (n,), device=dev, generator=g), n - 8, torch.randn(n, c, device=dev, generator=g), weight))
    want = [_step(s, True) for s in sets]
    torch.cuda.synchronize()
    for i in range(6):
        for k, (a, b) in enumerate(zip(_step(sets[i % 2], False), want[i % 2], strict=True)):
            assert torch.equal(a, b), (i, k)
