"""Many tensors copied in one launch: every byte of the right ones, at any alignment, and what one launch does not take."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


def test_every_pair_is_copied_and_nothing_else():
    from tagseq2tagseq_b200.lm_fused import copy_tensors
    g = torch.Generator(device=DEV).manual_seed(1)
    draw = lambda n, dtype: torch.randint(-2**31, 2**31 - 1, (n,), device=DEV, generator=g).to(torch.int32).view(torch.uint8)[:n * dtype.itemsize].clone().view(dtype)
    sizes = [1, 3, 8191, 8192, 8193, 16385] + [7] * 140  # one block's bytes and about, and more tensors than one launch takes
    srcs = [draw(n, dtype) for n in sizes for dtype in (torch.float32, torch.int32)]
    srcs += [draw(n, torch.uint8) for n in (1, 15, 16, 17, 32767, 32768, 32769)]
    srcs += [draw(20000, torch.int32)[1:], draw(40000, torch.bfloat16)[1:], draw(70001, torch.uint8)[3:]]  # 4, 2 and 1 bytes off a 16-byte boundary
    srcs += [draw(64, torch.int32).view(8, 8).t(), draw(0, torch.float32), torch.arange(5), draw(9, torch.int32)]  # strided, empty, from the host, converted
    backs = [torch.full((s.numel() * s.element_size() + 32,), 0x5a, dtype=torch.uint8, device=DEV) for s in srcs]  # sixteen bytes on either side
    dsts = [b[16:-16].view(s.dtype).view(s.shape) for b, s in zip(backs, srcs)]
    dsts[-1] = torch.empty(9, dtype=torch.int64, device=DEV)
    versions = [d._version for d in dsts]
    copy_tensors(dsts, srcs)
    for d, s, b in zip(dsts[:-1], srcs, backs):
        same = d.contiguous().view(-1).view(torch.uint8), s.to(DEV).contiguous().view(-1).view(torch.uint8)
        assert torch.equal(*same) and (b[:16] == 0x5a).all() and (b[-16:] == 0x5a).all()
    assert torch.equal(dsts[-1], srcs[-1].long()) and all(d._version > v for d, v in zip(dsts, versions))
    copy_tensors([], [])
    with pytest.raises(ValueError):
        copy_tensors(dsts[:2], srcs[:1])


def test_pairs_that_share_memory_are_copied_in_order():
    from tagseq2tagseq_b200.lm_fused import copy_tensors

    def chain(copy):
        base = torch.arange(300000, device=DEV, dtype=torch.float32)
        a, b, c = base[:100000], base[100000:200000], base[200000:]
        copy([b, c, a, b], [a, b, c, torch.full_like(b, 7)])      # each reads what the one before wrote, two write to one place
        copy([c.view(200, 500).t(), a[:100000]], [a.view(500, 200), c])  # a strided target between
        copy([a, a], [a, b])                                      # onto itself
        return base
    one_by_one = lambda dst, src: [d.copy_(s) for d, s in zip(dst, src)]
    assert torch.equal(chain(copy_tensors), chain(one_by_one))


def test_what_a_copy_does_besides_moving_bytes():
    from tagseq2tagseq_b200.lm_fused import copy_tensors
    x = torch.randn(5, device=DEV, requires_grad=True)
    w = torch.randn(5, device=DEV)
    d, e = torch.empty(5, device=DEV), torch.empty(5, device=DEV)
    copy_tensors([d, e], [x * 3, w])                              # the history of a source
    assert torch.equal(e, w) and torch.equal(torch.autograd.grad(d.sum(), x)[0], torch.full_like(w, 3))
    with torch.no_grad():
        d = torch.empty(5, device=DEV)
        copy_tensors([d, x], [x, w])
    assert not d.requires_grad and torch.equal(x.detach(), w)
    with pytest.raises(RuntimeError):                             # a leaf that learns
        copy_tensors([x], [w])
    copy_tensors([d], [torch._efficientzerotensor(5, device=DEV)])
    assert torch.equal(d, torch.zeros(5, device=DEV))
    with torch.inference_mode():
        frozen = torch.zeros(5, device=DEV)
    with pytest.raises(RuntimeError):                             # no writes to it outside
        copy_tensors([frozen], [w])
    with torch.autograd.forward_ad.dual_level():
        d = torch.empty(5, device=DEV)
        copy_tensors([d], [torch.autograd.forward_ad.make_dual(w, 2 * w)])
        assert torch.equal(torch.autograd.forward_ad.unpack_dual(d).tangent, 2 * w)

    def twice(a):
        out = torch.empty_like(a)
        copy_tensors([out], [a])
        return 2 * out
    rows = torch.randn(3, 5, device=DEV)
    assert torch.equal(torch.func.vmap(twice)(rows), 2 * rows)
