"""The forward's order of work over a batch: every query tile of every element and head is computed once, whichever way the elements are
ordered.  Uniform values make a row's result a mean over the keys it may read, so a row that was left out or taken from another
element's list shows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,h,t,d", [(3, 5, 700, 64), (4, 8, 2039, 64), (2, 12, 2500, 128), (4, 16, 3600, 128), (2, 16, 14400, 128), (3, 7, 9000, 128)])
def test_every_row_of_a_batch_is_the_mean_of_its_keys(b, h, t, d):
    """Batches whose keys and values fit the L2 and batches whose do not (the last but one), pairs of query tiles and shared ones."""
    from tagseq2tagseq_b200 import build_block_map, read_status
    from tagseq2tagseq_b200.attention import masked_attn
    dev = torch.device("cuda")
    at = torch.arange(t, device=dev)
    doc = torch.stack([at // (97 + 411 * i) for i in range(b)]).int()         # every element has lists of its own
    start = torch.stack([at // (97 + 411 * i) * (97 + 411 * i) for i in range(b)])
    q = torch.zeros(b, h, t, d, device=dev, dtype=torch.bfloat16)
    k = torch.zeros_like(q)
    v = torch.zeros_like(q)
    v[..., :] = ((at % 7).float()[None, None, :, None] + torch.arange(h, device=dev)[None, :, None, None] + 16 * torch.arange(b, device=dev)[:, None, None, None]).bfloat16()
    plan = build_block_map(doc).plan
    out, lse = masked_attn(q, k, v, doc, plan=plan)
    assert read_status(plan) == 0
    sums = torch.cat([torch.zeros(1, device=dev, dtype=torch.float64), (at % 7).double().cumsum(0)])
    n = (at[None] - start + 1).double()
    mean = (sums[at + 1][None] - sums[start]) / n
    want = mean[:, None, :] + torch.arange(h, device=dev)[None, :, None] + 16 * torch.arange(b, device=dev)[:, None, None]
    assert (lse - n.log()[:, None].float()).abs().max() <= 1e-4
    assert ((out.double() - want[..., None]).abs() / (want[..., None] + 1)).max() <= 2 ** -7   # bf16 result: half a step of 2^-8, and P = 1
