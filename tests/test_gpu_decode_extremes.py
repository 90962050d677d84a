"""The decoding step with infinite values in the cache: an allowed key hands its infinity on, a key without weight nothing."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda")


@pytest.mark.parametrize("tk", [1, 3, 33, 1500, 5000])
@pytest.mark.parametrize("d", [64, 128])
def test_infinite_values_of_allowed_keys_stay_infinite(tk, d):
    from tagseq2tagseq_b200.attention import masked_attn_decode
    g = torch.Generator(device=DEV).manual_seed(tk)
    q = torch.randn(1, 2, 1, d, device=DEV, generator=g).bfloat16()
    k, v = (torch.randn(1, 2, tk, d, device=DEV, generator=g).bfloat16() for _ in range(2))
    v[0, 0, tk - 1, 5], v[0, 1, tk // 2, 7] = math.inf, -math.inf
    out, lse = masked_attn_decode(q, k, v, torch.zeros(1, tk, dtype=torch.int32, device=DEV))
    assert out[0, 0, 0, 5] == math.inf and out[0, 1, 0, 7] == -math.inf
    out[0, 0, 0, 5] = out[0, 1, 0, 7] = 0
    assert out.isfinite().all() and lse.isfinite().all()


@pytest.mark.parametrize("at", [0, 40, 2999])
def test_values_of_keys_whose_weight_underflows_do_not_matter(at):
    """One key outweighs all others by more than fp32 can hold, wherever it comes in the order of the sums."""
    from tagseq2tagseq_b200.attention import masked_attn_decode
    tk, d = 3000, 64
    q = torch.ones(1, 1, 1, d, device=DEV).bfloat16()
    k, v = torch.zeros(1, 1, tk, d, device=DEV).bfloat16(), torch.full((1, 1, tk, d), math.inf, device=DEV).bfloat16()
    k[0, 0, at], v[0, 0, at] = 64.0, 3.0                          # score 64 * 64 / 8 = 512
    out, lse = masked_attn_decode(q, k, v, torch.zeros(1, tk, dtype=torch.int32, device=DEV))
    assert torch.equal(out, torch.full_like(out, 3.0)) and abs(float(lse) - 512.0) <= 1e-3
