"""What the native operators refuse before anything reaches a device: inputs that a kernel would read past, or that would be
cut without a word.  CPU tensors stand in for CUDA ones: the checks come first."""
import pytest
import torch

from tagseq2tagseq_b200 import DocSpan, _lib, from_reference

OPS = _lib.ops()


@pytest.mark.parametrize("doc_id", [2**32 + 1, 2**31, -2**31 - 1])
def test_document_ids_beyond_32_bits_are_refused(doc_id):
    spans = [DocSpan(1, "", 0, 40), DocSpan(doc_id, "", 40, 90)]
    with pytest.raises(OverflowError):
        from_reference(spans, None, 100, device=torch.device("cuda"))
    with pytest.raises(ValueError, match="32 bits"):
        OPS.pack_mask([0, 40], [40, 90], [1, doc_id], [], [], 100, 64, torch.device("cuda", 0))


def test_a_target_shorter_than_the_rows_is_refused():
    """The loss kernel reads one target per row, whichever way a head's loss takes."""
    from tagseq2tagseq_b200.lm_fused import head_loss
    with pytest.raises(ValueError, match="target"):
        OPS.cross_entropy(torch.zeros(4, 16, dtype=torch.bfloat16), torch.zeros(3, dtype=torch.int64))
    h, w = torch.zeros(2, 4, 64, dtype=torch.bfloat16), torch.zeros(16, 64)
    for grad in (False, True):
        for n in (7, 9):
            with pytest.raises(ValueError, match="target"):
                head_loss(h, w.requires_grad_(grad), torch.zeros(n, dtype=torch.int64))


def test_rows_that_cannot_be_counted_are_refused():
    """A division by zero columns would end the process; an odd gate and up row would make the kernel count more rows than
    there are."""
    with pytest.raises(ValueError, match="columns"):
        OPS.add_rmsnorm(torch.zeros(4, 0), None, torch.zeros(0), 1e-6)
    for f in (0, 17):
        with pytest.raises(ValueError, match="even"):
            OPS.swiglu(torch.zeros(16, f, dtype=torch.bfloat16))


def test_norm_and_attention_refuse_operands_they_would_read_past():
    x = torch.zeros(4, 64)
    for a, w in ((torch.zeros(3, 64, dtype=torch.bfloat16), torch.zeros(64)), (None, torch.zeros(63))):
        with pytest.raises(ValueError, match="add_rmsnorm"):
            OPS.add_rmsnorm(x, a, w, 1e-6)
    plan, ids = torch.zeros(4, dtype=torch.uint8), torch.zeros(2, 5, dtype=torch.int32)
    good = torch.zeros(5, 32)
    for cos, sin, doc, row in ((good[:4], good, ids, None), (good, good[:, :31], ids, None), (good, torch.zeros(5, 64)[:, ::2], ids, None),
                               (good, good, ids[:1], None), (good, good, ids, ids[:, 1:])):
        with pytest.raises(ValueError, match="qkv_attention"):
            OPS.qkv_attention(torch.zeros(2, 5, 3 * 2 * 64, dtype=torch.bfloat16), cos, sin, doc, None, row, None, plan, 2, 64)
