"""Shapes of the operators' results, for tracing callers.  Imported once the operators are loaded."""
import torch


@torch.library.register_fake("ts2ts::masked_attn_fwd")
def _(q, k, v, doc_ids, link_bits, q_row_ids, kv_col_ids, plan, scale):
    B, H, T, D = q.shape
    return q.new_empty((B, H, T, D)), q.new_empty((B, H, T), dtype=torch.float32)


@torch.library.register_fake("ts2ts::masked_attn_bwd")
def _(q, k, v, out, dout, lse, doc_ids, link_bits, q_row_ids, kv_col_ids, plan, scale):
    return torch.empty_like(q), torch.empty_like(k), torch.empty_like(v)


@torch.library.register_fake("ts2ts::masked_attn_decode")
def _(q, k_cache, v_cache, doc_ids, link_bits, q_row_ids, kv_col_ids, q_pos, scale):
    B, H, Tk, D = k_cache.shape
    return q.new_empty((B, H, 1, D)), q.new_empty((B, H), dtype=torch.float32)
