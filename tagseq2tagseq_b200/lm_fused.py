"""The decoder-layer operators over include/ts2ts_lm.h, plus the attention call on the packed QKV projection.  They stand
where the reference's layer uses fused modules (model/modules/layer.py:20-35, model/modules/training_module.py:205); every
kernel is one pass over HBM, fp32 arithmetic, bf16 activations.  Autograd lives in csrc/torch_ops.cpp.
CUDA only: there is no CPU path.
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch
import torch.nn as nn
import torch.nn.functional as F
from torch.autograd import forward_ad as fwAD

from . import _lib
from .mask_spec import MaskSpec

__all__ = ["add_rmsnorm", "qkv_attention", "swiglu", "cross_entropy", "head_loss", "embedding", "rope_half_tables", "cast_weights", "copy_tensors", "Linear", "AdamW"]

_lib.load_if_built()
_MAX_HEAD_COLUMNS = 110592  # a row of logits that ts2ts_ce_fwd_grad keeps in shared memory


def _need_cuda(*ts):
    for t in ts:
        if t is not None and not t.is_cuda:
            raise RuntimeError("the decoder-layer kernels run on CUDA tensors only (no CPU path exists)")


def _call(op, *args):
    if torch.compiler.is_compiling():  # the operators run their autograd functions at once: a compiled caller breaks its graph here
        return _uncompiled(op, *args)
    try:
        return op(*args)
    except RuntimeError as e:
        raise _lib.failed_call(e) from None


_uncompiled = torch.compiler.disable(_call)


def add_rmsnorm(x: torch.Tensor, a: Optional[torch.Tensor], weight: torch.Tensor, eps: float) -> Tuple[torch.Tensor, torch.Tensor]:
    """(x + a, rmsnorm(x + a) * weight): the fp32 residual stream and the bf16 input of the next linear layer."""
    _need_cuda(x, a, weight)
    return _call(_lib.ops().add_rmsnorm.default, x, a, weight, eps)


def rope_half_tables(T: int, head_dim: int, base: float, device) -> Tuple[torch.Tensor, torch.Tensor]:
    """cos and sin of the rotation angles, fp32 [T, head_dim / 2] (pair i rotates with frequency base^(-2i/head_dim))."""
    inv = 1.0 / (base ** (torch.arange(0, head_dim, 2, device=device, dtype=torch.float32) / head_dim))
    ang = torch.arange(T, device=device, dtype=torch.float32)[:, None] * inv[None, :]
    return ang.cos().contiguous(), ang.sin().contiguous()


def qkv_attention(qkv: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, mask: MaskSpec, n_heads: int, head_dim: int) -> torch.Tensor:
    """Rotary embedding + masked attention on the packed projection qkv [B,T,3*H*D] (bf16, overwritten: q and k are
    rotated in place).  cos / sin: fp32 [T, head_dim/2] from ``rope_half_tables``.  Returns [B,T,H*D]."""
    _need_cuda(qkv, cos, sin)
    return _call(_lib.ops().qkv_attention.default, qkv, cos, sin, mask.doc_ids, mask.link_bits, mask.q_row_ids, mask.kv_col_ids, mask.plan,
                 n_heads, head_dim)


def swiglu(gate_up: torch.Tensor) -> torch.Tensor:
    """silu(gate) * up with gate, up = gate_up.chunk(2, dim=-1)."""
    _need_cuda(gate_up)
    return _call(_lib.ops().swiglu.default, gate_up)


def cross_entropy(logits: torch.Tensor, target: torch.Tensor) -> torch.Tensor:
    """Mean cross-entropy of bf16 logits [N,V] against int64 targets [N]; the backward overwrites ``logits`` with
    their gradient, so the caller must not use them afterwards."""
    _need_cuda(logits, target)
    return _call(_lib.ops().cross_entropy.default, logits, target)


def one_pass_head(vocab: int, width: int) -> bool:
    """Whether the loss of a head of this size is the one-pass kernel's, which takes a copy of the weight."""
    return vocab % 8 == 0 and vocab <= _MAX_HEAD_COLUMNS and width % 8 == 0


def head_loss(h: torch.Tensor, weight: torch.Tensor, target: torch.Tensor, copy: Optional[torch.Tensor] = None) -> torch.Tensor:
    """Mean cross-entropy of the output head ``h @ weight.T`` against ``target``; the logits never leave this call.  ``copy``: what
    ``cast_weights`` made of the weight as it is now, for a caller that has it; its values are not looked at, and the gradient is the weight's."""
    if target.numel() != h.shape[:-1].numel():
        raise ValueError("head_loss: one target per row of h")
    _need_cuda(h, weight, target)
    V = weight.shape[0]
    if (torch.is_grad_enabled() and (h.requires_grad or weight.requires_grad) and h.dtype == torch.bfloat16 and weight.dtype == torch.float32
            and one_pass_head(V, h.shape[-1])):
        return _call(_lib.ops().head_loss.default, h, weight, target, copy)
    logits = F.linear(h, weight.to(h.dtype))
    return cross_entropy(logits.to(torch.bfloat16).view(-1, V), target.reshape(-1))


def embedding(weight: torch.Tensor, tokens: torch.Tensor) -> torch.Tensor:
    """Rows of an fp32 embedding table."""
    if (weight.is_cuda and weight.dtype == torch.float32 and weight.shape[1] % 4 == 0 and tokens.dtype == torch.int64
            and (torch.compiler.is_compiling() or not transformed())):
        return _call(_lib.ops().embedding.default, weight, tokens)
    return F.embedding(tokens, weight)


def transformed() -> bool:
    """Whether a torch.func transform or forward-mode differentiation is active: C++ autograd functions know neither."""
    return torch._C._functorch.peek_interpreter_stack() is not None or fwAD._current_level >= 0


def cast_weights(weights) -> list:
    """bf16 copies of contiguous fp32 CUDA weights, all in one launch."""
    _need_cuda(*weights)
    return _call(_lib.ops().cast_weights.default, weights)


def copy_tensors(dst, src) -> None:
    """``d.copy_(s)`` for every pair, in order; neighbours on one GPU that are of one type and size, contiguous and apart from each other in one launch."""
    if transformed() and not torch.compiler.is_compiling():
        for d, s in zip(dst, src, strict=True):
            d.copy_(s)
    else:
        _call(_lib.ops().copy_tensors.default, dst, src)


class Linear(nn.Linear):
    """A bias-free linear layer with an fp32 weight.  Under bf16 autocast, bf16 activations multiply the weight's bf16 copy,
    and the weight gradient is produced in fp32; anything else is torch's own layer."""

    def __init__(self, in_features: int, out_features: int):
        super().__init__(in_features, out_features, bias=False)

    def forward(self, x: torch.Tensor, copy: Optional[torch.Tensor] = None) -> torch.Tensor:
        """``copy``: as for ``head_loss``."""
        if (x.is_cuda and x.dtype == torch.bfloat16 and self.weight.dtype == torch.float32 and torch.is_autocast_enabled("cuda")
                and torch.get_autocast_dtype("cuda") == torch.bfloat16 and (torch.compiler.is_compiling() or not transformed())):
            return _call(_lib.ops().linear.default, x, self.weight, copy)
        return super().forward(x)


class AdamW(torch.optim.AdamW):
    """torch.optim.AdamW with its state layout, the step being one launch of ``ts2ts_adamw`` per parameter group.  With
    ``fused=True`` it is torch's step, which a gradient scaler leaves the unscaling and the skipping to."""

    def _native(self, group, params) -> bool:
        if getattr(self, "_step_supports_amp_scaling", False) or getattr(self, "grad_scale", None) is not None or getattr(self, "found_inf", None) is not None:
            return False
        return (not group["amsgrad"] and not group["maximize"] and not group["capturable"] and not group["differentiable"]
                and not isinstance(group["lr"], torch.Tensor)
                and all(p.is_cuda and p.device == params[0].device and p.dtype == torch.float32 and p.is_contiguous() and not p.grad.is_sparse
                        and p.grad.dtype == torch.float32 for p in params))

    @torch.no_grad()
    def step(self, closure=None):
        groups = [(g, [p for p in g["params"] if p.grad is not None]) for g in self.param_groups]
        # a captured step would repeat the bias corrections of the step that was captured: torch's refuses
        if torch.cuda.is_current_stream_capturing() or not all(self._native(g, ps) for g, ps in groups if ps):
            return super().step(closure)
        loss = None
        if closure is not None:
            with torch.enable_grad():
                loss = closure()
            groups = [(g, [p for p in g["params"] if p.grad is not None]) for g in self.param_groups]
        for g, params in groups:
            if not params:
                continue
            for p in params:
                st = self.state[p]
                if len(st) == 0:
                    st["step"] = torch.zeros((), dtype=torch.float32, device="cpu")
                    st["exp_avg"] = torch.zeros_like(p, memory_format=torch.contiguous_format)
                    st["exp_avg_sq"] = torch.zeros_like(p, memory_format=torch.contiguous_format)
                    continue
                # a state saved by an optimizer that counts on the device or in fp64, or from a tensor of other strides
                if st["step"].is_cuda or st["step"].dtype != torch.float32:
                    st["step"] = st["step"].float().cpu()
                for name in ("exp_avg", "exp_avg_sq"):
                    if not st[name].is_contiguous():
                        st[name] = st[name].contiguous()
            states = [self.state[p] for p in params]
            _call(_lib.ops().adamw.default, params, [p.grad.contiguous() for p in params], [s["exp_avg"] for s in states],
                  [s["exp_avg_sq"] for s in states], [s["step"] for s in states], g["lr"], *g["betas"], g["eps"], g["weight_decay"])
        return loss
