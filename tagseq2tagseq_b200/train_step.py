"""Decoder-only LM training step around the masked-attention operator, with DDP over NCCL.

This is the scaling half of the benchmark: the call order of the reference's training module
(model/modules/training_module.py:195-211: shift tokens, build the mask once, embed -> backbone -> norm -> logits ->
cross-entropy) and its DDP settings (main.py:404-415: static graph, no unused parameters, 256 MB buckets), with a
plain pre-norm decoder (RMSNorm, fused QKV, RoPE, SwiGLU) standing in for the reference's tunalab modules, which are
not available.  Every layer calls the masked-attention kernels on the packed QKV projection (lm_fused.qkv_attention);
the block plan is built once per micro-batch and shared by all layers, as the reference shares its BlockMask
(block_mask_creator.py:132-139).  The GEMMs are cuBLAS through torch; the memory-bound pieces between them (residual add +
RMSNorm, rotary embedding, SwiGLU, cross-entropy, the embedding's gradient, AdamW) are single-pass kernels of this library,
as the reference's are fused modules.
"""
from __future__ import annotations

import warnings
from collections import OrderedDict
from contextlib import nullcontext as _nullcontext
from dataclasses import dataclass
from typing import Optional

import torch
import torch.nn as nn
import torch.nn.modules.module as _module
from torch.overrides import _get_current_function_mode_stack
from torch.utils._device import DeviceContext

from .lm_fused import AdamW, Linear, add_rmsnorm, cast_weights, copy_tensors, cross_entropy, embedding, head_loss, one_pass_head, qkv_attention, rope_half_tables, swiglu, transformed
from .mask_spec import MaskSpec

RMS_EPS = float(torch.finfo(torch.float32).eps)  # what nn.RMSNorm uses for fp32 input when eps is None


@dataclass
class LMConfig:
    n_layers: int = 12
    d_model: int = 768
    n_heads: int = 12
    head_dim: int = 64
    mlp_hidden: int = 3072
    vocab: int = 50304
    rope_base: float = 10000.0

    @property
    def matmul_params(self) -> int:
        """Parameters that take part in a GEMM per token (all linear layers and the output head)."""
        d, hd = self.d_model, self.n_heads * self.head_dim
        per_layer = d * 3 * hd + hd * d + 3 * d * self.mlp_hidden
        return self.n_layers * per_layer + d * self.vocab


def config4() -> LMConfig:
    return LMConfig(12, 768, 12, 64, 3072, 50304)


def config5() -> LMConfig:
    # SwiGLU hidden int(8/3 * 2048) = 5461 (model/modules/layer.py:26) rounded up to a multiple of 128 for GEMM alignment
    return LMConfig(24, 2048, 16, 128, 5504, 50304)


def rope_tables(T: int, head_dim: int, base: float, device, dtype=torch.float32):
    """cos and sin of the rotation angles, both halves filled: [T, head_dim] each, computed in fp32."""
    inv = 1.0 / (base ** (torch.arange(0, head_dim, 2, device=device, dtype=torch.float32) / head_dim))
    ang = torch.arange(T, device=device, dtype=torch.float32)[:, None] * inv[None, :]
    return torch.cat([ang.cos(), ang.cos()], dim=-1).to(dtype), torch.cat([ang.sin(), ang.sin()], dim=-1).to(dtype)


def apply_rope(x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor) -> torch.Tensor:
    """x [..., T, *, *, D] with cos / sin broadcastable to it; rotates pairs (first half, second half) in x's dtype:
    x * cos + rotate_half(x) * sin with rotate_half(x) = (-x2, x1)."""
    h = x.shape[-1] // 2
    rot = torch.cat([-x[..., h:], x[..., :h]], dim=-1)
    return x * cos + rot * sin


def _plain(module: nn.Module, cls: type) -> bool:
    """Whether calling ``module`` is nothing but ``cls.forward``: that class itself, and no hook of anybody's."""
    return (type(module) is cls and "forward" not in module.__dict__ and not _module._has_any_global_hook()
            and not (module._forward_hooks or module._forward_pre_hooks or module._backward_hooks or module._backward_pre_hooks))


class Block(nn.Module):
    """Pre-norm decoder layer.  It receives the residual stream ``x`` (fp32) and the branch output ``a`` (bf16) that
    has not been added to it yet, so that the add fuses with the RMSNorm that follows; it returns the pair in the
    same form: x <- x + a; x <- x + attn(norm(x)) is returned as (x, mlp branch output)."""

    def __init__(self, cfg: LMConfig):
        super().__init__()
        hd = cfg.n_heads * cfg.head_dim
        self.cfg = cfg
        self.ln1 = nn.RMSNorm(cfg.d_model)
        self.qkv = Linear(cfg.d_model, 3 * hd)
        self.proj = Linear(hd, cfg.d_model)
        self.ln2 = nn.RMSNorm(cfg.d_model)
        self.gate_up = Linear(cfg.d_model, 2 * cfg.mlp_hidden)
        self.down = Linear(cfg.mlp_hidden, cfg.d_model)

    def linears(self):
        return (self.qkv, self.proj, self.gate_up, self.down)

    def forward(self, x, a, mask: MaskSpec, cos, sin, copies=((),) * 4):
        """``copies``: what each of ``linears()`` gets beside its input, the weight's bf16 copy or nothing."""
        c, (qkv, proj, gate_up, down) = self.cfg, copies
        x, h = add_rmsnorm(x, a, self.ln1.weight, RMS_EPS)
        attn = qkv_attention(self.qkv(h, *qkv), cos, sin, mask, c.n_heads, c.head_dim)   # rotary + masked attention, layer.py:32-35
        x, h = add_rmsnorm(x, self.proj(attn, *proj), self.ln2.weight, RMS_EPS)
        return x, self.down(swiglu(self.gate_up(h, *gate_up)), *down)


class DecoderLM(nn.Module):
    def __init__(self, cfg: LMConfig):
        super().__init__()
        self.cfg = cfg
        self.embed = nn.Embedding(cfg.vocab, cfg.d_model)
        self.blocks = nn.ModuleList(Block(cfg) for _ in range(cfg.n_layers))
        self.norm = nn.RMSNorm(cfg.d_model)
        self.head = Linear(cfg.d_model, cfg.vocab)
        for p in self.parameters():
            if p.dim() >= 2:
                nn.init.normal_(p, std=0.02)

    _rope = None  # (what they are for, the tables of the last sequence length, the stream that made them, their completion)

    def __getstate__(self):
        return {**self.__dict__, "_rope": None}

    def _rope_tables(self, T: int, device):
        """cos and sin of the rotation angles.  The last length's are kept; whoever reads them on another stream waits for the
        one that made them.  Tables made under a trace or inside a capture belong to that alone."""
        key = (T, device, self.cfg.head_dim, self.cfg.rope_base)
        make = lambda: rope_half_tables(T, self.cfg.head_dim, self.cfg.rope_base, device)
        cuda = device.type == "cuda"
        if torch.compiler.is_compiling() or torch._C._len_torch_dispatch_stack() or (cuda and torch.cuda.is_current_stream_capturing()):
            return make()
        kept = self._rope  # read once: another thread may put another length's there
        if kept is None or kept[0] != key:
            with torch.inference_mode(False):  # they are saved for a backward later on
                tables = make()
            here = torch.cuda.current_stream(device) if cuda else None
            self._rope = (key, tables, here, here.record_event() if cuda else None)
            return tables
        _, tables, maker, done = kept
        if cuda and torch.cuda.current_stream(device) != maker:
            here = torch.cuda.current_stream(device)
            here.wait_event(done)
            for t in tables:
                t.record_stream(here)
        return tables

    def _weight_copies(self):
        """The bf16 copies that this forward's linear layers keep for their backward, ((copy,), ...) by layer and then the head's (() where its loss takes none), made in
        one launch.  None where a layer would not take one, or somebody's code could look at a weight, or change it, on the way."""
        layers = [m for blk in self.blocks if _plain(blk, Block) for m in blk.linears()] + [self.head]
        if (len(layers) != 4 * len(self.blocks) + 1 or torch.compiler.is_compiling() or not torch.is_grad_enabled() or _observed()
                or not torch.is_autocast_enabled("cuda") or torch.get_autocast_dtype("cuda") != torch.bfloat16
                or any(cls.forward is not _OWN_FORWARD[cls] for cls in (Block, Linear))
                or not all(_plain(m, Linear) and m.bias is None for m in layers)):
            return None
        weights = [m.weight for m in layers]
        if not all(type(w) in (nn.Parameter, torch.Tensor) and w.is_cuda and w.device == weights[0].device and w.dtype == torch.float32 and w.is_contiguous() for w in weights):
            return None
        # Frozen weights below the first one that learns are kept by nobody.
        if not (weights[0].requires_grad or getattr(getattr(self.embed, "weight", None), "requires_grad", False)):
            return None
        head = one_pass_head(*weights[-1].shape)
        return [(c,) for c in cast_weights(weights if head else weights[:-1])] + ([] if head else [()])

    def forward(self, tokens: torch.Tensor, mask: MaskSpec, rope=None) -> torch.Tensor:
        """tokens int64 [B, T+1]; returns the mean next-token cross-entropy (training_module.py:195-211).  Runs under
        bf16 autocast: the linear layers compute in bf16, the residual stream, norms, rotary angles and the loss in fp32.
        ``rope``: the rotation tables, for a caller that keeps them."""
        inp, tgt = tokens[:, :-1], tokens[:, 1:]
        e = self.embed
        if _plain(e, nn.Embedding) and e.padding_idx is None and e.max_norm is None and not e.scale_grad_by_freq and not e.sparse:
            x = embedding(e.weight, inp).float()
        else:
            x = e(inp).float()
        cos, sin = self._rope_tables(inp.shape[1], inp.device) if rope is None else rope
        a = None
        copies = self._weight_copies()
        for i, blk in enumerate(self.blocks):
            x, a = blk(x, a, mask, cos, sin, copies[4 * i:4 * i + 4]) if copies else blk(x, a, mask, cos, sin)
        _, h = add_rmsnorm(x, a, self.norm.weight, RMS_EPS)
        if _plain(self.head, Linear) and self.head.bias is None:
            return head_loss(h, self.head.weight, tgt, *(copies[-1] if copies else ()))
        logits = self.head(h)
        return cross_entropy(logits.to(torch.bfloat16).view(-1, logits.shape[-1]), tgt.reshape(-1))


_OWN_FORWARD = {cls: cls.forward for cls in (DecoderLM, Block, Linear, nn.RMSNorm, nn.Embedding, nn.ModuleList)}


class _Layout:
    """What a model was made of when this was taken."""

    @staticmethod
    def _settings(m: nn.Module):
        if isinstance(m, (DecoderLM, Block)):
            return (m.cfg, *vars(m.cfg).values())
        return (m.padding_idx, m.max_norm, m.scale_grad_by_freq, m.sparse) if isinstance(m, nn.Embedding) else ()

    def __init__(self, model: nn.Module):
        self.mods = list(model.modules())
        self.own = all(type(m) in _OWN_FORWARD for m in self.mods)
        self.settings = [self._settings(m) for m in self.mods]
        self.children = [dict(m._modules) for m in self.mods]
        self.slots = [dict(m._parameters) for m in self.mods]  # with the empty ones
        self.params = [(p, p.data_ptr()) for slots in self.slots for p in slots.values() if p is not None]

    def holds(self, model: nn.Module) -> bool:
        same = lambda now, then: now.keys() == then.keys() and all(now[k] is v for k, v in then.items())
        return (model is self.mods[0] and self.own == all(type(m) in _OWN_FORWARD for m in self.mods)
                and all(same(m._modules, c) for m, c in zip(self.mods, self.children))
                and all(same(m._parameters, s) for m, s in zip(self.mods, self.slots))
                and all(p.data_ptr() == at for p, at in self.params)
                and all(self._settings(m) == s for m, s in zip(self.mods, self.settings)))

    def hooked(self) -> bool:
        """Whether some call inside a step is more than the class's own forward, or some gradient is watched or not wanted."""
        return (not all(_plain(m, type(m)) for m in self.mods) or any(cls.forward is not f for cls, f in _OWN_FORWARD.items())
                or not all(p.requires_grad and not p._backward_hooks and not p._post_accumulate_grad_hooks for p, _ in self.params))


def _observed() -> bool:
    """Whether something of the caller's is called for every operator or saved tensor, or follows derivatives of its own."""
    return bool(transformed() or torch._C._len_torch_dispatch_stack() or torch.is_anomaly_enabled()
                or any(not isinstance(m, DeviceContext) for m in _get_current_function_mode_stack())
                or torch._C._autograd._top_saved_tensors_default_hooks(True) is not None)


class _StepGraph:
    """Forward and backward of one micro-batch shape as a CUDA graph: its inputs are copied into buffers of the graph's own,
    the block plan is part of it, copies of the gradients it writes are handed to the parameters.  Link bits are padded with rows and
    columns that grant nothing, so that packs with different numbers of documents share a graph."""

    def __init__(self, owner: "TrainStep", tokens: torch.Tensor, mask: MaskSpec, key):
        own = lambda t: None if t is None else torch.empty_like(t, memory_format=torch.contiguous_format)
        self.tokens = own(tokens)
        self.mask = MaskSpec(own(mask.doc_ids), None, own(mask.q_row_ids), own(mask.kv_col_ids))
        if mask.link_bits is not None:
            self.mask.link_bits = torch.zeros((mask.link_bits.shape[0],) + key[-2:], dtype=torch.int64, device=tokens.device)
        self._load(tokens, mask)
        names, self.params = zip(*owner.model.named_parameters())
        # read by the graph, but allocated outside of it: the model keeps only the last sequence length's
        self.tables = owner.model._rope_tables(tokens.shape[1] - 1, tokens.device)
        torch.cuda.current_stream().synchronize()  # they are there for a replay on whichever stream
        # Aliases stand for the parameters: an autograd graph of the caller's that is still alive keeps the nodes that
        # collect the parameters' gradients on its own stream, which a capture must not touch.
        alias = {n: p.detach().requires_grad_() for n, p in zip(names, self.params)}
        self.graph = torch.cuda.CUDAGraph()
        side, here = torch.cuda.Stream(), torch.cuda.current_stream()
        side.wait_stream(here)
        with torch.cuda.stream(side):
            self.graph.capture_begin(capture_error_mode="thread_local")
            try:
                with torch.autocast("cuda", dtype=torch.bfloat16):
                    loss = torch.func.functional_call(owner.model, alias, (self.tokens, self.mask, self.tables))
                self.grads = torch.autograd.grad(loss, tuple(alias.values()))
                self.loss = loss.detach()
            finally:
                self.graph.capture_end()
        here.wait_stream(side)
        self.stream = here  # of the last use
        self.mask._block_map = None  # built by the graph, into its own pool

    def _load(self, tokens, mask):
        m = self.mask
        pairs = [(self.tokens, tokens), (m.doc_ids, mask.doc_ids), (m.q_row_ids, mask.q_row_ids), (m.kv_col_ids, mask.kv_col_ids)]
        if m.link_bits is not None:
            R, W = mask.link_bits.shape[1:]
            if m.link_bits.shape[1:] != (R, W):
                m.link_bits.zero_()
            pairs.append((m.link_bits[:, :R, :W], mask.link_bits))
        copy_tensors(*zip(*(p for p in pairs if p[0] is not None)))

    def run(self, tokens, mask) -> torch.Tensor:
        here = torch.cuda.current_stream()
        if here != self.stream:  # the buffers are in use until the last replay is through
            here.wait_stream(self.stream)
            m = self.mask
            for t in (self.tokens, m.doc_ids, m.link_bits, m.q_row_ids, m.kv_col_ids, *self.tables):
                if t is not None:
                    t.record_stream(here)
            self.stream = here
        self._load(tokens, mask)
        self.graph.replay()
        grads = [torch.empty_like(p) for p in self.params]  # the graph's own buffers are written again by the next step
        loss = torch.empty_like(self.loss)
        copy_tensors([*grads, loss], [*self.grads, self.loss])
        for p, g in zip(self.params, grads):
            p.grad = g
        return loss


class TrainStep:
    """One optimizer step on one packed sequence per rank: forward under bf16 autocast, backward (DDP all-reduces
    the gradients, overlapped with the backward), fused AdamW on fp32 parameters.

    DDP settings follow main.py:404-415 (static graph, no unused parameters, 256 MB buckets; the first bucket keeps
    torch's small default so that the last gradients to be produced start their all-reduce early).  With
    ``bf16_grads`` the buckets are cast to bf16 for the all-reduce and back (torch's ``bf16_compress_hook``), which
    halves the bytes on NVLink; the parameters and the optimizer state stay fp32.

    On one GPU, a step whose kernels are shorter than the host work of launching them (see ``_use_graph``) is replayed as
    a CUDA graph from the second micro-batch of its shape on.  ``use_graphs = False`` turns that off."""

    MAX_GRAPHS = 2   # micro-batch shapes whose graph, and with it a step's activations, is kept
    IDLE_STEPS = 64  # steps without a replay after which a graph makes room for another shape's

    def __init__(self, cfg: LMConfig, device: torch.device, world: int = 1, lr: float = 3e-4, seed: int = 0,
                 bf16_grads: bool = True, bucket_cap_mb: int = 256):
        torch.manual_seed(seed)  # identical initial weights on every rank
        self.cfg, self.device, self.world = cfg, device, world
        model = DecoderLM(cfg).to(device)
        self.model = model
        self.bf16_grads = bool(bf16_grads and world > 1)
        if world > 1:
            self.model = torch.nn.parallel.DistributedDataParallel(
                model, device_ids=[device.index], static_graph=True, find_unused_parameters=False, bucket_cap_mb=bucket_cap_mb,
                gradient_as_bucket_view=True)
            if self.bf16_grads:
                from torch.distributed.algorithms.ddp_comm_hooks import default_hooks
                self.model.register_comm_hook(None, default_hooks.bf16_compress_hook)
        self.opt = AdamW(model.parameters(), lr=lr, betas=(0.9, 0.95), weight_decay=0.1)
        self.use_graphs = True
        self._graphs: "OrderedDict[tuple, _StepGraph]" = OrderedDict()  # by last use
        self._seen: "OrderedDict[tuple, None]" = OrderedDict()  # shapes of earlier steps
        self._steps = 0
        self._refused = set()  # shapes that could not be captured
        self._layout = None

    @property
    def grad_bytes_per_step(self) -> int:
        """Bytes each rank contributes to the gradient all-reduce of one step."""
        n = sum(p.numel() for p in self.model.parameters())
        return n * (2 if self.bf16_grads else 4)

    def forward_backward(self, tokens: torch.Tensor, mask: MaskSpec, sync: bool = True) -> torch.Tensor:
        """Loss and gradients without the optimizer step.  ``sync=False`` skips the gradient all-reduce (DDP's
        ``no_sync``): the difference between the two is what the collective costs this rank."""
        if self.use_graphs and self.world == 1:
            key = self._graph_key(tokens, mask)
            if key is not None:
                return self._graphed(key, tokens, mask)
        elif self._graphs:
            self._graphs.clear()
        return self._eager(tokens, mask, sync)

    def _eager(self, tokens: torch.Tensor, mask: MaskSpec, sync: bool = True) -> torch.Tensor:
        self.opt.zero_grad(set_to_none=True)
        ctx = self.model.no_sync() if (not sync and self.world > 1) else _nullcontext()
        with ctx:
            with torch.autocast("cuda", dtype=torch.bfloat16):
                loss = self.model(tokens, mask)
            loss.backward()
        return loss.detach()

    # ------------------------------------------------------------------ CUDA graphs of small steps
    def _use_graph(self, n_tokens: int) -> bool:
        """Launching a step takes about half a millisecond of host time per layer and as much for the rest; the GEMMs
        take 6 FLOPs per parameter and token at 1.2 PFLOP/s or less.  Where the second is shorter, the GPU waits for the
        host (two layers of d256 at T=1024: 1.38 ms a step, of which 0.38 ms of kernels).  A graph holds on to a step's
        memory, which a thin model with a large vocabulary makes much of at the same FLOPs: one graph may take a 32nd of
        the card's."""
        return (6.0 * self.cfg.matmul_params * n_tokens / 1.2e12 < 0.5 * (self.cfg.n_layers + 1)
                and self._graph_bytes(n_tokens) <= torch.cuda.get_device_properties(self.device).total_memory / 32)

    def _graph_bytes(self, n_tokens: int) -> int:
        """About what a step's graph holds on to: weights' copies and gradients, saved activations, logits, and the largest
        intermediate gradients."""
        c = self.cfg
        hd = c.n_heads * c.head_dim
        layer = 14 * c.d_model + 8 * hd + 4 * c.n_heads + 6 * c.mlp_hidden  # residual twice in fp32, the rest in bf16
        return (6 * (c.matmul_params + c.d_model * c.vocab)
                + n_tokens * (c.n_layers * layer + 2 * c.vocab + 24 * c.d_model + 6 * max(c.mlp_hidden, 2 * hd)))

    def _graph_key(self, tokens: torch.Tensor, mask: MaskSpec):
        """What a graph is kept by, or None for a step that has to be launched: inputs that the launched step would look at
        more closely, or a caller that wants to see its operators."""
        if type(mask) is not MaskSpec or tokens.dim() != 2 or self.device.type != "cuda":
            return None
        doc, link, rows, cols = mask.doc_ids, mask.link_bits, mask.q_row_ids, mask.kv_col_ids
        B, T = tokens.shape[0], tokens.shape[1] - 1
        fits = lambda t, dtype: type(t) is torch.Tensor and t.device == self.device and t.dtype == dtype
        if not (fits(tokens, torch.int64) and B > 0 and T > 0 and self._use_graph(B * T)
                and all(fits(t, torch.int32) and t.shape == (B, T) for t in (doc, rows, cols) if t is not None)
                and (link is None or fits(link, torch.int64) and link.dim() == 3 and link.shape[0] == B and link.numel() > 0)
                and torch.cuda.current_device() == self.device.index):
            return None
        if torch.cuda.is_current_stream_capturing() or not torch.is_grad_enabled() or _observed() or not self._as_built():
            return None
        key = (B, T, rows is not None, cols is not None, torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction,
               torch.are_deterministic_algorithms_enabled())
        if link is not None:  # capacities in steps of 64 row classes and of powers of two words
            key += (-(-link.shape[1] // 64) * 64, 1 << (link.shape[2] - 1).bit_length())
        return key

    def _as_built(self) -> bool:
        """Whether a replay does what the model would do: the model is the one the graphs were captured from, made of this
        package's modules alone and configured as it was, its parameters are where they were, and nothing hangs on it that
        a replay would not call."""
        kept = self._layout
        if kept is None or not kept.holds(self.model):
            self._graphs.clear()  # captured again, from a layout taken now
            self._refused.clear()
            self._layout = kept = _Layout(self.model)
        return kept.own and not kept.hooked()

    def _graphed(self, key, tokens: torch.Tensor, mask: MaskSpec) -> torch.Tensor:
        self._steps += 1
        graph = self._graphs.get(key)
        if graph is None:
            # the first step of a shape runs as it is: libraries set themselves up
            if key in self._refused or not self._again(key) or not self._room():
                return self._eager(tokens, mask)
            try:
                graph = _StepGraph(self, tokens, mask, key)
            except RuntimeError as e:  # a step that cannot be captured, or no memory for it, still runs launch by launch
                warnings.warn(f"training step of {tuple(tokens.shape)} tokens could not be captured and stays launched: {e}")
                self._refused.add(key)
                return self._eager(tokens, mask)
        self._graphs[key] = graph
        self._graphs.move_to_end(key)
        graph.used_at = self._steps
        return graph.run(tokens, mask)

    def _again(self, key) -> bool:
        """Whether this shape has come before."""
        before = key in self._seen
        self._seen[key] = None
        self._seen.move_to_end(key)
        while len(self._seen) > 64:
            self._seen.popitem(last=False)
        return before

    def _room(self) -> bool:
        """Whether one more graph may be kept.  The one that was not replayed for longest makes room, but only if it has been
        idle for IDLE_STEPS: when more shapes take turns than graphs are kept, the others stay launched, and captures cost
        at most one in that many steps."""
        if len(self._graphs) < self.MAX_GRAPHS:
            return True
        oldest = next(iter(self._graphs))
        if self._steps - self._graphs[oldest].used_at <= self.IDLE_STEPS:
            return False
        del self._graphs[oldest]
        return True

    def step(self, tokens: torch.Tensor, mask: MaskSpec) -> torch.Tensor:
        loss = self.forward_backward(tokens, mask)
        self.opt.step()
        return loss


def train_flops_per_step(cfg: LMConfig, T: int, unmasked_pairs: int) -> float:
    """6 * P_matmul * T for the linear layers (forward + backward) plus 14 * D * H * N per layer for attention."""
    return 6.0 * cfg.matmul_params * T + cfg.n_layers * 14.0 * cfg.head_dim * cfg.n_heads * unmasked_pairs
