"""The workloads by which the speed of this package is judged: what a program that uses it has it do, through its public
entry points, from the smallest calls to the largest.

``listed()`` names representative cases, ``draw(rng)`` gives further ones of the same ranges, ``prepare`` makes what the
program holds before the call, ``run`` makes the call.  Five kinds:

  attn    the masked-attention operator (``masked_attn``, or the ``flex_attention`` drop-in on strided views of a packed
          QKV projection), forward alone or forward and backward, with the mask's block plan kept as every layer after
          the first finds it
  decode  one new token per sequence against cached keys and values (``masked_attn_decode``)
  mask    one micro-batch's mask from its tokens and document spans: link scan, grants, block plan
  plan    the block plan and its lists from per-token ids and link bits, as the pack scheduler asks for them
  train   one optimizer step of the decoder LM on a fresh micro-batch mask, gradients and parameters handed back
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from tagseq2tagseq_b200 import CrossDocLinkMaskCreator, DocSpan, MaskSpec, build_block_map, make_mask_creator_callable
from tagseq2tagseq_b200 import make_mask_creator_callable_from, synth
from tagseq2tagseq_b200.attention import flex_attention, masked_attn, masked_attn_decode
from tagseq2tagseq_b200.link_detect import MarkdownLinkDetector
from tagseq2tagseq_b200.train_step import LMConfig, TrainStep, train_flops_per_step

DEV = torch.device("cuda")


# ------------------------------------------------------------------------------------------------------------- cases
def _attn(name, B, T, H, D, p_link, median, lo, hi, heavy=0.0, mask="pack", layout="bhtd", backward=True):
    case = {"kind": "attn", "B": B, "T": T, "H": H, "D": D, "p_link": p_link, "median": median, "lo": lo, "hi": hi, "heavy": heavy,
            "mask": mask, "layout": layout, "backward": backward}
    return dict(case, name=name) if name else case


def _decode(name, B, Tk, H, D, p_link, median, lo, hi, heavy=0.0, uneven=False):
    case = {"kind": "decode", "B": B, "T": Tk, "H": H, "D": D, "p_link": p_link, "median": median, "lo": lo, "hi": hi, "heavy": heavy,
            "uneven": uneven}
    return dict(case, name=name) if name else case


def _mask(name, T, p_link, max_grants):
    case = {"kind": "mask", "B": 1, "T": T, "p_link": p_link, "median": 200, "lo": 32, "hi": 2048, "heavy": 0.0, "max_grants": max_grants}
    return dict(case, name=name) if name else case


def _plan(name, B, T, p_link, median, lo, hi, heavy):
    case = {"kind": "plan", "B": B, "T": T, "p_link": p_link, "median": median, "lo": lo, "hi": hi, "heavy": heavy}
    return dict(case, name=name) if name else case


def _train(name, layers, d_model, heads, head_dim, mlp, vocab, T, p_link, median, lo, hi):
    case = {"kind": "train", "layers": layers, "d_model": d_model, "heads": heads, "head_dim": head_dim, "mlp": mlp, "vocab": vocab,
            "B": 1, "T": T, "p_link": p_link, "median": median, "lo": lo, "hi": hi, "heavy": 0.0}
    return dict(case, name=name) if name else case


def listed():
    return [
        # the CPU-runnable configuration: a short pack of small documents, where launches and host work count
        _attn("attn_2k_doc_causal", 1, 2048, 8, 64, 0.0, 128, 16, 512),
        # recomputing a ragged prompt with its linked pages for the next token: forward only, through the drop-in on
        # strided views of the QKV projection
        _attn("attn_prefill_5003", 1, 5003, 12, 64, 0.15, 200, 32, 2048, layout="packed", backward=False),
        # a batch of whole sequences under the plain causal mask, one mask broadcast over the batch
        _attn("attn_4k_causal_batch4", 4, 4096, 16, 128, 0.0, 200, 32, 2048, mask="causal", layout="packed"),
        # one training layer's attention on a linked 16k pack
        _attn("attn_16k_linked", 1, 16384, 16, 128, 0.15, 200, 32, 2048),
        # the size the headline rate is quoted at: 32k packs with a heavy tail of long documents, dense links
        _attn("attn_32k_linked_heavy", 2, 32768, 16, 128, 0.3, 150, 16, 4096, heavy=0.05),
        # generation in small batches: short caches filled to different lengths
        _decode("decode_1111_batch8", 8, 1111, 12, 64, 0.0, 200, 32, 2048, uneven=True),
        # generation at the end of a long linked context
        _decode("decode_32k_linked", 2, 32768, 16, 128, 0.3, 150, 16, 4096, heavy=0.05),
        # the data loader's part of a step: a 16k pack's mask from tokens and spans
        _mask("mask_16k_markdown", 16384, 0.15, 256),
        # the pack scheduler's view of two 32k packs
        _plan("plan_32k_batch2", 2, 32768, 0.3, 150, 16, 4096, 0.05),
        # a toy model: every launch of the step is small
        _train("train_toy_1k", 2, 256, 4, 64, 1024, 4096, 1024, 0.2, 60, 8, 300),
        # the two model widths of the training benchmark.  Depth is cut to four layers: deeper models repeat the same
        # work per layer, and four layers' gradients and parameters can be handed back whole
        _train("train_d768_16k", 4, 768, 12, 64, 3072, 50304, 16384, 0.15, 200, 32, 2048),
        _train("train_d2048_32k", 4, 2048, 16, 128, 5504, 50304, 32768, 0.3, 200, 32, 2048),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attn"] * 4 + ["decode"] * 2 + ["mask", "plan"] + ["train"] * 2)
    p_link = rng.choice([0.0, 0.05, 0.15, 0.3])
    median = _log_int(rng, 80, 400)
    if kind == "attn":
        T = _log_int(rng, 200, 32768)
        D = rng.choice([64, 128])
        B = rng.choice([1, 2, 4] if T <= 16384 else [1, 2])
        H = rng.choice([2, 3, 8, 12, 16])
        mask = "causal" if T <= 8192 and rng.random() < 0.25 else "pack"
        return _attn(None, B, T, H, D, 0.0 if mask == "causal" else p_link, median, 16, 2048, heavy=0.05 if T > 16384 else 0.0, mask=mask,
                     layout=rng.choice(["bhtd", "packed"]), backward=rng.random() < 0.7)
    if kind == "decode":
        T = _log_int(rng, 100, 65536)
        B = rng.choice([1, 2, 4, 8, 16] if T <= 8192 else [1, 2])
        return _decode(None, B, T, rng.choice([8, 12, 16]), rng.choice([64, 128]), p_link, median, 16, 4096, heavy=0.05 if T > 16384 else 0.0,
                       uneven=rng.random() < 0.5)
    if kind == "mask":
        return _mask(None, _log_int(rng, 1024, 32768), rng.choice([0.05, 0.15, 0.3]), rng.choice([64, 256]))
    if kind == "plan":
        T = _log_int(rng, 1024, 32768)
        return _plan(None, rng.choice([1, 2, 4]), T, p_link, median, 16, 4096, 0.05 if T > 16384 else 0.0)
    head_dim = rng.choice([64, 128])
    d_model = rng.choice([256, 512, 768, 1024, 2048])
    return _train(None, rng.choice([2, 3, 4]), d_model, d_model // head_dim, head_dim, rng.choice([2, 4]) * d_model, rng.choice([4096, 32768, 50304]),
                  _log_int(rng, 700, 16384), p_link, median, 16, 2048)


# ------------------------------------------------------------------------------------------------------------- inputs
def _packs(case, seed):
    heavy = dict(heavy_frac=case["heavy"], heavy_lo=4096, heavy_hi=8192) if case["heavy"] else {}
    return [synth.make_pack(seed * 1000 + b, case["T"], case["median"], case["lo"], case["hi"], p_link=case["p_link"], **heavy)
            for b in range(case["B"])]


def _mask_tensors(packs):
    doc, link = synth.stack_packs(packs)
    return torch.from_numpy(doc).to(DEV), None if link is None else torch.from_numpy(link).to(DEV)


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _normal(gen, *shape):
    return torch.randn(*shape, device=DEV, generator=gen, dtype=torch.float32).bfloat16()


# A byte-level vocabulary of GPT-2's size with its link tokens where the detector expects them: '[' 58, ' [' 685,
# '](' 16151, and a few tokens that hold a ')'; every other id is a word of its own.
_VOCAB = [b" w%d" % i for i in range(50257)]
_VOCAB[8], _VOCAB[737], _VOCAB[828] = b")", b").", b"),"
_VOCAB[58], _VOCAB[685], _VOCAB[16151] = b"[", b" [", b"]("


def _decode_tokens(ids):
    return b"".join([_VOCAB[i] for i in ids]).decode("utf-8", errors="replace")


@functools.lru_cache(maxsize=None)
def _detector():
    """A program has one detector for its whole life."""
    return MarkdownLinkDetector(_decode_tokens, window_tokens=50)


def _markdown_pack(case, seed):
    """Token stream and spans of a pack of pages that link to earlier pages: '[', two words, '](', the page's two-word
    name, ')' wherever the page has room for the link.  Page lengths and links belong to the case, the text, the names
    and the links' places to the seed, so that every seed's mask has as many link classes."""
    pack = _packs(case, case["T"])[0]
    rng = np.random.default_rng(seed)
    tokens = rng.integers(17000, 50000, case["T"])
    starts = np.concatenate([[0], np.cumsum(pack.lengths)])
    names = rng.integers(1000, 16000, (pack.lengths.size, 2))
    targets = {}
    for a, b in pack.links:
        targets.setdefault(a, []).append(b)
    for a, linked in targets.items():
        slots = int(pack.lengths[a]) // 12
        for slot, b in zip(rng.permutation(slots), linked):
            at = int(starts[a]) + 12 * int(slot) + int(rng.integers(0, 5))
            tokens[at:at + 7] = [rng.choice([58, 685]), rng.integers(17000, 50000), rng.integers(17000, 50000), 16151, *names[b], rng.choice([8, 737, 828])]
    spans = [DocSpan(i, "", int(starts[i]), int(starts[i + 1]), False, [], _decode_tokens([int(t) for t in names[i]]).strip())
             for i in range(pack.lengths.size)]
    return torch.from_numpy(tokens)[None].to(DEV), spans


def prepare(case, seed):
    kind, gen = case["kind"], _generator(seed)
    state = {"kind": kind}
    if kind == "attn":
        B, T, H, D = case["B"], case["T"], case["H"], case["D"]
        if case["mask"] == "causal":
            spec = make_mask_creator_callable("causal")(tokens=torch.zeros((1, T), dtype=torch.int64, device=DEV), doc_spans=[])
            spec.expanded(B).plan  # kept on the spec; the operator itself takes a mask of as many sequences as q has
            spec = spec if case["layout"] == "packed" else spec.expanded(B)
        else:
            spec = MaskSpec(*_mask_tensors(_packs(case, seed)))
            spec.plan
        if case["layout"] == "packed":
            qkv = _normal(gen, B, T, 3, H, D)
            q, k, v = (qkv[:, :, i].permute(0, 2, 1, 3) for i in range(3))
        else:
            q, k, v = (_normal(gen, B, H, T, D) for _ in range(3))
        for t in (q, k, v):
            t.requires_grad_(case["backward"])
        state.update(spec=spec, q=q, k=k, v=v, through="flex" if case["layout"] == "packed" else "op", backward=case["backward"])
        if case["backward"]:
            state["do"] = _normal(gen, B, H, T, D)
    elif kind == "decode":
        B, T, H, D = case["B"], case["T"], case["H"], case["D"]
        doc, link = _mask_tensors(_packs(case, seed))
        pos = torch.randint(T // 2, T, (B,), device=DEV, generator=gen, dtype=torch.int32) if case["uneven"] else None
        state.update(doc=doc, link=link, pos=pos, q=_normal(gen, B, H, 1, D), k=_normal(gen, B, H, T, D), v=_normal(gen, B, H, T, D))
    elif kind == "mask":
        tokens, spans = _markdown_pack(case, seed)
        creator = make_mask_creator_callable_from(CrossDocLinkMaskCreator(_detector(), max_grants=case["max_grants"]))
        state.update(creator=creator, tokens=tokens, spans=spans)
    elif kind == "plan":
        doc, link = _mask_tensors(_packs(case, seed))
        state.update(doc=doc, link=link)
    else:
        cfg = LMConfig(case["layers"], case["d_model"], case["heads"], case["head_dim"], case["mlp"], case["vocab"])
        with torch.device(DEV):  # weights are drawn on the GPU
            step = TrainStep(cfg, torch.device("cuda", torch.cuda.current_device()), seed=seed)
        doc, link = _mask_tensors(_packs(case, seed))
        tokens = torch.randint(0, cfg.vocab, (1, case["T"] + 1), device=DEV, generator=gen)
        state.update(step=step, doc=doc, link=link, tokens=tokens, params=list(step.model.parameters()))
    return state


# ------------------------------------------------------------------------------------------------------------- the calls
def run(state):
    kind = state["kind"]
    if kind == "attn":
        q, k, v, spec = state["q"], state["k"], state["v"], state["spec"]
        if state["through"] == "flex":
            out, lse = flex_attention(q, k, v, block_mask=spec, return_lse=True)
        else:
            out, lse = masked_attn(q, k, v, spec.doc_ids, spec.link_bits, plan=spec.plan)
        if not state["backward"]:
            return {"out": out, "lse": lse}
        dq, dk, dv = torch.autograd.grad(out, (q, k, v), state["do"])
        return {"out": out, "lse": lse, "dq": dq, "dk": dk, "dv": dv}
    if kind == "decode":
        out, lse = masked_attn_decode(state["q"], state["k"], state["v"], state["doc"], state["link"], q_pos=state["pos"])
        return {"out": out, "lse": lse}
    if kind == "mask":
        spec = state["creator"](tokens=state["tokens"], doc_spans=state["spans"])
        return {"doc_ids": spec.doc_ids, "link_bits": spec.link_bits, "q_row_ids": spec.q_row_ids, "kv_col_ids": spec.kv_col_ids,
                "lists": list(spec.block_map(with_lists=True)[1:])}
    if kind == "plan":
        return list(build_block_map(state["doc"], state["link"], with_lists=True)[1:])
    loss = state["step"].step(state["tokens"], MaskSpec(state["doc"], state["link"]))
    return {"loss": loss, "params": state["params"], "grads": [p.grad for p in state["params"]]}


# ------------------------------------------------------------------------------------------------------------- what a pass cannot do without
@functools.lru_cache(maxsize=None)
def _mean_pairs(items):
    """Allowed (query, key) pairs of one pass: the mean over a few seeds of the case's packs."""
    case = dict(items)
    if case.get("mask") == "causal":
        return case["B"] * case["T"] * (case["T"] + 1) / 2
    seeds = range(4)
    return sum(p.unmasked_pairs() for s in seeds for p in _packs(case, 77 + s)) / len(seeds)


@functools.lru_cache(maxsize=None)
def _mean_decode_keys(items):
    """Keys the last token of each sequence may read, summed over the batch: the mean over a few seeds."""
    case = dict(items)
    total, seeds = 0, range(8)
    for s in seeds:
        for pack in _packs(case, 77 + s):
            last = pack.lengths.size - 1
            reads = [b for a, b in pack.links if a == last] + [last]
            total += int(pack.lengths[reads].sum())
    return total / len(seeds) * (0.75 if case["uneven"] else 1.0)


def work(case):
    kind = case["kind"]
    items = tuple(sorted(case.items()))
    T, B = case["T"], case["B"]
    if kind == "attn":
        H, D, n = case["H"], case["D"], _mean_pairs(items)
        rows = B * H * T
        nbytes = rows * (4 * 2 * D + 4) + (rows * (8 * 2 * D + 4) if case["backward"] else 0)
        return {"bytes": nbytes, "flops": (14 if case["backward"] else 4) * D * H * n}
    if kind == "decode":
        H, D, keys = case["H"], case["D"], _mean_decode_keys(items)
        return {"bytes": H * keys * 4 * D + 8 * B * T, "flops": 4 * D * H * keys}
    if kind in ("mask", "plan"):
        nb = (T + 127) // 128
        read = 8 * T if kind == "mask" else 4 * B * T
        return {"bytes": read + B * (nb * nb * (1 + 4 * 4) + 12 * T * (kind == "mask")), "flops": 0}
    cfg = LMConfig(case["layers"], case["d_model"], case["heads"], case["head_dim"], case["mlp"], case["vocab"])
    params = cfg.matmul_params + cfg.d_model * (cfg.vocab + 2 * cfg.n_layers + 1)
    # fp32 parameters and the two Adam moments are read and written, gradients written
    return {"bytes": 28 * params, "flops": train_flops_per_step(cfg, T, _mean_pairs(items))}


def tolerance(case):
    if case["kind"] in ("mask", "plan"):
        return "exact"
    if case["kind"] == "train":
        return {"rel": 2e-2}  # bf16 activations and gradients through every layer, and two steps of the optimizer on top
    return {"rel": 1e-2}      # bf16 operands and results, probabilities rounded to bf16 before the second product
