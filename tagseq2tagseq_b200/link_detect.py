"""Markdown link detector whose token scan runs on the GPU.

Mirror of the reference's ``MarkdownLinkDetector`` (model/graph_traversal/markdown_link_detector.py:19-108): same
constructor arguments, same ``detect_links(input_ids) -> List[LinkInfo]`` and ``index_doc_span`` (the LinkDetector
protocol, model/graph_traversal/link_detector.py:22-84), so it can be handed to ``CrossDocLinkMaskCreator``
unchanged.  The reference walks the sequence with one ``.item()`` per token it looks at; here the positions of every
"[ ... ](" ... ")" candidate come from ``ts2ts_detect_links`` in one pass over the device tensor, and only the few
target tokens of each candidate are decoded (with the reference's own growing-window rule, so the
strings and the non-empty test are the reference's).

The per-token table "this token's bytes contain ')'" is built once from ``decode_fn`` over ``vocab_size`` ids.  It is
exact for byte-level BPE vocabularies (GPT-2's): ')' is a single ASCII byte, which no neighbouring token can change.
"""
from __future__ import annotations

from typing import Any, Callable, Dict, List, Optional, Tuple

import torch

from . import _lib
from .mask_spec import LinkInfo


class MarkdownLinkDetector:
    def __init__(self, decode_fn: Callable[[List[int]], str], window_tokens: int = 50,
                 link_start_token_ids: Optional[List[int]] = None, link_mid_token_id: int = 16151,
                 vocab_size: int = 50257):
        if link_start_token_ids is None:
            link_start_token_ids = [58, 685]  # '[' and ' [' in GPT-2
        if not 1 <= len(set(link_start_token_ids)) <= 8:
            raise ValueError("between 1 and 8 link start token ids are supported")
        self.decode_fn = decode_fn
        self.window_tokens = int(window_tokens)
        self.link_start_token_ids = set(link_start_token_ids)
        self.link_mid_token_id = int(link_mid_token_id)
        self.vocab_size = int(vocab_size)
        self._close_host: Optional[torch.Tensor] = None
        self._close_dev = {}

    def index_doc_span(self, span: Any) -> str:
        """Exact match against ``raw_identifier`` (markdown_link_detector.py:53-55)."""
        return span.raw_identifier

    # ------------------------------------------------------------------ device side
    def _close_flags(self, device: torch.device) -> torch.Tensor:
        if self._close_host is None:
            flags = torch.zeros(self.vocab_size, dtype=torch.uint8)
            for tok in range(self.vocab_size):
                try:
                    if ")" in self.decode_fn([tok]):
                        flags[tok] = 1
                except Exception:  # ids the tokenizer does not know never close a link
                    pass
            self._close_host = flags
        key = (device.type, device.index)
        if key not in self._close_dev:
            self._close_dev[key] = self._close_host.to(device)
        return self._close_dev[key]

    def _scan(self, input_ids: torch.Tensor):
        """({mid, start, close} of every candidate, the tokens of all targets one after the other), as lists."""
        if input_ids.dim() != 1:
            raise ValueError("input_ids must be 1-D")
        if not input_ids.is_cuda:
            raise RuntimeError("the link scan runs on the GPU: input_ids must be a CUDA tensor (there is no CPU path)")
        if input_ids.dtype not in (torch.int32, torch.int64):
            raise TypeError("input_ids must be int32 or int64")
        if input_ids.shape[0] == 0:
            return [], []
        try:
            links, targets = _lib.ops().link_candidates.default(input_ids, self.link_mid_token_id, sorted(self.link_start_token_ids),
                                                                self._close_flags(input_ids.device), 100, self.window_tokens)
        except RuntimeError as e:
            raise _lib.failed_call(e) from None
        return links.tolist(), targets.tolist()

    def candidates(self, input_ids: torch.Tensor) -> List[Tuple[int, int, int]]:
        """(position of '](', position of '[', position of the closing token) for every candidate, ascending."""
        return [tuple(r) for r in self._scan(input_ids)[0]]

    # ------------------------------------------------------------------ protocol
    def detect_links(self, input_ids: torch.Tensor) -> List[LinkInfo]:
        new = tuple.__new__
        return [new(LinkInfo, link) for link in self._links(input_ids)]

    _own_detect_links = detect_links

    def _links(self, input_ids: torch.Tensor):
        """(position after the closing token, target) of every link, one after the other."""
        cands, targets = self._scan(input_ids)
        decode, done = self.decode_fn, 0
        for mid, _start, close in cands:
            end = done + close - mid
            target, closed, _ = decode(targets[done:end]).partition(")")
            done = end
            if not closed:
                # the per-token table promised a ')' that the joint decoding does not show (not a byte-level
                # vocabulary): fall back to the reference's growing window for this candidate
                target, at = self._grow(input_ids[mid + 1:mid + 1 + self.window_tokens].tolist())
                if at < 0:
                    continue
                close = mid + 1 + at
            target = target.strip()
            if target:
                yield close + 1, target

    def matched(self, input_ids: torch.Tensor, index: Dict[str, Tuple[int, int]]) -> List[Tuple[int, int]]:
        """(link_end_pos, document) of every link whose target's document, ``index``'s (doc id, start), starts before it, by position."""
        get, out, last, ascend = index.get, [], 0, True
        for pos, target in self._links(input_ids):
            hit = get(target)
            if hit is not None and hit[1] < pos:
                ascend = ascend and pos >= last
                last = pos
                out.append((pos, hit[0]))
        if not ascend:  # only behind a growing window
            out.sort(key=lambda pair: pair[0])
        return out

    def _grow(self, window: List[int]) -> Tuple[str, int]:
        """(text before ')', index of the token that closes it) of the shortest decodable prefix, or ("", -1)."""
        for j in range(len(window)):
            target, closed, _ = self.decode_fn(window[:j + 1]).partition(")")
            if closed:
                return target, j
        return "", -1
