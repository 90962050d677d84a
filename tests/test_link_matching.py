"""Links matched as they are found give the pairs, in the order, that a list of links and a table of positions give."""
import random

import pytest
import torch

from tagseq2tagseq_b200 import CrossDocLinkMaskCreator, DocSpan
from tagseq2tagseq_b200.link_detect import MarkdownLinkDetector

WORDS = ["", " ", "a", "b", " a ", "c)", ")", "x)y", "a)"]


class _Scanned(MarkdownLinkDetector):
    """The device's answer is given: candidates and the tokens behind them."""

    def _scan(self, input_ids):
        cands = self.given
        return cands, [int(t) for mid, _, close in cands for t in input_ids[mid + 1:close + 1]]


@pytest.mark.parametrize("seed", range(30))
def test_matched_links_are_those_of_the_two_steps(seed):
    rng = random.Random(seed)
    detector = _Scanned(lambda ids: "".join(WORDS[i] for i in ids), window_tokens=rng.choice([1, 3, 6]))
    n = rng.randint(1, 40)
    tokens = torch.tensor([rng.randrange(len(WORDS)) for _ in range(n)])
    detector.given = []
    for mid in range(n - 1):                                   # closing places that rise, some of them without a ')' for the growing window to look further
        if rng.random() < 0.6:
            low = detector.given[-1][2] if detector.given else 0
            detector.given.append([mid, mid, min(n - 1, max(mid + 1, low, mid + rng.randint(0, 3)))])
    spans = [DocSpan(i, "", i * 4, i * 4 + 4, False, [], rng.choice(["a", "b", "c", "x", "", "nobody"])) for i in range(n // 4 + 1)]
    creator = CrossDocLinkMaskCreator(detector)
    table = creator._match_links_to_docs(detector.detect_links(tokens), spans)
    assert detector.matched(tokens, creator._index(spans)) == [(pos, doc) for pos in sorted(table) for doc in table[pos]]


def test_a_growing_window_may_close_behind_the_next_link():
    """The first candidate's text has no ')' where the scan closed it and closes three tokens later, behind the second one's."""
    texts = {1: "a", 2: "b", 3: ")", 4: "�"}
    detector = _Scanned(lambda ids: "a b)" if ids == [4, 1, 4, 2, 3] else "".join(texts[i] for i in ids) if ids != [4] and ids[0] != 4 else "b)" if ids == [4, 2] else "?",
                        window_tokens=5)
    tokens = torch.tensor([0, 4, 1, 4, 2, 3, 0, 0])
    detector.given = [[0, 0, 1], [2, 2, 4]]
    spans = [DocSpan(7, "", 0, 1, False, [], "a b"), DocSpan(8, "", 1, 2, False, [], "b")]
    creator = CrossDocLinkMaskCreator(detector)
    links = [tuple(link) for link in detector.detect_links(tokens)]
    assert links == [(6, "a b"), (5, "b")]
    assert detector.matched(tokens, creator._index(spans)) == [(5, 8), (6, 7)]


@pytest.mark.gpu
@pytest.mark.parametrize("where", ["class", "subclass", "object"])
def test_a_matching_of_the_callers_own_is_asked(where, monkeypatch):
    detector = _Scanned(lambda ids: "".join(WORDS[i] for i in ids))
    tokens = torch.tensor([[0, 0, 0, 0, 0, 2, 6, 0]], device="cuda")
    detector.given = [[4, 4, 6]]                               # "a)"
    spans = [DocSpan(0, "", 0, 4, False, [], "a"), DocSpan(1, "", 4, 8, False, [], "b")]
    assert CrossDocLinkMaskCreator(detector)(tokens, spans).link_bits is not None
    calls = []

    def nothing(self, links, doc_spans):
        calls.append([tuple(link) for link in links])
        return {}

    kind = type("Own", (CrossDocLinkMaskCreator,), {"_match_links_to_docs": nothing}) if where == "subclass" else CrossDocLinkMaskCreator
    if where == "class":
        monkeypatch.setattr(CrossDocLinkMaskCreator, "_match_links_to_docs", nothing)
    creator = kind(detector)
    if where == "object":
        creator._match_links_to_docs = nothing.__get__(creator)
    assert creator(tokens, spans).link_bits is None and calls == [[(7, "a")]]
