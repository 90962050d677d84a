"""Rules for the waits of the attention kernels that no output shows when they are broken, read from the sources (CPU only)."""
import os
import re

import pytest

from tagseq2tagseq_b200 import build


def _source(name):
    return re.sub(r"//(?! -{20}).*", "", open(os.path.join(build.CSRC, name)).read())


def _unfenced(text):
    """Accesses to tensor memory that a thread may reach after a wait for MMAs without tcgen05.fence::after_thread_sync in between.

    From each wait on a barrier that tcgen05.commit signals the text is followed to the end of the thread's role (a ruled comment).
    A fence counts for its own block and those inside it, and ends the search once it stands where every path passes."""
    bad = []
    for bar in sorted(set(re.findall(r"mma_commit\(&(\w+)", text))):
        for wait in re.finditer(r"mbar_wait\w*\(&%s\b" % bar, text):
            depth, covered = 0, None
            for tok in re.finditer(r"[{}]|// -{20}|tc_fence_after\(\)|(?:tmem_ld|tmem_st|mma_ss|mma_ts)\d+\(", text[wait.end():]):
                word = tok.group()
                if word == "{":
                    depth += 1
                elif word == "}":
                    depth -= 1
                    covered = None if covered is not None and depth < covered else covered
                elif word.startswith("//"):
                    break
                elif word.startswith("tc_fence_after"):
                    if depth <= 0:
                        break
                    covered = depth if covered is None else covered
                elif covered is None:
                    bad.append((bar, text[:wait.start()].count("\n") + 1, word))
                    break
    return bad


@pytest.mark.parametrize("name", ["attn_fwd.cu", "attn_bwd.cu"])
def test_tensor_memory_is_touched_behind_a_fence_after_a_wait_for_mmas(name):
    assert _unfenced(_source(name)) == []


@pytest.mark.parametrize("name,role", [("attn_fwd.cu", "softmax + epilogue"), ("attn_bwd.cu", "exp / dS warps"), ("attn_bwd.cu", "dQ reduction warps")])
def test_warps_whose_lanes_all_wait_get_one_answer(name, role):
    """In roles of whole warps a wait that only some lanes pass would leave the rest missing from the next vote, __syncwarp or
    tensor-memory instruction: a lane's own answer is for a wait that one thread makes alone, or is not looked at."""
    body = re.search(r"// -{20,} %s(.*?)(?=// -{20}|__syncthreads\(\))" % re.escape(role), _source(name), re.S).group(1)
    own = re.findall(r"^.*\b(?:mbar_wait|wait_longer)\(.*$", body, re.M)
    unasked = r"\s*(?:if \(n_tiles > 0\) mbar_wait|if \(!mbar_try_wait\(.*?\)\) wait_longer)\([^;]*;\s*"
    voted = r".*(?:tid == 0 && |__all_sync\(0xffffffffu, mbar_wait\().*"
    assert "mbar_wait_warp(" in body and [line.strip() for line in own if not re.fullmatch(unasked + "|" + voted, line)] == []
