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
    unasked = r"\s*if \((?:n_tiles > 0 && )?!mbar_try_wait\(.*?\)\) wait_longer\([^;]*;\s*"
    lone_or_voted = r".*(?:tid == 0 && |row == 0 && |__all_sync\(0xffffffffu, mbar_wait\().*"
    assert "mbar_wait_warp(" in body and [line.strip() for line in own if not re.fullmatch(unasked + "|" + lone_or_voted, line)] == []


@pytest.mark.parametrize("name", ["attn_fwd.cu", "attn_bwd.cu"])
def test_roles_meet_only_where_a_thread_that_has_left_is_not_waited_for(name):
    """A named barrier (or __syncthreads inside a role) waits for a fixed number of threads without a limit; a thread whose bounded
    wait ran out never comes."""
    text = _source(name)
    roles = text[text.index("// ---"):text.index("if (*abort_")]
    assert not re.search(r"\b(?:bar|barrier)\.(?:cta\.)?(?:sync|red|arrive)", text) and roles.count("__syncthreads") == 1


def test_scores_overwrite_the_probabilities_of_the_last_tile_once_their_product_is_complete():
    """With one S^T buffer S^T(i+1) goes over P^T(i), which dV(i), an MMA with another accumulator, reads: only its completion orders the
    two, not the order of issue."""
    text = _source("attn_bwd.cu")
    one_buffer = text[text.index("if (Cfg::kSBufs == 1 && more) {"):]
    assert re.match(r"[^{]*\{[^}]*mbar_wait\(&bar_gv\[i % Cfg::kDoStages\], \(i / Cfg::kDoStages\) & 1,[^}]*issue_st\(i \+ 1,", one_buffer)


@pytest.mark.parametrize("name,code,uses", [("attn_fwd.cu", "1901", r"fwd_setup<D>\(at\)"), ("attn_bwd.cu", "2900", r"mbar_init\(|tmem_alloc\(")])
def test_a_misplaced_shared_memory_window_is_refused_before_it_is_written(name, code, uses):
    kernel = re.search(r"__global__ void __launch_bounds__\(\w+, 1\)\nattn_\w+_kernel\(.*?\n}", _source(name), re.S).group()
    refused = re.search(r"atomicCAS\([\w.]*status, 0, %s\);(?:\s*wait_previous\(\);)?\s*return;" % code, kernel)
    assert refused and refused.end() < re.search(uses, kernel).start() and "wait_previous();" in kernel[:refused.end()]


def _unsettled(text):
    """Pointers that a kernel with a wait of its own for the launch before it reads through the read-only path without settled() behind that wait: its
    __restrict__ parameters to constant memory, and what it passes to __ldg.  The rows of a gradient that an embedding adds up are found through indices that it has loaded."""
    bad = []
    for kernel in re.finditer(r"__global__ void (?:__launch_bounds__\([^)]*\) )?(\w+)\((.*?)\) \{\n(.*?)\n\}", text, re.S):
        name, params, body = kernel.groups()
        wait = re.search(r"\bwait_previous\(\);", body)
        if wait is None:  # the kernels inside a chain: what they read without having made it was complete before the chain
            assert "after_previous();" in body, name
            continue
        pointers = set(re.findall(r"const \w+\* __restrict__ (\w+)", params)) | set(re.findall(r"__ldg\((?:reinterpret_cast<[^>]*>\()?&?(\w+)", body))
        bad += [(name, p) for p in sorted(pointers - ({"dx"} if name == "embedding_bwd_kernel" else set())) if not re.search(r"\b%s = settled\(" % p, body[wait.end():])]
    return bad


@pytest.mark.parametrize("name", ["adamw.cu", "block_map.cu", "link_scan.cu", "lm_fused.cu"])
def test_read_only_loads_stay_behind_the_wait_for_the_launch_before(name):
    """A read-only load whose address is known at the start may be moved up across the wait (the attention kernels' addresses come from what they load)."""
    text = _source(name)
    assert len(re.findall(r"__global__", text)) == len(re.findall(r"\b(?:wait|after)_previous\(\);", text)) and _unsettled(text) == []


@pytest.mark.gpu
@pytest.mark.parametrize("d", [64, 128])
# pairs of query tiles; query tiles that two teams share, and those as the lists call for them, the entry one of either team's
@pytest.mark.parametrize("h,place", [(16, 1), (4, 0), (4, 1), (4, 2), (8, 1), (8, 2)])
def test_a_list_entry_that_is_no_tile_ends_in_a_status(d, h, place):
    """The forward's own check of its lists: the block that meets the entry (as its second or a later item, or its only one) drains and
    leaves, the code is in the status word, the same plan with the entry put right serves the next call, and a plan built again too."""
    import torch
    from tagseq2tagseq_b200 import build_block_map, read_status
    from tagseq2tagseq_b200.attention import masked_attn
    t, nb = 4096, 32
    dev = torch.device("cuda")
    doc = torch.zeros((1, t), dtype=torch.int32, device=dev)
    g = torch.Generator(device=dev).manual_seed(1)
    q, k, v = (torch.randn(1, h, t, d, generator=g, device=dev).bfloat16() for _ in range(3))
    want, want_lse = masked_attn(q, k, v, doc, plan=build_block_map(doc).plan)
    plan = build_block_map(doc).plan
    at = 256                                                    # the layout of csrc/plan.h: status, run_cnt, runs, state, fwd_cnt, fwd_idx
    for size in (nb * 4, nb * 128 * 16, nb * nb):
        at = -(-(at + size) // 256) * 256
    cnt = plan.view(torch.int32)[at // 4:at // 4 + nb]
    lists = plan.view(torch.int32)[(at + 256) // 4:][:nb * nb].view(nb, nb)
    assert cnt.tolist() == list(range(1, nb + 1)) and (lists[3, :4] & ~(1 << 30)).tolist() == [0, 1, 2, 3]
    right = lists[2, place].item()
    lists[2, place] = nb + 5                                    # of the last pair but one in the order of launch
    masked_attn(q, k, v, doc, plan=plan)
    assert read_status(plan) in (1014, 1038)                    # the producer or a softmax warp, whoever came first
    assert plan.view(torch.int32)[8:10].tolist() == [0, 0]      # the counters that items are drawn from start again
    lists[2, place] = right
    out, lse = masked_attn(q, k, v, doc, plan=plan)
    assert torch.equal(out, want) and torch.equal(lse, want_lse)
    out, lse = masked_attn(q, k, v, doc, plan=build_block_map(doc).plan)
    assert torch.equal(out, want) and torch.equal(lse, want_lse)
