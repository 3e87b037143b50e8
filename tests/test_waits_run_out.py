"""CPU: waits that run out, read as text.  A wait has a limit, and after it a kernel runs to its end.  Its shared and tensor memory then go to
another CTA, so that what it started has to be over: the last products by a commit of their own, the last copies by their barriers,
each waited for whether or not another wait has run out."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "cold_compress_b200" / "csrc"
WITH_TENSOR_MEMORY = [f for f in sorted(CSRC.rglob("*.cu")) if "tcgen05.alloc" in f.read_text()]


def _bare(path):
    return re.sub(r"//[^\n]*", "", path.read_text())


def test_the_kernels_are_found():
    assert {f.name for f in WITH_TENSOR_MEMORY} == {"prefill_attn.cu", "attn_tc_kernels.cu", "moe_tc_kernels.cu"}


@pytest.mark.parametrize("path", WITH_TENSOR_MEMORY, ids=lambda f: f.stem)
def test_products_are_over_before_tensor_memory_is_given_back(path):
    text = _bare(path)
    assert re.search(r"mbar_wait_out\(uint32_t bar, uint32_t parity\) \{\s*for \(uint32_t n = 0; n < WAIT_LIMIT && !mbar_try\w*\(bar, parity\); \+\+n\) \{\}\s*\}", text)
    last = text[text.rindex("mma_commit("):]
    assert re.match(r"mma_commit\((\w+)\);\s*(__syncwarp\(\);\s*)?mbar_wait_out\(\1, 0\);", last)      # nothing on the way asks for `failed`
    assert "tcgen05.mma" not in last and not re.search(r"\bu?mma_[st]s\(", last) and "tcgen05.dealloc" in last


@pytest.mark.parametrize("path", [f for f in WITH_TENSOR_MEMORY if "tma_load" in f.read_text()], ids=lambda f: f.stem)
def test_copies_are_over_before_the_end(path):
    text = _bare(path)
    after = text[[m.end() for m in re.finditer(r"tma_load\w*\(", text)][-1]:]
    drain = re.search(r"\n([^\n]*)for \(int m = [^;]*; m < (\w+); \+\+m\) mbar_wait_out\(FULL[^;]*, \(m / STAGES\) & 1\);", after)
    assert drain and not drain.group(1).strip() and not re.search(r"if \(\*failed\)([^;]*|\s*\{[^}]*)$", after[:drain.start()])


@pytest.mark.parametrize("path", [f for f in WITH_TENSOR_MEMORY if "elect_one()" in f.read_text()], ids=lambda f: f.stem)
def test_lanes_that_elect_one_leave_a_loop_together(path):
    """Loops around elect.sync, which wants all lanes of the warp, ask for `failed` as a warp."""
    text = _bare(path)
    role = text[text.rindex("warp == ", 0, text.index("umma_commit(S_FULL" if "umma_commit(S_FULL" in text else "mma_commit(EMPTY")):text.rindex("elect_one()")]
    heads = re.findall(r"for \(([^;]*;[^;]*;[^{]*)\{", role)
    asking = [h for h in heads if "failed" in h or "lost()" in h]
    assert asking and all("lost()" in h or "__any_sync(0xffffffffu, *failed)" in h for h in asking)
    assert "lost()" not in role or re.search(r"auto lost = \[&\] \{ return __any_sync\(0xffffffffu, \*failed\) != 0; \};", role)
    assert not re.search(r"if \(\*failed\)", role)


def test_one_token_attention_fetches_nothing_more_and_waits_for_what_is_under_way():
    """attn_decode_mma_kernel has a flag of its own: it is raised before a barrier and looked at between that one and the next."""
    text = _bare(CSRC / "seq" / "seq_kernels.cu")
    body = text[text.index("attn_decode_mma_kernel(const CcSeqAttn a"):]
    loop = body[body.index("for (int tile = tile0; tile < tile_end; ++tile) {"):body.index("int* counters")]
    assert loop.count("md_bar_wait(&bars[b][0], turn)") == loop.count("md_bar_wait(&bars[b][1], turn)") == 1
    marked = loop.index("if (!landed) s_lost = 1;")
    met, known, done = (loop.index(x, marked) for x in ("__syncthreads();", "const bool lost = s_lost;", "if (lost) {"))
    assert loop.rindex("md_bar_wait(&bars[b][1], turn)", 0, marked) and met < known < done < loop.index("__syncthreads();", known)      # the same for all threads
    assert "md_bar_wait(" not in loop[marked:done]
    end = loop[done:]
    lost, rest = end[:end.index("break;")], end[end.index("break;"):]
    assert "md_bar_wait(&bars[b][i], turn);" in lost and "md_bar_wait(&bars[b ^ 1][i], ((tile + 1 - tile0) >> 1) & 1);" in lost and "NAN" in lost
    assert "fetch(" not in lost and loop.count("fetch(tile + 1)") == 2 and rest.count("fetch(tile + 1)") == 1      # the other one is of two buffers, before the waits
