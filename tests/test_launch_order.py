"""CPU: kernels that start under their predecessor, read as text.  Until griddepcontrol.wait the predecessor's stores are not
promised to be visible, and the predecessor may be anyone's, so no value may come from memory before it."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "cold_compress_b200" / "csrc"
LOADS = re.compile(r"ld_weights\(|load8\(|read8\(|__ldg\(|__ldcg\(|load<|Bounded<|cp_async|tma_load|ld\.global|\b[a-z]\.\w+\[|\*\s*[ap]\.")


def _kernels(text):
    """(name, head, body) of every __global__ function."""
    text = re.sub(r"__launch_bounds__\([^)]*\)", "", text)
    for m in re.finditer(r"__global__[^;{]*?\b(\w+)\s*\([^{;]*\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), m.group(0), re.sub(r"//[^\n]*", "", text[m.end():i])


EARLY = [(f.name, name, head, body) for f in sorted((CSRC / "seq").glob("*.cu")) for name, head, body in _kernels(f.read_text()) if "pdl_wait" in body]


def test_the_kernels_are_found():
    launched = sum(len(re.findall(r"launch_under\(", f.read_text())) for f in (CSRC / "seq").glob("*.cu"))
    assert len(EARLY) >= 13 and launched >= len(EARLY)
    assert not any(".nc." in f.read_text() for f in (CSRC / "seq").glob("*.cu*"))


@pytest.mark.parametrize("file,name,head,body", EARLY, ids=[f"{e[0][:-3]}-{e[1]}" for e in EARLY])
def test_nothing_is_read_before_the_wait(file, name, head, body):
    before = body[:body.index("pdl_wait")].replace("g.job[j]", "")      # a job among the kernel's own parameters
    assert not LOADS.search(before), LOADS.search(before)
    assert "launch_dependents" not in before and "pdl_release" not in before


@pytest.mark.parametrize("file,name,head,body", EARLY, ids=[f"{e[0][:-3]}-{e[1]}" for e in EARLY])
def test_no_memory_is_read_through_the_read_only_path(file, name, head, body):
    assert "__restrict__" not in head.replace("__grid_constant__", "")
    assert "__ldg" not in body and "load8(" not in body and "warp_dot" not in body and ".nc." not in body


def test_kernels_that_read_ahead_release_no_one_before_they_have_waited():
    """A kernel may read its cache or its weights ahead because its predecessor does not write them.  That says nothing about
    older kernels, which therefore have to be done: every kernel releases its dependents only after its own wait."""
    gemv = (CSRC / "gemv.cu").read_text()
    assert 0 < gemv.index("pdl_wait();") < gemv.index("pdl_launch_dependents();") and gemv.count("pdl_launch_dependents();") == 1
    lines = [re.sub(r"//.*", "", x).strip() for x in (CSRC / "decode_step.cu").read_text().split("\n")]
    lines = [x for x in lines if x]
    waits, releases = ([i for i, x in enumerate(lines) if call in x] for call in ("pdl_wait();", "pdl_launch_dependents();"))
    assert len(waits) == len(releases) == 2
    assert lines[waits[0]] == "if (!ahead) pdl_wait();" and lines[releases[0]] == "if (!ahead) pdl_launch_dependents();" and waits[0] < releases[0]
    assert lines[waits[1] - 1] == "if (ahead) {" and releases[1] == waits[1] + 1
