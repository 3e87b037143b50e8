"""CPU: the fused decode step, read as text, where an order between warps is not something that a run can be expected to show."""
import re
from pathlib import Path

SRC = (Path(__file__).resolve().parent.parent / "cold_compress_b200" / "csrc" / "decode_step.cu").read_text()


def _between(start, end):
    part = SRC[SRC.index(start) + len(start):]
    return re.sub(r"//[^\n]*", "", part[:part.index(end)])


def test_the_exchange_of_candidates_sends_no_logit_from_the_rows():
    """A warp goes on to the softmax, which overwrites the logits, as soon as its own CTA's record is complete.  Other warps may still be
    sending this CTA's record to its peers then, so what they send must lie where the softmax does not write."""
    sent = _between("__syncthreads();  // logits and row maxima visible", "mbar_wait(&xbar[1], 0);")
    assert "st_async_u32(" in sent and not re.search(r"\blg(w)?\s*\[", sent)


def test_the_maximum_of_one_cta_takes_no_logit_from_the_rows():
    """The same where one CTA holds a head: the warps of a query head find its maximum one by one, and the first may be storing."""
    found = _between("mbar_wait(&xbar[1], 0);", "float* lgw = lg + wg * stride;")
    assert "gm = fmaxf(" in found and not re.search(r"\blg\s*\[", found)
