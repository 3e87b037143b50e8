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


def test_an_evicting_hybrid_head_looks_at_its_own_slots_only():
    """The count of a head that appends goes on beyond its last slot, so it is no bound for a walk over slots."""
    walk = _between("cache.py:844-894", "ckey = k < ckey ? k : ckey;")
    assert "if (s >= live_limit) continue;" in walk and "hyb_cts)" not in walk
    import torch
    from oracle.oracle import OracleCache
    H, L = 3, 20
    oc = OracleCache("hybrid", H, 1, 64, L, hybrid_strategies=[{"strategy": "special_punc_heavy_hitter", "heavy_hitter_frac": 0.2}])
    oc.set_head_strategies([0] * H)
    oc.mask[:], oc.pos[:], oc.cache_cts[:] = True, torch.arange(L, dtype=torch.int32), L
    gen, seen = torch.Generator().manual_seed(0), []
    for t in range(12):
        q, k, v = (torch.randn(H, 64, generator=gen).to(torch.bfloat16) for _ in range(3))
        seen.append(oc.decode_step(q, k, v, L + t, is_punc=t % 3 == 0)[1])
    assert int(oc.cache_cts.max()) > L + 1 and int(torch.stack(seen).max()) < L
