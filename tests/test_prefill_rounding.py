"""The packed form of a logit's two roundings (csrc/prefill_attn.cu: round_logits) over every bf16 number."""
import re
from pathlib import Path

import numpy as np


def _bf16(x):
    """double -> nearest bf16 (ties to even, subnormals kept), as a double."""
    _, e = np.frexp(x)
    unit = np.ldexp(1.0, np.maximum(e - 8, -133))
    r = np.rint(x / unit) * unit
    return np.where(np.abs(r) >= 2.0 ** 128, np.copysign(np.inf, x), r)


def test_packed_scaling_of_logits_rounds_as_fp32_does():
    src = (Path(__file__).resolve().parent.parent / "cold_compress_b200" / "csrc" / "prefill_attn.cu").read_text()
    hi, lo, eighth = (np.array([int(re.search(rf"{n} = 0x([0-9a-f]{{4}})\1u", src).group(1), 16) << 16], dtype=np.uint32).view(np.float32)[0].astype(float)
                      for n in ("SCALE128_HI", "SCALE128_LO", "SCALE64"))
    x32 = (np.arange(65536, dtype=np.uint32) << 16).view(np.float32)
    x32 = x32[np.isfinite(x32)]
    x = x32.astype(float)
    want = _bf16((x32 * np.float32(1 / np.sqrt(128.0))).astype(float))
    got = _bf16(x * hi + _bf16(x * lo))       # x hi and the sum are exact in double
    assert np.array_equal(got[np.abs(x) >= 2.0 ** -100], want[np.abs(x) >= 2.0 ** -100])
    assert np.abs(got - want).max() < 2.0 ** -126
    assert eighth == 0.125
