"""CPU: what cc_prefill_attention refuses before it touches a device."""
import ctypes as C

import pytest


def _args(**more):
    from cold_compress_b200 import _lib
    a = _lib.CcPrefillAttnArgs()
    for t in "qkvy":
        setattr(a, t, 4096)
        setattr(a, f"{t}_stride_s", 64)
        setattr(a, f"{t}_stride_h", 64 * 32)
    a.seq_len, a.n_kv_heads, a.q_per_kv, a.head_dim, a.attn_mode = 32, 1, 1, 64, _lib.ATTN_NAIVE_BF16
    for name, value in more.items():
        setattr(a, name, value)
    return a


@pytest.mark.parametrize("value", [2, -1, 0x3F800000])
def test_a_form_of_the_sums_that_there_is_not(value):
    """The field had no meaning in the first version of the structure: what a caller left there must not choose a form."""
    from cold_compress_b200 import _lib
    lib = _lib.load()
    assert lib.cc_abi_version() == _lib.ABI_VERSION >= 2
    for sums in (None, 8192):
        a = _args(stats_bf16=value, col_sum=sums)
        assert lib.cc_prefill_attention(C.byref(a), None) < 0 and b"stats_bf16" in lib.cc_last_error()
