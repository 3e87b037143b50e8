"""Segments of the matrix-state recurrence where a number is infinite or none, and decays whose product over a batch or a segment
underflows although none of them is zero: what comes out is infinite or no number exactly where it is token after token."""
import pytest
import torch

pytestmark = pytest.mark.gpu
INF, NAN = float("inf"), float("nan")


def _spoil(where, value, r, k, v, raw, S, T, HD, D):
    t, c = T // 3, HD - D // 2            # in the last head
    if where == "state":
        S[-1, 1, D // 2] = value
    elif where == "two rows of the state":
        S[-1, 1, D // 2], S[0, 0, 0], S[0, 1, 0] = value, value, -value
    else:
        {"r": r, "k": k, "v": v, "raw": raw}[where][t, c] = value


@pytest.mark.parametrize("T, H, D", [(300, 2, 64), (513, 3, 40), (700, 1, 128), (4096, 2, 16)])
@pytest.mark.parametrize("w0", [-4.0, 0.5, 1.5])
@pytest.mark.parametrize("where", ["state", "two rows of the state", "r", "k", "v", "raw"])
@pytest.mark.parametrize("value", [INF, -INF, NAN])
def test_what_is_not_finite_is_where_it_is_token_after_token(T, H, D, w0, where, value, monkeypatch):
    from cold_compress_b200 import seq_ops
    gen = torch.Generator(device="cuda").manual_seed(T + D)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    r, k, v, raw = (randn(T, H * D) for _ in range(4))
    base, u, S0 = w0 + 0.3 * randn(H * D), randn(H * D), randn(H, D, D)
    k[5], r[7], v[9] = 0.0, 0.0, 0.0
    _spoil(where, value, r, k, v, raw, S0, T, H * D, D)

    def run(segments_from):
        monkeypatch.setattr(seq_ops, "WKV_SEGMENTS_FROM", segments_from)
        state, o = S0.clone(), torch.empty(T, H * D, device="cuda")
        seq_ops.wkv(r, k, v, raw, base, u, state, o, H, D)
        return o, state

    for cut, plain in zip(run(1), run(1 << 30)):
        assert torch.equal(cut.isnan(), plain.isnan()) and torch.equal(cut.isposinf(), plain.isposinf()) and torch.equal(cut.isneginf(), plain.isneginf())
        known = plain.isfinite()
        # the same sums in another order, in fp32
        assert ((cut[known].double() - plain[known].double()).norm() <= 1e-5 * plain[known].double().norm())
