"""Segments of the matrix-state recurrence side by side, against the recurrence in 64 bits and against token after token: sizes that
are not whole batches, tiles or segments, states that are not empty, decays from almost one to zero."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(r, k, v, w, u, S):
    T, (H, D) = r.shape[0], u.shape
    r, k, v, w = (t.double().view(T, H, D) for t in (r, k, v, w))
    out, S = [], S.double()
    for t in range(T):
        kv = k[t].unsqueeze(-1) * v[t].unsqueeze(-2)
        out.append(torch.einsum("hij,hi->hj", S + u.double().unsqueeze(-1) * kv, r[t]).reshape(-1))
        S = w[t].unsqueeze(-1) * S + kv
    return torch.stack(out), S


@pytest.mark.parametrize("T, H, D", [(33, 1, 64), (64, 3, 4), (257, 2, 64), (300, 5, 72), (511, 1, 128), (290, 40, 20), (1000, 2, 100), (260, 150, 64)])
@pytest.mark.parametrize("w0", [-9.0, -2.0, 4.0])
def test_segments_against_the_recurrence(T, H, D, w0, monkeypatch):
    from cold_compress_b200 import _lib, seq_ops
    assert _lib.load_seq().cc_seq_wkv_segments_workspace(T, H, D) > 0
    gen = torch.Generator(device="cuda").manual_seed(T + D)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    r, k, v, raw = (randn(T, H * D) for _ in range(4))
    base, u, S0 = w0 + randn(H * D), 0.5 * randn(H, D), randn(H, D, D)
    want, S = _exact(r, k, v, torch.exp(-torch.exp(raw.double() + base.double())), u, S0)

    def run(segments_from):
        monkeypatch.setattr(seq_ops, "WKV_SEGMENTS_FROM", segments_from)
        state, o = S0.clone(), torch.empty(T, H * D, device="cuda")
        seq_ops.wkv(r, k, v, raw, base, u.reshape(-1).contiguous(), state, o, H, D)
        return [((got.double() - exact).norm() / exact.norm()).item() for got, exact in ((o, want), (state, S))]

    cut, plain = run(1), run(1 << 30)
    # fp32 sums of D products over a state that keeps up to T tokens: a random walk of T + D roundings of 2^-24; and the decays
    # themselves are numbers of 32 bits, each up to 2^-24 off, of which up to T multiply a token that is kept (w0 = -9)
    bound = 2.0 ** -24 * ((T + D) ** 0.5 + T)
    assert max(cut) <= bound
    assert all(a <= 1.25 * b + 2.0 ** -26 for a, b in zip(cut, plain))      # and no further off than token after token


@pytest.mark.parametrize("T, H, D", [(1100, 128, 64), (901, 128, 60), (420, 128, 128), (259, 500, 64), (384, 230, 100)])
def test_eight_segments_an_sm_against_the_recurrence(T, H, D, monkeypatch):
    """Long enough for the second cut, among them heads that six segments an SM would leave uncut."""
    test_segments_against_the_recurrence(T, H, D, -2.0, monkeypatch)


def test_what_is_not_served_goes_token_after_token():
    from cold_compress_b200 import _lib, seq_ops
    lib = _lib.load_seq()
    assert [lib.cc_seq_wkv_segments_workspace(*s) for s in ((400, 2, 33), (400, 2, 132), (32, 2, 64), (400, 900, 64))] == [0] * 4
    T, H, D = 400, 2, 33                                     # not a multiple of 4: never cut
    gen = torch.Generator(device="cuda").manual_seed(1)
    rows = [torch.randn(T * H * D + 1, device="cuda", generator=gen) for _ in range(4)]
    base, u = torch.randn(H * D, device="cuda", generator=gen) - 2, torch.randn(H * D, device="cuda", generator=gen)

    def run(shift):                                          # rows that start 4 bytes after a 16-byte boundary, and not
        args = [(t[1:] if shift else t[1:].clone()).view(T, H * D) for t in rows]
        state, o = torch.zeros(H, D, D, device="cuda"), torch.empty(T, H * D, device="cuda")
        seq_ops.wkv(*args, base, u, state, o, H, D)
        return o, state

    for a, b in zip(run(True), run(False)):
        assert torch.equal(a, b)
    w = _lib.CcSeqWkv()
    assert lib.cc_seq_wkv_segments(w, None, 0, None) < 0 and b"wkv_segments" in lib.cc_seq_last_error()


@pytest.mark.parametrize("T, H, D", [(257, 3, 64), (400, 2, 100), (300, 5, 20)])
def test_rows_and_a_state_on_any_boundary_of_a_float_give_the_same_bits(T, H, D):
    from cold_compress_b200 import _lib, seq_ops
    assert _lib.load_seq().cc_seq_wkv_segments_workspace(T, H, D) > 0 and T >= seq_ops.WKV_SEGMENTS_FROM
    gen = torch.Generator(device="cuda").manual_seed(D)
    rows = [torch.randn(T, H * D, device="cuda", generator=gen) for _ in range(4)]
    base, u, S0 = torch.randn(H * D, device="cuda", generator=gen) - 2, torch.randn(H * D, device="cuda", generator=gen), torch.randn(H, D, D, device="cuda", generator=gen)

    def at(t, floats):
        held = torch.empty(t.numel() + 4, device="cuda")
        held[floats:floats + t.numel()] = t.reshape(-1)
        return held[floats:floats + t.numel()].view(t.shape)

    def run(*floats):
        args, state, o = [at(t, n) for t, n in zip(rows, floats)], at(S0, floats[4]), at(torch.zeros(T, H * D, device="cuda"), floats[5])
        seq_ops.wkv(*args, base, u, state, o, H, D)
        return o, state

    want = run(0, 0, 0, 0, 0, 0)
    for floats in ((1, 0, 0, 0, 0, 0), (0, 2, 0, 0, 0, 0), (0, 0, 3, 0, 0, 0), (0, 0, 0, 1, 0, 0), (0, 0, 0, 0, 1, 0), (1, 2, 3, 1, 2, 3)):
        for a, b in zip(run(*floats), want):
            assert torch.equal(a, b), floats
