"""The matrix-state recurrence gives the same bits however a sequence is cut into calls that go token after token (shorter than
WKV_SEGMENTS_FROM, or of heads that are not cut into segments): below and above the length from which the decays come from a launch of
their own, across staged batches of 32 tokens, with head sizes that are not whole column tiles or 16-byte vectors.  Calls whose segments
go side by side agree with them to rounding."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H, D", [(1, 8), (2, 16), (3, 33), (2, 64), (1, 72), (2, 128), (1, 200)])
def test_any_cut_of_a_sequence_gives_the_same_bits(H, D):
    from cold_compress_b200 import seq_ops
    T = 2 * seq_ops.WKV_DECAY_FROM + 37
    assert T < seq_ops.WKV_SEGMENTS_FROM
    gen = torch.Generator(device="cuda").manual_seed(D)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    r, k, v, wraw = (randn(T, H * D) for _ in range(4))
    w0, u = randn(H * D) - 1.5, 0.5 * randn(H * D)

    def run(portions):
        state, out, at = torch.zeros(H, D, D, device="cuda"), [], 0
        for m in portions:
            o = torch.empty(m, H * D, device="cuda")
            seq_ops.wkv(*(t[at:at + m].contiguous() for t in (r, k, v, wraw)), w0, u, state, o, H, D)
            out.append(o)
            at += m
        assert at == T
        return torch.cat(out), state

    whole, state = run((T,))
    n = seq_ops.WKV_DECAY_FROM
    for portions in ((1, n - 1, n, T - 2 * n), (n + 1, 31, T - n - 32), (33,) * (T // 33) + (T % 33,) * (T % 33 > 0)):
        got, s = run(portions)
        assert torch.equal(got, whole) and torch.equal(s, state)
    w = torch.exp(-torch.exp(wraw.double() + w0.double())).view(T, H, D, 1)
    S, want = torch.zeros(H, D, D, dtype=torch.float64, device="cuda"), []
    rd, kd, vd, ud = (t.double().view(-1, H, D) for t in (r, k, v, u))
    for t in range(T):
        kv = kd[t].unsqueeze(-1) * vd[t].unsqueeze(-2)
        want.append(torch.einsum("hij,hi->hj", S + ud[0].unsqueeze(-1) * kv, rd[t]).reshape(-1))
        S = w[t] * S + kv
    want = torch.stack(want)
    # D products summed in fp32 and a state that forgets: a few roundings of the sum's size
    assert ((whole.double() - want).norm() / want.norm()).item() <= 4 * 2.0 ** -23 and ((state.double() - S).norm() / S.norm()).item() <= 4 * 2.0 ** -23


@pytest.mark.parametrize("H, D", [(3, 24), (9, 256), (10, 200), (46, 64), (49, 40), (80, 64), (33, 128)])
def test_column_tiles_of_both_widths_give_the_same_bits(H, D):
    """More heads than one wave of CTAs takes: short portions walk tiles of 32 columns, a long one 16 or 32 by the number of
    heads, a few heads at a time always 16 (or a single tile of narrow heads)."""
    from cold_compress_b200 import seq_ops
    T = seq_ops.WKV_DECAY_FROM + 5
    gen = torch.Generator(device="cuda").manual_seed(D + H)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    r, k, v, wraw = (randn(T, H, D) for _ in range(4))
    w0, u = randn(H, D) - 1.5, 0.5 * randn(H, D)

    def run(heads, portions):
        n, state, out, at = heads.stop - heads.start, torch.zeros(heads.stop - heads.start, D, D, device="cuda"), [], 0
        for m in portions:
            o = torch.empty(m, n * D, device="cuda")
            seq_ops.wkv(*(t[at:at + m, heads].reshape(m, n * D).contiguous() for t in (r, k, v, wraw)), w0[heads].reshape(-1).contiguous(),
                        u[heads].reshape(-1).contiguous(), state, o, n, D)
            out.append(o.view(m, n, D))
            at += m
        return torch.cat(out), state

    whole, state = run(slice(0, H), (T,))
    cut, cut_state = run(slice(0, H), (1, 30, T - 31))
    assert torch.equal(cut, whole) and torch.equal(cut_state, state)
    for h in range(0, H, 2):
        some, s = run(slice(h, min(h + 2, H)), (T,))
        assert torch.equal(some, whole[:, h:h + 2]) and torch.equal(s, state[h:h + 2])


@pytest.mark.parametrize("H, D", [(2, 64), (5, 100), (3, 20)])
def test_a_state_goes_through_calls_of_both_kinds(H, D):
    """One sequence in segmented and in shorter calls, the state carried through, against one call and against 64 bits."""
    from cold_compress_b200 import _lib, seq_ops
    cuts = [(956,), (300, 1, 255, 400), (255, 256, 1, 444), (64, 500, 63, 329)]
    for n in (256, 300, 400, 444, 500, 956):
        assert n >= seq_ops.WKV_SEGMENTS_FROM and (_lib.load_seq().cc_seq_wkv_segments_workspace(n, H, D) > 0 or D == 100 and n < 384)
    T = sum(cuts[0])
    gen = torch.Generator(device="cuda").manual_seed(D)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    r, k, v, wraw = (randn(T, H * D) for _ in range(4))
    w0, u, S0 = randn(H * D) - 2.5, 0.5 * randn(H * D), randn(H, D, D)
    w = torch.exp(-torch.exp(wraw.double() + w0.double())).view(T, H, D, 1)
    S, want = S0.double(), []
    rd, kd, vd, ud = (t.double().view(-1, H, D) for t in (r, k, v, u))
    for t in range(T):
        kv = kd[t].unsqueeze(-1) * vd[t].unsqueeze(-2)
        want.append(torch.einsum("hij,hi->hj", S + ud[0].unsqueeze(-1) * kv, rd[t]).reshape(-1))
        S = w[t] * S + kv
    want = torch.stack(want)
    for portions in cuts:
        state, out, at = S0.clone(), [], 0
        for m in portions:
            o = torch.empty(m, H * D, device="cuda")
            seq_ops.wkv(*(t[at:at + m].contiguous() for t in (r, k, v, wraw)), w0, u, state, o, H, D)
            out.append(o)
            at += m
        # D products summed in fp32 over a state of some dozens of tokens: a few roundings of the sum's size
        assert at == T and ((torch.cat(out).double() - want).norm() / want.norm()).item() <= 8 * 2.0 ** -23
        assert ((state.double() - S).norm() / S.norm()).item() <= 8 * 2.0 ** -23
