"""Prompt attention with score reductions (csrc/prefill_attn.cu) at the edges of its tiles, for every group size, against the
materialised map; tolerances are those of test_gpu_prefill.py, for the same quantities."""
import pytest
import torch

from prefill_utils import assert_close_bf16, check_prefill_y

pytestmark = pytest.mark.gpu


def _inputs(G, D, S, kv=2):
    gen = torch.Generator().manual_seed(1000 * G + 10 * S + D)
    q = torch.randn(1, kv * G, S, D, generator=gen).bfloat16()
    k = torch.randn(1, kv, S, D, generator=gen).bfloat16()
    return q, k, torch.randn(1, kv, S, D, generator=gen).bfloat16()


def _check(q, k, v, what):
    from cold_compress_b200.attention_utils import prefill_attention_stats
    from oracle.prefill import full_map, reductions
    S, D = q.shape[2], q.shape[3]
    windows = (1, max(2, S // 3), S + 5)
    y, st = prefill_attention_stats(q.cuda(), k.cuda(), v.cuda(), obs_len=16, windows=windows)
    y_ref, pooled = full_map(q, k, v)
    ref = reductions(pooled, 16, windows)
    check_prefill_y(y[0].reshape(-1, D), y_ref[0].reshape(-1, D), what)
    assert_close_bf16(st.col_sum[0], ref.col_sum[0], f"{what} col_sum", max_ulp=1.0, min_equal=0.90, floor=2.0 ** -14)
    assert_close_bf16(st.obs_mean[0], ref.obs_mean[0], f"{what} obs_mean", max_ulp=1.0, min_equal=0.90, floor=2.0 ** -14)
    for w in windows:
        assert torch.allclose(st.band_sum[w].cpu(), ref.band_sum[w], rtol=1e-2, atol=2e-3), f"{what} band {w}"


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("G", [1, 2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("S", [1, 15, 33, 127, 128, 129, 256, 391])
def test_every_group_at_the_edges_of_tiles(G, D, S):
    _check(*_inputs(G, D, S), f"G {G} D {D} S {S}")


@pytest.mark.parametrize("G,D", [(4, 128), (7, 64)])
def test_maxima_that_rise_from_tile_to_tile(G, D):
    """Every tile's maximum lies further above the ones before than a sum's reference may: sums are formed again."""
    q, k, v = _inputs(G, D, 600)
    q, k = torch.ones_like(q) + 0.1 * q, (k + torch.arange(600).view(1, 1, -1, 1) / 40).bfloat16()
    _check(q, k, v, "rising")
    _check(q, k.flip(2), v, "falling")


@pytest.mark.parametrize("G,D,S", [(7, 128, 145), (3, 64, 161), (4, 128, 70)])
def test_logits_of_minus_infinity(G, D, S):
    """Keys that no query gives any weight, and rows of the tile without a query or a head, whose logits are NaN there."""
    q, k, v = _inputs(G, D, S)
    q[..., 0] = q[..., 0].abs() + 1
    k[0, :, 5::7, 0] = float("-inf")
    _check(q, k, v, "minus infinity")


def test_without_statistics_in_fp32():
    from cold_compress_b200.attention_utils import prefill_attention
    q, k, v = (t.cuda() for t in _inputs(5, 128, 391))
    y = prefill_attention(q, k, v)
    w = torch.matmul(q.float(), k.float().repeat_interleave(5, 1).transpose(2, 3)) * 128 ** -0.5
    w = w.masked_fill(torch.ones(391, 391, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    want = torch.softmax(w, -1) @ v.float().repeat_interleave(5, 1)
    # one rounding of a weight and one of the result: 2^-9 of the largest value each, and half as much again for sums
    assert (y.float() - want).abs().max() < 3 * 2.0 ** -9 * v.float().abs().max()


@pytest.mark.parametrize("G,D,S", [(4, 128, 40), (1, 64, 300), (8, 128, 129)])
def test_windows_of_no_token_and_of_every_token(G, D, S):
    """A row i counts for key j while i - j < w: none does for w <= 0, all do for any w of at least S."""
    from cold_compress_b200.attention_utils import prefill_attention_stats
    q, k, v = (t.cuda() for t in _inputs(G, D, S))
    top = 2 ** 31 - 1
    _, st = prefill_attention_stats(q, k, v, obs_len=16, windows=(0, -3, -top - 1, top))
    for w in (0, -3, -top - 1):
        assert not st.band_sum[w].any(), f"band {w}"
    assert torch.equal(st.band_sum[top].to(torch.bfloat16), st.col_sum[0])


@pytest.mark.parametrize("S,obs_len", [(7, 16), (15, 16), (40, 1), (40, 3), (391, 7), (391, 16), (391, 100)])
def test_sums_in_bf16_are_the_rounded_sums(S, obs_len):
    """Bit for bit what tensor operations make of the fp32 sums, for means over any number of rows."""
    from cold_compress_b200 import _lib, ops
    q, k, v = (t[0].cuda() for t in _inputs(4, 64, S))
    n = min(obs_len, S)
    ws = torch.empty(ops.prefill_attention_workspace(S, 2, 4, n, 0), dtype=torch.uint8, device="cuda")
    got = []
    for dtype in (torch.float32, torch.bfloat16):
        col, obs = (torch.full((2, S), 7.0, dtype=dtype, device="cuda") for _ in range(2))
        ops.prefill_attention(q, k, v, torch.empty_like(q), _lib.ATTN_NAIVE_BF16, n, [], col, obs, None, ws)
        got.append((col, obs))
    (col, obs), (col16, obs16) = got
    assert torch.equal(col16, col.bfloat16()) and torch.equal(obs16, (obs / n).bfloat16())


@pytest.mark.parametrize("G,QB,D", [(1, 128, 64), (2, 64, 128), (4, 32, 128), (7, 16, 64)])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("row", [0, 37, 130])
def test_rows_that_are_no_numbers(G, QB, D, value, row):
    """A query whose logits are NaN or +inf: its row of y, and the sums over every key before the end of its block of queries."""
    from cold_compress_b200.attention_utils import prefill_attention_stats
    from oracle.prefill import full_map, reductions
    S, windows = 200, (150, 300)
    q, k, v = _inputs(G, D, S)
    k[..., 0] = k[..., 0].abs() + 1                  # +inf times these: no key's logit is -inf
    q[0, 0, row, 0] = value
    y, st = prefill_attention_stats(q.cuda(), k.cuda(), v.cuda(), obs_len=100, windows=windows)
    _, pooled = full_map(q, k, v)
    assert y[0, 0, row].isnan().all() and int(y.isnan().sum()) == D      # (the restatement's product on the CPU takes it on to a neighbour)
    end = min(S, (row // QB + 1) * QB)
    assert pooled[0, 0, row].isnan().all() and int(pooled.isnan().sum()) == S
    pooled[0, 0, row, end:] = 0                      # not visited
    ref = reductions(pooled, 100, windows)
    for got, want, what in ((st.col_sum[0].cpu(), ref.col_sum[0], "col_sum"), (st.obs_mean[0].cpu(), ref.obs_mean[0], "obs_mean")):
        assert torch.equal(got.isnan(), want.isnan()), what
        assert_close_bf16(got.nan_to_num(), want.nan_to_num(), what, max_ulp=1.0, min_equal=0.90, floor=2.0 ** -14)
    for w in windows:
        inside = (row - torch.arange(S)) < w         # the kernel leaves out what lies outside, the restatement multiplies it by zero
        assert torch.equal(st.band_sum[w][0].cpu().isnan(), (torch.arange(S) < end) & inside)
        assert not st.band_sum[w][1:].isnan().any()


@pytest.mark.parametrize("G,D", [(1, 64), (3, 128), (8, 64)])
@pytest.mark.parametrize("S", [391, 512])
def test_bands_whose_edges_lie_anywhere_in_a_tile(G, D, S):
    """Tiles of keys inside a window, outside of it and crossed by its edge, around the sizes of tiles and of blocks of queries."""
    from cold_compress_b200.attention_utils import prefill_attention_stats
    from oracle.prefill import full_map, reductions
    q, k, v = _inputs(G, D, S)
    ref = reductions(full_map(q, k, v)[1], 16, every := (1, 2, 16, 31, 32, 33, 63, 64, 96, 127, 128, 129, 160, 255, 256, 257, 300, S - 1, S, S + 1))
    for i in range(0, len(every), 4):
        _, st = prefill_attention_stats(q.cuda(), k.cuda(), v.cuda(), obs_len=16, windows=every[i:i + 4])
        for w in every[i:i + 4]:
            assert torch.allclose(st.band_sum[w].cpu(), ref.band_sum[w], rtol=1e-2, atol=2e-3), f"band {w}"
