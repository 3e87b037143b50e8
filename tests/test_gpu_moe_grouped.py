"""The grouped expert products of a prompt portion at the edges of their tiles: groups of one row, of exactly 128 and of 129,
empty groups, inner and outer sizes that are not whole tiles, with and without a gate."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ids(T, top, n_out, how, gen):
    """Choices [T, top], different within a row."""
    if how == "one":            # every token takes the same experts: the others are empty
        return torch.arange(top, dtype=torch.int32).repeat(T, 1)
    return torch.stack([torch.randperm(n_out, generator=gen)[:top] for _ in range(T)]).to(torch.int32)


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("T, E, F, n, identity, top, how", [
    (5, 64, 64, 4, 0, 2, "any"), (16, 72, 40, 5, 2, 3, "any"), (128, 64, 128, 3, 0, 2, "one"), (129, 136, 264, 3, 0, 1, "one"),
    (300, 200, 136, 16, 2, 4, "any"), (77, 8, 8, 2, 1, 2, "any"), (700, 512, 384, 8, 0, 4, "any"), (33, 1032, 520, 40, 0, 3, "any"),
])
def test_grouped_experts_match_64_bit_products(T, E, F, n, identity, top, how, gated):
    from cold_compress_b200 import _lib, seq_ops
    from cold_compress_b200.detatar import RoutedExperts
    gen = torch.Generator().manual_seed(T + E)
    m = RoutedExperts(E, n, identity, F, top, 1, 1, 0, _lib.ACT_SILU, torch.bfloat16, gated=gated)
    for p in (m.w_gu, m.w_d):
        p.data.copy_(torch.randn(p.shape, generator=gen) * E ** -0.5)
    h = torch.randn(T, E, generator=gen).bfloat16()
    ids = _ids(T, top, n + identity, how, gen)
    m, h, ids = m.cuda(), h.cuda(), ids.cuda()
    assert seq_ops.moe_grouped_serves(m.w_gu, m.w_d, h)
    slot, y = m.expert_rows(ids, h)
    slot, seen = slot.view(T, top), ids < n
    assert torch.equal(slot >= 0, seen) and slot[seen].unique().numel() == int(seen.sum())
    for e in range(n):
        t, k = (ids == e).nonzero(as_tuple=True)
        if not t.numel():
            continue
        up = h[t].double() @ m.w_gu[e].double().t()
        act = torch.nn.functional.silu(up[:, :F]) * (up[:, F:] if gated else 1.0)
        want = act @ m.w_d[e].double().t()
        # the unit's result is rounded to bf16 (2^-9 each, independent), products accumulate in fp32
        assert ((y[slot[t, k].long()].double() - want).norm() / want.norm()).item() <= 2.0 ** -8
