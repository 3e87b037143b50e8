"""The grouped expert products on pairs of CTAs (width 2048 and more, 160 rows an expert and more): groups of exactly 256 rows, of one
more and one less, of half a tile, empty ones, inner and outer sizes that are not whole tiles; the check and its bound are those of
test_gpu_moe_grouped.py."""
import pytest

from test_gpu_moe_grouped import test_grouped_experts_match_64_bit_products as _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("T, E, F, n, identity, top, how", [
    (256, 2048, 128, 3, 0, 2, "one"), (257, 2048, 136, 3, 0, 2, "one"), (255, 2056, 264, 2, 0, 1, "any"), (384, 2048, 40, 2, 1, 1, "any"), (385, 2048, 8, 2, 0, 1, "one"),
    (700, 2120, 520, 9, 2, 4, "any"), (1500, 2048, 72, 16, 2, 4, "any"),
])
def test_pairs_match_64_bit_products(T, E, F, n, identity, top, how, gated):
    _check(T, E, F, n, identity, top, how, gated)
