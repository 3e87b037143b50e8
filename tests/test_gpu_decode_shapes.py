"""The fused decode step at the edges of its plans, bit for bit against the oracle: one CTA per head, clusters of every size, rows that end
inside a chunk or a pair, chunks walked as one run and through a ring that is refilled, one warp per query head and several."""
import pytest

from test_gpu_parity import _seeded_state_run

pytestmark = pytest.mark.gpu

SHAPES = [  # strategy, KV heads, query heads per KV head, head size, slots, filled
    ("recent_global", 8, 4, 128, 15, 15), ("heavy_hitter", 3, 1, 64, 16, 9), ("l2", 8, 8, 128, 17, 17), ("heavy_hitter", 4, 7, 128, 33, 33),
    ("recent_global", 2, 7, 64, 47, 20), ("l2", 1, 1, 64, 65, 65), ("heavy_hitter", 8, 8, 64, 97, 97), ("recent_global", 8, 1, 128, 129, 129),
    ("heavy_hitter", 8, 4, 128, 255, 255), ("l2", 4, 7, 128, 257, 250), ("heavy_hitter", 5, 6, 128, 385, 385), ("recent_global", 2, 7, 64, 511, 511),
    ("heavy_hitter", 8, 2, 128, 1023, 1023), ("l2", 8, 4, 128, 1025, 1025), ("heavy_hitter", 16, 2, 128, 700, 700), ("recent_global", 64, 1, 64, 1500, 1500),
]


@pytest.mark.parametrize("strategy,Hkv,G,D,L,filled", SHAPES)
def test_edges_of_the_plans_match_the_oracle(strategy, Hkv, G, D, L, filled):
    _seeded_state_run(strategy, Hkv, G, D, L, filled, 16)
