"""One-token attention over bf16 rows whose tiles come as boxes (widths of whole 64 columns): tiles that end with the token itself, rings
that wrap within a tile, kept positions, rows without a position that are no numbers, query rows on any boundary of a float.  Checks
and bounds are those of test_gpu_attention_mma.py."""
import math

import pytest
import torch

from test_gpu_attention_mma import _layer, _run

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _check(y, want, s, Dk, past):
    tol = 2.0 ** -24 * (2 * (Dk / 16 + 8) * max(s[s > -math.inf].abs().max().item(), 1.0) + past / 32 + 32)      # as there
    assert ((y.double() - want).norm() / want.norm()).item() <= tol
    assert ((y.double() - want).abs().max() / want.abs().max()).item() <= 2 * tol


@pytest.mark.parametrize("H,G,Dk,Dv", [(12, 4, 64, 64), (8, 2, 128, 128), (3, 1, 192, 64)])
@pytest.mark.parametrize("past,window,keep", [(100, 129, 0), (500, 129, 0), (1000, 1000, 0), (1128, 1000, 0), (3000, 1000, 7), (511, 256, 0), (512, 256, 0), (2100, 256, 4),
                                              (40000, 2048, 0)])
@pytest.mark.parametrize("sink", [0, 1])
def test_rings_that_wrap_within_a_tile(H, G, Dk, Dv, past, window, keep, sink):
    _check(*_run(H, G, Dk, Dv, past, window, keep, sink), Dk, past)


def _nan_beyond(cache, k, v, at):
    empty = cache.pos[0, 0] < 0
    cache.k_cache[0][:, empty], cache.v_cache[0][:, empty] = math.nan, math.inf


@pytest.mark.parametrize("past", [125, 126, 127, 128, 130, 143, 144, 255, 256, 700])
@pytest.mark.parametrize("H,G,Dk,Dv", [(32, 8, 128, 128), (10, 2, 64, 128)])
def test_slots_without_a_position_take_no_part(H, G, Dk, Dv, past):
    _check(*_run(H, G, Dk, Dv, past, spoil=_nan_beyond), Dk, past)


def test_query_rows_on_a_boundary_of_a_float():
    from cold_compress_b200 import _lib
    H, G, D, past = 8, 2, 128, 500
    got = []
    for shift in (0, 1, 2, 3):
        cache, at, k, v, g = _layer(G, D, D, past, seed=3)
        q = torch.zeros(H * D + 4, device=DEV)
        q[shift:shift + H * D] = torch.randn(H * D, device=DEV, generator=g)
        k1, v1 = torch.randn(1, G, D, device=DEV, generator=g).bfloat16(), torch.randn(1, G, D, device=DEV, generator=g).bfloat16()
        y, ip = torch.empty(1, H, D, device=DEV), torch.full((1,), past, dtype=torch.int32, device=DEV)
        cache.sequence_step(q[shift:shift + H * D].view(1, H, D), k1, v1, ip, y, sink_mode=_lib.SINK_NONE, scale=D ** -0.5)
        got.append(y)
    assert all(torch.equal(y, got[0]) for y in got)


@pytest.mark.parametrize("past,window,keep", [(1128, 1000, 0), (3000, 1000, 7), (300, 128, 4), (131, 100, 30)])
def test_widest_rows_of_rings_and_kept_positions(past, window, keep):
    """Rows of a tile that is no single run, copied 16 bytes a lane: 32 of them a row."""
    _check(*_run(16, 2, 256, 256, past, window, keep, 0), 256, past)
