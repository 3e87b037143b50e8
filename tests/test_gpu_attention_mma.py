"""One-token attention over bf16 rows on the tensor cores, against 64 bits: rows of every width that it serves, one to eight query heads
per key head, positions at the edges of tiles and runs, rings that have wrapped, kept first positions, and numbers that are none."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _layer(G, Dk, Dv, past, window=0, keep=0, seed=0, room=3):
    from cold_compress_b200.cache import get_cache_constructor
    g = torch.Generator(device=DEV).manual_seed(seed)
    L = window + keep if window else past + room
    cls, _ = get_cache_constructor("recent_global" if window else "full")
    cache = cls(1, G, Dk, torch.bfloat16, max_cache_length=L, global_tokens=keep, max_seq_length=1 << 20, cache_bits=None, v_head_dim=Dv).to(DEV)
    at = torch.arange(past, device=DEV)
    at = at[(at < keep) | (at >= past - (L - keep))]
    slot = torch.where(at < keep, at, keep + (at - keep) % (L - keep))
    k, v = (torch.randn(G, at.numel(), D, device=DEV, generator=g).bfloat16() for D in (Dk, Dv))
    cache.k_cache[0][:, slot], cache.v_cache[0][:, slot] = k, v
    cache.pos[0, 0, slot], cache.mask[0, :, 0, slot] = at.to(torch.int32), True
    cache.cache_cts.fill_(at.numel())
    return cache, at, k, v, g


def _run(H, G, Dk, Dv, past, window=0, keep=0, sink=0, softcap=0.0, dtype=torch.float32, spoil=None, seed=0):
    from cold_compress_b200 import _lib
    cache, at, k, v, g = _layer(G, Dk, Dv, past, window, keep, seed)
    if spoil is not None:
        spoil(cache, k, v, at)
    q = 1.3 * torch.randn(1, H, Dk, device=DEV, generator=g)
    k1, v1 = torch.randn(1, G, Dk, device=DEV, generator=g).bfloat16(), torch.randn(1, G, Dv, device=DEV, generator=g).bfloat16()
    sinks = torch.randn(H, device=DEV, generator=g) if sink == 1 else None
    y, ip = torch.empty(1, H, Dv, device=DEV, dtype=dtype), torch.full((1,), past, dtype=torch.int32, device=DEV)
    cache.sequence_step(q, k1, v1, ip, y, window=window, sink=sinks, sink_mode=(_lib.SINK_NONE, _lib.SINK_LEARNED, _lib.SINK_ZERO)[sink],
                        scale=Dk ** -0.5, softcap=softcap)
    K, V = torch.cat([k, k1.transpose(0, 1)], 1).double(), torch.cat([v, v1.transpose(0, 1)], 1).double()
    j = torch.cat([at, torch.tensor([past], device=DEV)])
    s = torch.einsum("grd,gnd->grn", q[0].double().view(G, H // G, Dk), K) * Dk ** -0.5
    if softcap:
        s = softcap * torch.tanh(s / softcap)
    if window:
        s = s.masked_fill(~((past - j < window) | (j < keep)), -math.inf)
    extra = sinks.double().view(G, -1, 1) if sink == 1 else torch.zeros(G, H // G, 1, device=DEV, dtype=torch.float64) if sink == 2 else None
    w = torch.softmax(s if extra is None else torch.cat([s, extra], -1), -1)[..., :s.shape[-1]]
    y64 = torch.where(w.unsqueeze(-1) > 0, w.unsqueeze(-1) * V.unsqueeze(1), 0.0 * w.unsqueeze(-1)).sum(2).reshape(H, Dv)
    slot = past if not window else keep + (past - keep) % (cache.max_cache_length - keep) if past >= keep else past
    assert torch.equal(cache.k_cache[0][:, slot], k1[0]) and torch.equal(cache.v_cache[0][:, slot], v1[0]) and int(cache.pos[0, 0, slot]) == past
    return y[0], y64, s


SHAPES = [(8, 1, 8, 8), (3, 3, 16, 24), (14, 2, 72, 40), (6, 2, 128, 64), (16, 16, 96, 128), (32, 8, 128, 128), (5, 1, 136, 248), (16, 2, 256, 256)]


@pytest.mark.parametrize("H,G,Dk,Dv", SHAPES)
@pytest.mark.parametrize("past", [0, 1, 127, 128, 129, 1000, 5003])
def test_rows_and_edges(H, G, Dk, Dv, past):
    y, want, s = _run(H, G, Dk, Dv, past)
    # a score: (Dk / 16 + 8) roundings of its size; a weight: twice that and its exponential; the sums over keys as many as there are steps
    top = s.abs().max().item()
    tol = 2.0 ** -24 * (2 * (Dk / 16 + 8) * max(top, 1.0) + past / 32 + 32)
    assert ((y.double() - want).norm() / want.norm()).item() <= tol
    assert ((y.double() - want).abs().max() / want.abs().max()).item() <= 2 * tol


@pytest.mark.parametrize("H,G,Dk,Dv", [(32, 16, 32, 32), (32, 16, 8, 24), (32, 16, 48, 32), (16, 16, 72, 72), (16, 16, 64, 80), (16, 16, 64, 64), (48, 16, 32, 32)])
@pytest.mark.parametrize("past", [2290, 2310, 4590, 4620, 9200, 9300])
def test_narrow_rows_of_few_query_heads(H, G, Dk, Dv, past):
    """Around the numbers of tiles from which one or two query heads leave the tensor cores (18 runs a head of 128 keys a tile)."""
    y, want, s = _run(H, G, Dk, Dv, past)
    tol = 2.0 ** -24 * (2 * (Dk / 16 + 8) * max(s.abs().max().item(), 1.0) + past / 32 + 32)      # as above
    assert ((y.double() - want).norm() / want.norm()).item() <= tol


@pytest.mark.parametrize("past,window,keep", [(10, 64, 0), (500, 64, 0), (1000, 129, 4), (3000, 1000, 7), (70, 64, 4)])
@pytest.mark.parametrize("sink,softcap", [(0, 0.0), (1, 30.0), (2, 0.0)])
def test_rings_kept_positions_sinks_and_caps(past, window, keep, sink, softcap):
    y, want, _ = _run(12, 4, 64, 72, past, window, keep, sink, softcap, torch.bfloat16)
    assert ((y.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all()


def _at(name, value):
    def spoil(cache, k, v, at):
        i, rows = at.numel() // 2, {"k": (k, cache.k_cache), "v": (v, cache.v_cache)}[name[0]]
        for t in (rows[0][:, i], rows[1][0][:, int(at[i])]):
            t[..., 3] = value
    return spoil


@pytest.mark.parametrize("past", [60, 700])
def test_numbers_that_are_none(past):
    inf = float("inf")
    y, want, _ = _run(8, 2, 64, 64, past, spoil=_at("v", inf))
    assert torch.equal(y.isposinf(), want.isposinf()) and int(y.isposinf().sum()) == 8 and not y.isnan().any()
    y, want, _ = _run(8, 2, 64, 64, past, spoil=_at("v", float("nan")))
    assert torch.equal(y.isnan(), want.isnan()) and int(y.isnan().sum()) == 8
    y, want, s = _run(8, 2, 64, 64, past, spoil=_at("k", inf))         # scores of +inf leave NaN, of -inf a weight of zero
    plus = s.isposinf().any(-1).reshape(-1)
    assert plus.any() and (~plus).any() and y[plus].isnan().all()
    assert ((y[~plus].double() - want[~plus]).abs() <= 1e-5).all()


def test_a_slot_without_its_position_counts_for_nothing():
    def forget(cache, k, v, at):
        i = int(at[at.numel() // 3])
        cache.pos[0, 0, i] = -1
        cache.v_cache[0][:, i] = float("nan")
        cache.k_cache[0][:, i] = float("inf")
    from cold_compress_b200 import _lib
    cache, at, k, v, g = _layer(2, 64, 64, 300)
    forget(cache, k, v, at)
    q = torch.randn(1, 8, 64, device=DEV, generator=g)
    k1, v1 = (torch.randn(1, 2, 64, device=DEV, generator=g).bfloat16() for _ in range(2))
    y, ip = torch.empty(1, 8, 64, device=DEV), torch.full((1,), 300, dtype=torch.int32, device=DEV)
    cache.sequence_step(q, k1, v1, ip, y, sink_mode=_lib.SINK_NONE, scale=0.125)
    gone = at.numel() // 3
    K, V = (torch.cat([t[:, :gone], t[:, gone + 1:], n.transpose(0, 1)], 1).double() for t, n in ((k, k1), (v, v1)))
    w = torch.softmax(torch.einsum("grd,gnd->grn", q[0].double().view(2, 4, 64), K) * 0.125, -1)
    assert ((y[0].double() - torch.einsum("grn,gnd->grd", w, V).reshape(8, 64)).abs() <= 1e-5).all()


def _two_keys(q, keys, values, scale):
    """y [8, 64] of eight query heads over two positions, keys and values [2, 64]."""
    from cold_compress_b200 import _lib
    cache, _, _, _, _ = _layer(1, 64, 64, 1)
    cache.k_cache[0, 0, 0], cache.v_cache[0, 0, 0] = keys[0], values[0]
    y, ip = torch.empty(1, 8, 64, device=DEV), torch.ones(1, dtype=torch.int32, device=DEV)
    cache.sequence_step(q.view(1, 8, 64), keys[1].view(1, 1, 64), values[1].view(1, 1, 64), ip, y, sink_mode=_lib.SINK_NONE, scale=scale)
    return y[0].double()


def test_all_three_parts_of_a_query_count():
    """Queries whose first and second part cancel between two channels: the score is what the third one holds."""
    j = torch.arange(1, 9, device=DEV)
    q, keys, values = torch.zeros(8, 64, device=DEV), torch.zeros(2, 64, device=DEV).bfloat16(), torch.zeros(2, 64, device=DEV).bfloat16()
    q[:, 0], q[:, 1] = 1 + 2.0 ** -9 + j * 2.0 ** -20, 1 + 2.0 ** -9
    keys[0, 0], keys[0, 1], values[0] = 1, -1, 1
    # scores j / 4 and 0, exact in fp32; the exponentials and the quotient are a few roundings
    y = _two_keys(q, keys, values, 2.0 ** 18)
    assert ((y - torch.sigmoid(j.double() / 4).view(8, 1)).abs() <= 8 * 2.0 ** -24).all()


def test_all_three_parts_of_a_weight_count():
    """Weights of 1 and of almost 1 on values of opposite sign: the sum is what the third part of the second one holds."""
    j = torch.arange(1, 9, device=DEV)
    q, keys, values = torch.zeros(8, 64, device=DEV), torch.zeros(2, 64, device=DEV).bfloat16(), torch.ones(2, 64, device=DEV).bfloat16()
    q[:, 0] = j * 2.0 ** -18
    keys[1, 0], values[1] = -1, -1
    w = torch.exp(-j.double() * 2.0 ** -18)
    # the smaller weight is one rounding of a number just below 1 and an exponential's error (2 units of 2^-24), the sum exact
    y = _two_keys(q, keys, values, 1.0)
    assert ((y - ((1 - w) / (1 + w)).view(8, 1)).abs() <= 3 * 2.0 ** -24).all()
