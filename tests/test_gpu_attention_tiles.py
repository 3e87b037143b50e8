"""Prompt-portion attention over bf16 rows (tensor-core kernel) at the sizes where its tiling can go wrong: row tiles of 128
(query, head) pairs, key tiles of 128, padded row widths, portions of a few tokens, masks that cut through tiles, slots
that hold another position, and what the soft cap, the distance penalty, sinks and kept first positions add."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

# T, past, H, G, Dk, Dv, options
SHAPES = [
    (1, 0, 17, 1, 128, 128, {}),                      # one token of a wide group
    (2, 126, 2, 2, 128, 128, {}),                     # keys end exactly at a tile
    (3, 126, 2, 2, 128, 128, {}),                     # ... and one past it
    (64, 0, 4, 2, 128, 128, dict(sink=1)),            # rows fill one tile exactly
    (65, 0, 4, 2, 64, 64, dict(sink=2)),              # ... two rows more
    (43, 7, 9, 3, 72, 40, {}),                        # three heads per key head: tokens cross row tiles; odd widths
    (300, 0, 4, 1, 8, 16, {}),                        # narrowest rows
    (130, 515, 4, 2, 96, 128, dict(window=64)),       # window below a key tile
    (257, 600, 4, 2, 128, 96, dict(window=129, sink=1)),
    (200, 777, 4, 2, 64, 72, dict(window=100, keep=7, softcap=20.0, dist=True, sink=1)),
    (150, 300, 4, 2, 128, 128, dict(block=128)),
    (40, 4000, 8, 1, 128, 128, dict(softcap=5.0)),    # many key tiles for one row tile
    (129, 0, 2, 2, 128, 128, dict(dist=True)),
]


def _reference(q, k, v, past, scale, o, sink, dist):
    T, H, _ = q.shape
    R = H // k.shape[1]
    kk, vv = (t.double().repeat_interleave(R, 1).transpose(0, 1) for t in (k, v))
    i, j = past + torch.arange(T, device=q.device).view(-1, 1), torch.arange(past + T, device=q.device).view(1, -1)
    seen = j <= i
    if o.get("window"):
        seen &= (i - j < o["window"]) | (j < o.get("keep", 0))
    if o.get("block"):
        seen &= j >= i // o["block"] * o["block"]
    s = torch.matmul(q.double().transpose(0, 1), kk.transpose(1, 2)) * scale
    if o.get("softcap"):
        s = o["softcap"] * torch.tanh(s / o["softcap"])
    if dist is not None:
        s = s - dist[0].double().view(H, 1, 1) * torch.log1p(dist[1].double().view(H, 1, 1) * (i - j).clamp(min=0).double())
    s = s.masked_fill(~seen, -math.inf)
    extra = sink.double().view(H, 1, 1) if sink is not None else torch.full((H, 1, 1), 0.0 if o.get("sink") == 2 else -math.inf, dtype=torch.float64, device=q.device)
    p = torch.softmax(torch.cat([s, extra.expand(H, T, 1)], -1), -1)[..., :-1]
    return torch.matmul(p, vv).transpose(0, 1)


@pytest.mark.parametrize("stale", [False, True])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"T{s[0]}-past{s[1]}-H{s[2]}-G{s[3]}-{s[4]}x{s[5]}" + "".join(f"-{k}{v}" for k, v in s[6].items()))
def test_portion_matches_64_bit_attention(shape, stale):
    from cold_compress_b200 import _lib
    from cold_compress_b200.cache import get_cache_constructor
    T, past, H, G, Dk, Dv, o = shape
    dev, gen = "cuda", torch.Generator(device="cuda").manual_seed(T + past)
    window, block, keep = o.get("window", 0), o.get("block", 0), o.get("keep", 0)
    L = window + keep + 5 if window else block or past + T + 3
    cls, _ = get_cache_constructor("recent_global" if window or block else "full")
    cache = cls(1, G, Dk, torch.bfloat16, max_cache_length=L, global_tokens=keep, max_seq_length=1 << 20, cache_bits=None, v_head_dim=Dv).to(dev)
    randn = lambda *s: torch.randn(*s, device=dev, generator=gen)  # noqa: E731
    k, v = randn(past + T, G, Dk).bfloat16(), randn(past + T, G, Dv).bfloat16()
    held = torch.full((L,), -1, dtype=torch.long)
    for j in range(past):
        held[j if j < keep else keep + (j - keep) % (L - keep)] = j
    for slot, j in enumerate(held.tolist()):
        if j >= 0:
            cache.k_cache[0, :, slot], cache.v_cache[0, :, slot] = k[j], v[j]
    if stale:      # empty slots hold rows of an earlier sequence, never finite keys of this one
        cache.k_cache[0][:, held < 0], cache.v_cache[0][:, held < 0] = math.inf, math.nan
    cache.pos[0, 0], cache.mask[0, :, 0] = held.int().to(dev), (held >= 0).to(dev)
    q = 1.3 * randn(T, H, Dk)
    sink = randn(H) if o.get("sink") == 1 else None
    dist = (torch.rand(H, device=dev, generator=gen) * 0.5, torch.rand(H, device=dev, generator=gen)) if o.get("dist") else None
    want = _reference(q, k, v, past, Dk ** -0.5, o, sink, dist)
    mode = {None: _lib.SINK_NONE, 1: _lib.SINK_LEARNED, 2: _lib.SINK_ZERO}[o.get("sink")]
    for dtype in (torch.float32, torch.bfloat16):
        y = torch.empty(T, H, Dv, dtype=dtype, device=dev)
        before = cache.state_dict()
        before = {n: t.clone() for n, t in before.items()}
        cache.sequence_step(q, k[past:].contiguous(), v[past:].contiguous(), torch.full((1,), past, dtype=torch.int32, device=dev), y,
                            window=window, sink=sink, sink_mode=mode, scale=Dk ** -0.5, softcap=o.get("softcap", 0.0), dist=dist, block=block)
        cache.load_state_dict(before)
        err = ((y.double() - want).norm() / want.norm()).item()
        # fp32: a score is a sum of Dk + 2 truncated parts (relative 2^-23 each in the worst case, about 2^-24 sqrt(Dk) in the
        # mean), it enters the weight through exp, and scores here stay below 8; bf16 adds the rounding of the output
        bound = 8 * 2.0 ** -24 * math.sqrt(max(Dk, 64))
        assert err <= (bound if dtype == torch.float32 else 2.0 ** -8), (err, bound)


# past, H, G, Dk, Dv, options: one token
TOKEN_SHAPES = [
    (0, 4, 2, 128, 128, dict(sink=1)),                 # the token alone
    (62, 2, 2, 64, 64, {}), (63, 8, 2, 128, 128, {}), (64, 8, 1, 128, 128, dict(sink=2)),      # around a tile of 64 keys
    (127, 7, 1, 72, 40, {}), (1000, 6, 2, 96, 128, {}),                                        # rows that are not powers of two
    (4200, 32, 8, 128, 128, dict(sink=1)), (20000, 2, 1, 128, 64, {}),                         # several tiles per run
    (3000, 4, 4, 256, 256, {}), (777, 10, 1, 128, 128, {}), (500, 4, 2, 130, 70, {}),          # widest rows; the general kernel
    (900, 4, 2, 128, 128, dict(window=300)), (900, 4, 2, 64, 72, dict(window=65, keep=5, softcap=15.0, dist=True, sink=1)),
    (300, 8, 2, 128, 128, dict(block=128)),
]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", TOKEN_SHAPES, ids=lambda s: f"past{s[0]}-H{s[1]}-G{s[2]}-{s[3]}x{s[4]}" + "".join(f"-{k}{v}" for k, v in s[5].items()))
def test_one_token_matches_64_bit_attention(shape, dtype):
    from cold_compress_b200 import _lib
    from cold_compress_b200.cache import get_cache_constructor
    past, H, G, Dk, Dv, o = shape
    dev, gen = "cuda", torch.Generator(device="cuda").manual_seed(past + H)
    window, block, keep = o.get("window", 0), o.get("block", 0), o.get("keep", 0)
    L = window + keep + 5 if window else block or past + 40
    cls, _ = get_cache_constructor("recent_global" if window or block else "full")
    cache = cls(1, G, Dk, dtype, max_cache_length=L, global_tokens=keep, max_seq_length=1 << 20, cache_bits=None, v_head_dim=Dv).to(dev)
    randn = lambda *s: torch.randn(*s, device=dev, generator=gen)  # noqa: E731
    k, v = randn(past + 2, G, Dk).to(dtype), randn(past + 2, G, Dv).to(dtype)
    held = torch.full((L,), -1, dtype=torch.long)
    for j in range(past):
        held[j if j < keep else keep + (j - keep) % (L - keep)] = j
    at = held >= 0
    cache.k_cache.fill_(math.inf)      # what empty slots hold is never a key
    cache.v_cache.fill_(math.nan)
    cache.k_cache[0][:, at], cache.v_cache[0][:, at] = k[held[at]].transpose(0, 1), v[held[at]].transpose(0, 1)
    cache.pos[0, 0], cache.mask[0, :, 0] = held.int().to(dev), at.to(dev)
    sink = randn(H) if o.get("sink") == 1 else None
    dist = (torch.rand(H, device=dev, generator=gen) * 0.5, torch.rand(H, device=dev, generator=gen)) if o.get("dist") else None
    mode = {None: _lib.SINK_NONE, 1: _lib.SINK_LEARNED, 2: _lib.SINK_ZERO}[o.get("sink")]
    for p in (past, past + 1):         # the second token reads the row that the first has left
        q, y = 1.3 * randn(1, H, Dk), torch.empty(1, H, Dv, device=dev)
        want = _reference(q, k[:p + 1], v[:p + 1], p, Dk ** -0.5, o, sink, dist)
        cache.sequence_step(q, k[p:p + 1].contiguous(), v[p:p + 1].contiguous(), torch.full((1,), p, dtype=torch.int32, device=dev), y,
                            window=window, sink=sink, sink_mode=mode, scale=Dk ** -0.5, softcap=o.get("softcap", 0.0), dist=dist, block=block)
        # fp32 sums of Dk products and of up to `past` weighted values in one rounding each, scores below 8 through exp
        assert ((y.double() - want).norm() / want.norm()).item() <= 8 * 2.0 ** -24 * math.sqrt(max(Dk, 64))
        slot = p if p < keep else keep + (p - keep) % (L - keep)
        assert cache.pos[0, 0, slot].item() == p and torch.equal(cache.k_cache[0, :, slot], k[p]) and torch.equal(cache.v_cache[0, :, slot], v[p])
