"""Prompt-portion attention over bf16 rows (tensor-core kernel) away from the usual score range: scores of any finite size."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _portion(q, k, v, past, scale, sink=None, dtype=torch.float32, **kw):
    """y of the portion q [T, H, D] behind `past` tokens, k and v [past + T, G, D] bf16, through the public cache."""
    from cold_compress_b200 import _lib
    from cold_compress_b200.cache import get_cache_constructor
    T, H, _ = q.shape
    G, Dk, Dv = k.shape[1], k.shape[2], v.shape[2]
    cls, _ = get_cache_constructor("full")
    cache = cls(1, G, Dk, torch.bfloat16, max_cache_length=past + T + 3, global_tokens=0, max_seq_length=1 << 20, cache_bits=None, v_head_dim=Dv).to("cuda")
    cache.k_cache[0, :, :past], cache.v_cache[0, :, :past] = k[:past].transpose(0, 1), v[:past].transpose(0, 1)
    cache.pos[0, 0, :past], cache.mask[0, :, 0, :past] = torch.arange(past, dtype=torch.int32, device="cuda"), True
    y = torch.empty(T, H, Dv, dtype=dtype, device="cuda")
    cache.sequence_step(q, k[past:].contiguous(), v[past:].contiguous(), torch.full((1,), past, dtype=torch.int32, device="cuda"), y, sink=sink,
                        sink_mode=_lib.SINK_NONE if sink is None else _lib.SINK_LEARNED, scale=scale, **kw)
    return y


def _scores(q, k, past, scale):
    T, H, _ = q.shape
    s = torch.matmul(q.double().transpose(0, 1), k.double().repeat_interleave(H // k.shape[1], 1).transpose(0, 1).transpose(1, 2)) * scale
    return s.masked_fill(torch.arange(past + T, device=q.device).view(1, -1) > past + torch.arange(T, device=q.device).view(-1, 1), -math.inf)


@pytest.mark.parametrize("learned", [False, True])
@pytest.mark.parametrize("scale", [1.0, -1.0, 0.5])     # a scale that is not positive takes the general shape of a score
def test_scores_of_any_size_keep_their_softmax(scale, learned):
    T, past, G, D = 130, 300, 2, 64
    gen = torch.Generator(device="cuda").manual_seed(3)
    grid = lambda *s: torch.randint(-8, 9, s, device="cuda", generator=gen) / 4  # noqa: E731
    top = torch.tensor([12000.0, 22800.0, -23000.0, 24000.0, -40000.5, 1e5, -1e5, 131072.0], device="cuda")
    H = top.numel()
    # channel 0 moves all scores of a head; the others leave a spread of a few units.  Every product and sum is a multiple of
    # 1/16 below 2^18: exact in fp32, so the scores themselves carry no error at any size
    q, k = grid(T, H, D), grid(past + T, G, D)
    q[..., 9:] = 0
    q[..., 0], k[..., 0] = top, 1
    k, v = k.bfloat16(), torch.randn(past + T, G, D, device="cuda", generator=gen).bfloat16()
    sink = top * scale + 2 if learned else None
    s = _scores(q, k, past, scale)
    extra = sink.double().view(H, 1, 1).expand(H, T, 1) if learned else s.new_full((H, T, 1), -math.inf)
    w = torch.softmax(torch.cat([s, extra], -1), -1)[..., :-1]
    want = torch.matmul(w, v.double().repeat_interleave(H // G, 1).transpose(0, 1)).transpose(0, 1)
    y = _portion(q, k, v, past, scale, sink)
    # what is left is the exponential (2 units of 2^-23) and fp32 sums, per head
    for h in range(H):
        err = ((y[:, h].double() - want[:, h]).norm() / want[:, h].norm()).item()
        assert err <= 8 * 2.0 ** -24 * math.sqrt(D), (top[h].item(), err)


def _want(q, k, v, past, scale, seen=None):
    """64-bit attention in which a key that is not seen takes no part, whatever it holds; 0 for weights of 0."""
    s = _scores(q, torch.nan_to_num(k.double(), 0.0, 0.0, 0.0), past, scale)
    if seen is not None:
        s = s.masked_fill(~seen, -math.inf)
    return torch.matmul(torch.softmax(s, -1), torch.nan_to_num(v.double(), 0.0, 0.0, 0.0).repeat_interleave(q.shape[1] // k.shape[1], 1).transpose(0, 1)).transpose(0, 1)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("softcap", [0.0, 30.0])
@pytest.mark.parametrize("where", [0, 77, 299, 300, 310, 429])       # a row of the cache or of the portion, first, last, between
@pytest.mark.parametrize("kind", ["key -inf", "key +inf", "value inf", "value nan", "query inf"])
def test_what_is_not_finite_stays_where_it_belongs(kind, where, softcap, dtype):
    T, past, H, G, D, scale = 130, 300, 6, 2, 72, 72 ** -0.5
    gen = torch.Generator(device="cuda").manual_seed(where)
    q, k, v = (torch.randn(n, h, D, device="cuda", generator=gen) for n, h in ((T, H), (past + T, G), (past + T, G)))
    k, v = k.bfloat16(), v.bfloat16()
    q[..., 5], q[..., 9] = -q[..., 5].abs(), 0.5       # three parts of 0.5 are 0.5, 0 and 0
    t = max(0, where - past)                           # queries t, t + 1, ... see the row
    if kind.startswith("key"):
        k[where, 0, 5] = math.inf if kind == "key -inf" else -math.inf
    elif kind.startswith("value"):
        v[where, 0, 9] = math.inf if kind == "value inf" else math.nan
    else:
        q[t, 1, 9] = math.inf
    if softcap and not kind.startswith("value"):
        pytest.skip("the cap makes these scores finite or NaN by a tanh of its own")
    y = _portion(q, k, v, past, scale, dtype=dtype, softcap=softcap).double()
    seen = None
    if kind == "key -inf":     # a weight of zero: the key of head group 0 might as well not be there
        seen = torch.ones(H, T, past + T, dtype=torch.bool, device="cuda")
        seen[:H // G, :, where] = False
    clean = q.nan_to_num(0.0, 0.0, 0.0)
    if softcap:
        s = _scores(clean, k, past, scale)
        s = torch.where(s.isinf(), s, softcap * torch.tanh(s / softcap))
        want = torch.matmul(torch.softmax(s, -1), torch.nan_to_num(v.double(), 0.0, 0.0, 0.0).repeat_interleave(H // G, 1).transpose(0, 1)).transpose(0, 1)
    else:
        want = _want(clean, k, v, past, scale, seen)
    if kind == "key +inf":
        want[t:, :H // G] = math.nan
    elif kind.startswith("value"):
        want[t:, :H // G, 9] = math.inf if kind == "value inf" else math.nan
    elif kind == "query inf":
        want[t, 1] = math.nan                          # infinities of both signs among the scores
    if where == 0 and kind == "key -inf" and past == 0:
        want[0, :H // G] = 0
    assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isinf(), want.isinf())
    keep = want.isfinite()
    err = ((y - want)[keep].norm() / want[keep].norm()).item()
    assert err <= (8 * 2.0 ** -24 * math.sqrt(D) if dtype == torch.float32 else 2.0 ** -8), err


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("shape", [
    (4735, 32, 8, 128, 128, {}), (4736, 8, 8, 128, 128, {}), (5500, 32, 8, 128, 128, dict(sink=1)),      # as many tiles as runs, one more, some runs of two
    (9000, 8, 8, 64, 64, {}), (9001, 16, 16, 64, 64, dict(sink=2)),                                      # runs that fetch ahead
    (2400, 64, 8, 128, 128, {}), (6000, 64, 8, 64, 128, {}),                                             # eight query heads: one CTA per SM
    (8200, 2, 1, 256, 128, {}), (5000, 6, 2, 256, 256, {}),                                              # tiles of 64 keys, more of them than runs
    (6000, 16, 16, 128, 128, dict(window=3000, sink=1)),
], ids=lambda s: f"past{s[0]}-H{s[1]}-G{s[2]}-{s[3]}x{s[4]}" + "".join(f"-{k}{v}" for k, v in s[5].items()))
def test_one_token_over_runs_of_several_tiles(shape, dtype):
    import test_gpu_attention_tiles as tiles
    tiles.test_one_token_matches_64_bit_attention(shape, dtype)
