"""The fused decode step with a strategy per head, bit for bit against the oracle, at the edges of its plans: heads that append, evict
and drop in one launch, in one CTA per head with several warps to a query head's rows and in clusters, filling and full."""
import numpy as np
import pytest
import torch

from golden_utils import bits, check_y

pytestmark = pytest.mark.gpu

STRATEGIES = [{"strategy": "special"}, {"strategy": "special_punc"}, {"strategy": "window", "recent_window": 0.2},
              {"strategy": "window_heavy_hitter", "recent_window": 0.1, "heavy_hitter_frac": 0.3},
              {"strategy": "special_punc_heavy_hitter", "heavy_hitter_frac": 0.2}, {"strategy": "full"}]


def _cache(Hkv, G, D, L, filled, heavy, without=()):
    from device_utils import make_device_cache, oracle_like, synthetic_fill
    names = [s for s in STRATEGIES if (heavy or "heavy" not in s["strategy"]) and s["strategy"] not in without]
    cache = make_device_cache("hybrid", Hkv, D, L, hybrid_strategies=names)
    nxt = synthetic_fill(cache, filled, seed=L + Hkv)
    cache._q_per_kv = G
    cache.set_head_strategies([h % len(names) for h in range(Hkv)])
    gen = torch.Generator().manual_seed(L)
    cache.num_special.fill_(2)
    cache.special_mask[:, :, 4:6] = True
    cache.punc_mask[:, :, 7:filled:9] = True
    cache.num_punc.fill_(len(range(7, filled, 9)))
    if heavy:
        seen = torch.randint(1, 30, (Hkv, filled), generator=gen)
        ring = (torch.rand(Hkv, filled, 30, generator=gen) / filled).to(torch.bfloat16) * (torch.arange(30) < seen.unsqueeze(-1))
        cache.attn_history_num[0, :, :filled, :30] = ring.cuda()
        cache.attn_history_denom[0, :, :filled] = seen.to(torch.int32).cuda()
        cache.attn_counter.fill_(30)
        cache.resync_history()
    return cache, oracle_like(cache, G), nxt, gen


def _steps(cache, oc, Hkv, G, D, nxt, gen, punc, steps):
    ip = torch.zeros(1, dtype=torch.int32, device="cuda")
    for t in range(steps):
        q = (torch.randn(Hkv * G, D, generator=gen) * 1.5).to(torch.bfloat16)
        k, v = ((torch.randn(Hkv, D, generator=gen) * 1.2).to(torch.bfloat16) for _ in range(2))
        ip.fill_(nxt + t)
        y = cache.decode_step(q.view(1, -1, 1, D).cuda(), k.view(1, -1, 1, D).cuda(), v.view(1, -1, 1, D).cuda(), ip, is_punc=punc(t))[0, :, 0].cpu()
        yo, idx, probs = oc.decode_step(q, k, v, nxt + t, is_punc=punc(t))
        assert torch.equal(cache._fill_idx.cpu(), idx) and int(idx.max()) < cache.max_cache_length, f"step {t}"
        assert torch.equal(cache.pos[0].cpu(), oc.pos), f"step {t}"
        if probs is not None:
            assert np.array_equal(bits(cache._out["probs"]), bits(probs)), f"step {t}"
        check_y(y, yo, G, (), f"step {t}")
    for n in ("mask", "cache_cts", "k_cache", "v_cache", "attn_history_denom", "attn_history_num", "punc_mask", "num_punc"):
        a, b = getattr(cache, n, None), getattr(oc, n, None)
        if torch.is_tensor(a) and torch.is_tensor(b):
            assert torch.equal(a.cpu().reshape(b.shape).to(b.dtype), b), f"final {n} differs"


SHAPES = [(80, 2, 64, 100, 100), (80, 4, 64, 100, 70), (76, 1, 128, 47, 47), (8, 4, 128, 300, 300), (8, 4, 128, 300, 200), (3, 7, 64, 130, 130),
          (8, 8, 128, 1024, 1000), (6, 2, 128, 600, 600)]


@pytest.mark.parametrize("Hkv,G,D,L,filled", SHAPES)
@pytest.mark.parametrize("heavy", [True, False])
def test_heads_that_append_evict_and_drop(Hkv, G, D, L, filled, heavy):
    cache, oc, nxt, gen = _cache(Hkv, G, D, L, filled, heavy)
    _steps(cache, oc, Hkv, G, D, nxt, gen, lambda t: t % 5 == 4, 12)


@pytest.mark.parametrize("Hkv,G,D,L", [(76, 1, 128, 47), (8, 4, 128, 300), (4, 7, 64, 64), (8, 2, 128, 1024)])
def test_counts_that_go_on_beyond_the_last_slot(Hkv, G, D, L):
    """A head that appends counts on when its cache is full (a punctuation token takes the last slot again); when it next evicts, it
    chooses among its own slots."""
    cache, oc, nxt, gen = _cache(Hkv, G, D, L, L, True, without=("special", "special_punc"))
    _steps(cache, oc, Hkv, G, D, nxt, gen, lambda t: t % 4 < 2, 16)
    assert int(oc.cache_cts.max()) > L + 1
