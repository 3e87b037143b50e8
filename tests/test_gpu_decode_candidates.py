"""The fused decode step where every CTA's candidate for eviction holds the largest logit of its rows, so that the maximum which all CTAs
of a head have to agree on comes from a candidate that stays: bit for bit against the oracle."""
import numpy as np
import pytest
import torch

from golden_utils import bits, check_y

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strategy", ["heavy_hitter", "recent_global", "l2"])
@pytest.mark.parametrize("Hkv,G,D,L", [(8, 8, 128, 1024), (8, 4, 128, 1024), (8, 4, 128, 512), (4, 7, 128, 300), (2, 7, 64, 47), (64, 1, 64, 1500)])
def test_candidates_that_stay_decide_the_maximum(strategy, Hkv, G, D, L):
    from device_utils import make_device_cache, oracle_like, synthetic_fill
    for seed in range(6):
        gen = torch.Generator().manual_seed(seed + L)
        cache = make_device_cache(strategy, Hkv, D, L)
        nxt = synthetic_fill(cache, L, seed=seed)
        cache._q_per_kv = G
        # one slot of every 16 is the one to go: little history, the largest norm, the oldest position
        mine = torch.arange(0, L, 16) + torch.randint(0, 16, ((L + 15) // 16,), generator=gen)
        mine = mine[(mine < L) & (mine >= 4)]
        q = torch.randn(Hkv, 1, D, generator=gen).expand(Hkv, G, D) + 0.1 * torch.randn(Hkv, G, D, generator=gen)
        rows = cache.k_cache[0].cpu().float() * 0.3
        rows[:, mine] = q[:, :1] * (1.0 + 0.2 * torch.rand(Hkv, mine.numel(), 1, generator=gen))
        cache.k_cache[0].copy_(rows.to(torch.bfloat16))
        if strategy == "heavy_hitter":
            cache.attn_history_num[0, :, mine] *= 1e-4
        elif strategy == "l2":
            cache.update_state(None, None, None, True, None)
        else:
            pos = torch.arange(L)
            rest = torch.tensor([s for s in range(4, L) if s not in set(mine.tolist())], dtype=torch.long)
            pos[torch.cat([mine, rest])] = torch.arange(4, L)
            cache.pos[0].copy_(pos.to(torch.int32))
        oc = oracle_like(cache, G)
        ip = torch.tensor([nxt], dtype=torch.int32, device="cuda")
        q, k, v = q.reshape(Hkv * G, D).to(torch.bfloat16), torch.randn(Hkv, D, generator=gen).to(torch.bfloat16), torch.randn(Hkv, D, generator=gen).to(torch.bfloat16)
        y = cache.decode_step(q.view(1, -1, 1, D).cuda(), k.view(1, -1, 1, D).cuda(), v.view(1, -1, 1, D).cuda(), ip)[0, :, 0].cpu()
        yo, idx, probs = oc.decode_step(q, k, v, nxt)
        assert torch.equal(cache._fill_idx.cpu(), idx) and set(idx.tolist()) <= set(mine.tolist())
        if probs is not None:
            assert np.array_equal(bits(cache._out["probs"]), bits(probs))
        check_y(y, yo, G, (), f"seed {seed}")
