"""The fused decode step adds its rows of values in one fixed order, whatever carries them: a warp's neighbouring rows have sums of their
own, down all chunks of the CTA, then the rows, the warps and the CTAs of a head in turn.  With one query head per key head the
probabilities are known, so the attention output is known to the last bit."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
F = np.float32


def _expected(p, v, ctas, chunk, D):
    """bf16 bits [D]; p [L] and v [L, D] fp32."""
    rpw, L = 256 // D, len(p)
    chunks = [range(c * chunk, min(L, (c + 1) * chunk)) for c in range((L + chunk - 1) // chunk)]
    head = np.zeros(D, F)
    for cta in range(ctas):
        warps = np.zeros((8, D), F)
        for w in range(8):
            sums = np.zeros((rpw, D), F)
            for c in chunks[cta::ctas]:
                for s in c:
                    r = s % chunk
                    if r // rpw % 8 == w:      # a fused multiply-add: one rounding
                        sums[r % rpw] = (np.longdouble(p[s]) * v[s].astype(np.longdouble) + sums[r % rpw].astype(np.longdouble)).astype(F)
            warps[w] = (sums[0] + sums[2]) + (sums[1] + sums[3]) if rpw == 4 else sums[0] + sums[1]
        part = warps[0]
        for w in range(1, 8):
            part = part + warps[w]
        head = part if cta == 0 else head + part
    return torch.from_numpy(head).to(torch.bfloat16)


@pytest.mark.parametrize("Hkv,D,L", [(8, 128, 1024), (8, 128, 64), (8, 128, 2000), (4, 64, 300), (80, 64, 100), (3, 64, 47), (8, 128, 511)])
def test_values_are_added_in_a_fixed_order(Hkv, D, L):
    from cold_compress_b200 import _lib, ops
    from device_utils import make_device_cache, synthetic_fill
    for seed in range(3):
        gen = torch.Generator().manual_seed(seed + L)
        cache = make_device_cache("heavy_hitter", Hkv, D, L)
        nxt = synthetic_fill(cache, L, seed=seed)
        cache._q_per_kv = 1
        # large rows that cancel each other, all with the same probability: what is left is the new row and every rounding on the way
        goes = int(torch.randint(4, L - 10, (1,), generator=gen))
        cache.attn_history_num[0, :, goes] = 0.0
        rest = torch.tensor([s for s in range(L) if s != goes])
        rest = rest[torch.randperm(L - 1, generator=gen)]
        n = (L - 1) // 2
        big = (torch.randn(Hkv, n, D, generator=gen) * 2.0 ** 14).to(torch.bfloat16)
        rows = cache.v_cache[0].cpu()
        rows[:, rest[:n]], rows[:, rest[n:2 * n]] = big, -big
        cache.v_cache[0].copy_(rows)
        q = torch.zeros(1, Hkv, 1, D, dtype=torch.bfloat16, device="cuda")
        k, v = (torch.randn(1, Hkv, 1, D, generator=gen).to(torch.bfloat16).cuda() for _ in range(2))
        y = cache.decode_step(q, k, v, torch.tensor([nxt], dtype=torch.int32, device="cuda"))[0, :, 0].cpu()
        assert (cache._fill_idx == goes).all()
        ctas = _lib.load().cc_decode_cluster_size(C.byref(ops._c_state(cache._state_list(), cache._meta(1))))
        chunk = 64
        while chunk > 16 and (L + chunk - 1) // chunk < ctas:
            chunk //= 2
        p, rows = cache._out["probs"].view(Hkv, L).float().cpu().numpy(), cache.v_cache[0].float().cpu().numpy()
        for h in range(min(Hkv, 4)):
            assert torch.equal(y[h], _expected(p[h], rows[h], ctas, chunk, D)), (seed, h)
