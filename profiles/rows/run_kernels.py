"""One or two launches each of the prompt, one-token, recurrence, expert and product kernels (the command captured under ncu)."""
import sys
from pathlib import Path

import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent.parent))
from cold_compress_b200 import _lib, seq_ops  # noqa: E402
from cold_compress_b200.attention_utils import prefill_attention_stats  # noqa: E402
from cold_compress_b200.cache import get_cache_constructor  # noqa: E402

BF16, dev = torch.bfloat16, "cuda"


def rows(T, past, H, G, D, dtype=BF16):
    cls, _ = get_cache_constructor("full")
    c = cls(1, G, D, dtype, max_cache_length=past + T + 3, global_tokens=0, max_seq_length=1 << 20, cache_bits=None).to(dev)
    c.k_cache.normal_()
    c.v_cache.normal_()
    c.pos[0, 0, :past], c.mask[0, :, 0, :past] = torch.arange(past, dtype=torch.int32, device=dev), True
    q, k, v = torch.randn(T, H, D, device=dev), torch.randn(T, G, D, device=dev).to(dtype), torch.randn(T, G, D, device=dev).to(dtype)
    y, at, sink = torch.empty(T, H, D, dtype=BF16, device=dev), torch.full((1,), past, dtype=torch.int32, device=dev), torch.randn(H, device=dev)
    c.sequence_step(q, k, v, at, y, sink=sink, sink_mode=_lib.SINK_LEARNED, scale=D ** -0.5)


def scores(S, H, G, D):
    q, k, v = (torch.randn(1, n, S, D, device=dev).to(BF16) for n in (H, G, G))
    prefill_attention_stats(q, k, v)


def recurrence(T, H, D):
    r, k, v, w = (torch.randn(T, H * D, device=dev) for _ in range(4))
    seq_ops.wkv(r, k, v, w, torch.randn(H * D, device=dev), torch.randn(H * D, device=dev), torch.zeros(H, D, D, device=dev), torch.empty(T, H * D, device=dev), H, D)


def experts(T, top, n, E, F):
    ids = torch.rand(T, n, device=dev).topk(top, -1).indices.int().contiguous()
    M = T * top
    counts, slot, perm = (torch.empty(m, dtype=torch.int32, device=dev) for m in (n, M, M))
    seq_ops.moe_group(ids, n, counts, slot, perm)
    gu, d, h = (torch.randn(*s, device=dev).to(BF16) * 0.02 for s in ((n, 2 * F, E), (n, E, F), (T, E)))
    seq_ops.moe_grouped(gu, d, h, perm, counts, torch.empty(M, E, dtype=BF16, device=dev), torch.empty(M, F, dtype=BF16, device=dev),
                        torch.empty(M, E, device=dev), _lib.ACT_SILU)


def products(N, K):
    seq_ops.gemv_multi([(torch.randn(1, K, device=dev), torch.randn(N, K, device=dev).to(BF16), torch.empty(1, N, device=dev))])


torch.manual_seed(0)
for _ in range(2):
    rows(4096, 0, 32, 8, 128)
    rows(1, 4096, 32, 8, 128)
    rows(1, 12000, 32, 8, 128)
    scores(4096, 32, 8, 128)
    recurrence(2048, 32, 64)
    experts(2048, 4, 16, 2048, 1536)
    products(16384, 2048)
torch.cuda.synchronize()
print("done")
