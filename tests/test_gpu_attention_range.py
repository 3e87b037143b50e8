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
