"""Cache steps that read ahead of their predecessor, back to back: two caches in turn, so that the kernel before the predecessor
is the one that writes the cache."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots,between", [(64, "step"), (64, "product"), (512, "step"), (2048, "product")])
@pytest.mark.parametrize("policy", ["recent_global", "heavy_hitter"])
def test_reading_ahead_of_a_predecessor_that_leaves_the_cache_alone(policy, slots, between):
    from cold_compress_b200 import ops
    from cold_compress_b200.cache import get_cache_constructor
    kv, group, dim, steps = 8, 4, 128, 60
    gen = torch.Generator(device="cuda").manual_seed(slots)
    randn = lambda *s: torch.randn(*s, device="cuda", generator=gen).bfloat16()  # noqa: E731
    cls, relevant = get_cache_constructor(policy)
    kw = dict(max_cache_length=slots, global_tokens=4, max_seq_length=1 << 14, cache_bits=None, recent_window=8, history_window_size=1,
              attn_thresholding=False)
    kw = {n: kw[n] for n in relevant}
    tokens = [(randn(1, kv * group, 1, dim), randn(1, kv, 1, dim), randn(1, kv, 1, dim)) for _ in range(steps)]
    prompt = randn(1, kv, slots, dim), randn(1, kv, slots, dim)
    w, x, out = randn(4096, 4096), randn(4096), torch.empty(4096, dtype=torch.bfloat16, device="cuda")
    positions = [torch.full((1,), slots + t, dtype=torch.int32, device="cuda") for t in range(steps)]

    def run(ahead):
        caches = [cls(1, kv, dim, torch.bfloat16, **kw).to("cuda") for _ in range(2 if between == "step" else 1)]
        for c in caches:
            c._prefill_update(torch.arange(slots, device="cuda"), *prompt)
            if hasattr(c, "attn_history_num"):
                c.attn_history_num.zero_()
                c.attn_history_denom.fill_(1)
        torch.cuda.synchronize()
        for t in range(steps):
            for c in caches:
                y = c.decode_step(*tokens[t], positions[t], overlap_predecessor=ahead)
                if not ahead:
                    torch.cuda.synchronize()
            if between == "product":
                ops.gemv_residual(x, None, 1e-5, w, None, out, [], [], None)
        torch.cuda.synchronize()
        return y.clone(), [{n: v.clone() for n, v in c.state_dict().items()} for c in caches]

    y0, s0 = run(False)
    for _ in range(3):
        y1, s1 = run(True)
        assert torch.equal(y0, y1)
        for a, b in zip(s0, s1):
            for n in a:
                assert torch.equal(a[n], b[n]), n
