"""Prompt attention with score reductions away from the usual range of logits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_weights_add_up_at_any_size_of_the_logits():
    """Rows of large logits whose key quarters have maxima a fraction of a unit apart: the probabilities of a row still add up to
    one.  Logits are exact in fp32 (multiples of 1/128 near 16384), so what could be missing is lost in the softmax alone."""
    from cold_compress_b200 import _lib, ops
    S, D, G = 1024, 64, 4
    gen = torch.Generator(device="cuda").manual_seed(0)
    q, k = torch.zeros(G, S, D, device="cuda"), torch.zeros(1, S, D, device="cuda")
    q[..., 0], q[..., 1], q[..., 2], k[..., 0] = 2.0 ** 17, 1, 1, 1          # the scale is 1 / 8
    k[0, :, 2] = torch.randint(-128, 129, (S,), device="cuda", generator=gen) / 16
    for c, d in enumerate((-45, 12, -41, 43)):                               # one maximum for each quarter of a tile's keys
        k[0, 32 * c, 1], k[0, 32 * c, 2] = 16, d / 16
    q, k, v = q.bfloat16(), k.bfloat16(), torch.randn(1, S, D, device="cuda", generator=gen).bfloat16()
    y, col, obs = torch.empty_like(q), torch.empty(1, S, device="cuda"), torch.empty(1, S, device="cuda")
    ws = torch.empty(ops.prefill_attention_workspace(S, 1, G, 256, 0), dtype=torch.uint8, device="cuda")
    ops.prefill_attention(q, k, v, y, _lib.ATTN_MATH_FP32, 256, [], col, obs, None, ws)
    # bf16 roundings of S G S / 2 probabilities average out; what is left is far below one of them (2^-9)
    assert abs(col.sum().item() / S - 1) < 2.0 ** -14 and abs(obs.sum().item() / 256 - 1) < 2.0 ** -14
