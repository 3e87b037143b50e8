"""Rows of a prompt portion stored behind its attention (cache_append_rows_kernel) against the rule itself, bit for bit: the last
token of a slot stays, first positions keep their slots, every slot that was empty is counted once."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("T,G,Dk,Dv,L,keep,p0", [(1, 1, 8, 8, 4, 0, 0), (31, 3, 64, 64, 64, 0, 50), (33, 1, 128, 128, 32, 0, 7), (257, 5, 72, 40, 300, 0, 123),
                                                 (1001, 4, 128, 128, 1024, 0, 3333), (130, 2, 96, 128, 64, 4, 0), (130, 2, 64, 64, 64, 4, 1000),
                                                 (4099, 1, 8, 8, 5000, 0, 0), (700, 64, 16, 8, 512, 3, 2)])
def test_append_stores_what_the_rule_says(T, G, Dk, Dv, L, keep, p0, dtype):
    from cold_compress_b200 import seq_ops
    gen = torch.Generator().manual_seed(T + G)
    ring = L - keep
    k, v = torch.randn(T, G, Dk, generator=gen).to(dtype), torch.randn(T, G, Dv, generator=gen).to(dtype)
    kc, vc = torch.randn(1, G, L, Dk, generator=gen).to(dtype), torch.randn(1, G, L, Dv, generator=gen).to(dtype)
    pos, mask, cts = torch.full((1, 1, L), -1, dtype=torch.int32), torch.zeros(1, G, 1, L, dtype=torch.bool), torch.zeros(1, dtype=torch.int32)
    for j in range(max(0, p0 - ring // 2), p0):                       # half of the ring holds earlier positions
        s = j if j < keep else keep + (j - keep) % ring
        pos[0, 0, s], mask[0, :, 0, s] = j, True
    cts[0] = int((pos >= 0).sum())
    got = [t.clone().cuda() for t in (kc, vc, pos, mask, cts)]
    for t in range(T):
        p = p0 + t
        s = p if p < keep else keep + (p - keep) % ring
        cts[0] += int(pos[0, 0, s] < 0)
        kc[0, :, s], vc[0, :, s], pos[0, 0, s], mask[0, :, 0, s] = k[t], v[t], p, True
    q, y = torch.zeros(T, G, Dk, device="cuda"), torch.zeros(T, G, Dv, device="cuda", dtype=dtype)
    seq_ops.seq_attention(q, k.cuda(), v.cuda(), got[0], got[1], got[2], got[3], got[4], torch.tensor([p0], dtype=torch.int32, device="cuda"), y, None,
                          ring if keep else 0, 0, 1.0, seq_ops.ATTN_APPEND_ONLY, None, 0, keep)
    for a, b, what in zip(got, (kc, vc, pos, mask, cts), ("keys", "values", "positions", "marks", "count")):
        assert torch.equal(a.cpu(), b), what


@pytest.mark.parametrize("T,G,Dk,Dv,L,keep,p0", [(4201, 17, 64, 64, 4400, 0, 11), (4201, 17, 64, 64, 3000, 5, 2), (2, 64, 64, 64, 70, 4, 3), (1, 300, 8, 16, 9, 0, 0)])
def test_many_rows_and_few_tokens_of_many_heads(T, G, Dk, Dv, L, keep, p0):
    """Above the line from which a thread stores four rows, and marks that are many more than tokens."""
    test_append_stores_what_the_rule_says(T, G, Dk, Dv, L, keep, p0, torch.bfloat16)
