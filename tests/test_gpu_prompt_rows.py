"""The row kernels of a prompt layer against the tensor operations they stand for, and the calls that keep those operations."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _bf16(*shape, seed=0, scale=1.0):
    return (torch.randn(*shape, generator=torch.Generator().manual_seed(seed)) * scale).bfloat16().cuda()


def _adjacent(got, want, share=0.02):
    """Equal or neighbouring bf16 values, and equal almost everywhere."""
    a, b = got.float(), want.float()
    assert torch.all((a - b).abs() <= 2.0 ** -7 * torch.maximum(a.abs(), b.abs()))
    assert (a != b).float().mean().item() <= share


@pytest.mark.parametrize("rows, dim", [(1, 8), (3, 896), (7, 2048), (5, 2056), (2, 4096), (129, 3584), (2, 8200), (1, 16384)])
def test_rms_norm_rows(rows, dim):
    from cold_compress_b200.model import RMSNorm
    m = RMSNorm(dim, eps=1e-5)
    m.weight.data = 1.0 + 0.3 * torch.randn(dim)
    m = m.to(torch.bfloat16).cuda()
    x = _bf16(1, rows, dim, seed=dim, scale=3.0)
    want = m(x)                      # gradients wanted: tensor operations
    assert want.requires_grad
    with torch.no_grad():
        got = m(x)
    _adjacent(got, want.detach())    # the mean of the squares is summed in another order


@pytest.mark.parametrize("S, Hq, Hkv, D", [(1, 1, 1, 8), (5, 14, 2, 64), (33, 28, 4, 128), (130, 8, 8, 128), (7, 3, 1, 72)])
def test_rotated_rows(S, Hq, Hkv, D):
    from cold_compress_b200 import ops
    from cold_compress_b200.model import apply_rotary_emb, precompute_freqs_cis
    qkv = _bf16(S, (Hq + 2 * Hkv) * D, seed=S)
    freqs = precompute_freqs_cis(S, D, 10000, torch.bfloat16).cuda()
    q, k = torch.empty(S, Hq, D, dtype=torch.bfloat16, device="cuda"), torch.empty(S, Hkv, D, dtype=torch.bfloat16, device="cuda")
    ops.rope_rows(qkv, freqs, q, k)
    assert torch.equal(q, apply_rotary_emb(qkv[:, :Hq * D].reshape(1, S, Hq, D), freqs)[0])
    assert torch.equal(k, apply_rotary_emb(qkv[:, Hq * D:(Hq + Hkv) * D].reshape(1, S, Hkv, D), freqs)[0])


@pytest.mark.parametrize("n", [8, 2040, 100 * 4864])
def test_gated_unit_rows(n):
    from cold_compress_b200 import ops
    a, b = _bf16(n, seed=1, scale=4.0), _bf16(n, seed=2)
    a[:4] = torch.tensor([float("inf"), -float("inf"), -100.0, 0.0])
    out = torch.empty_like(a)
    ops.silu_mul(a, b, out)
    want = F.silu(a) * b
    finite = want.isfinite()
    assert torch.equal(out[~finite].nan_to_num(7.0), want[~finite].nan_to_num(7.0))
    _adjacent(out[finite], want[finite], share=1e-3)


def test_calls_that_keep_the_tensor_operations():
    from cold_compress_b200 import ops
    from cold_compress_b200.model import RMSNorm
    x = _bf16(4, 64)
    assert ops.plain_rows(x)
    assert not ops.plain_rows(x.float()) and not ops.plain_rows(x.t()) and not ops.plain_rows(x[:, :60]) and not ops.plain_rows(x.view(-1)[1:57].view(7, 8))
    assert not ops.plain_rows(x.clone().requires_grad_()) and not ops.plain_rows(x[:0])
    m = RMSNorm(64).to(torch.bfloat16).cuda().requires_grad_(False)
    want = m(x)
    with torch.no_grad():
        batched = torch.vmap(m)(x.view(2, 2, 64))
        _adjacent(batched.view(4, 64), want)
        out, tangent = torch.func.jvp(m, (x,), (x,))
    _adjacent(out, want)
    assert tangent.shape == x.shape


@pytest.mark.parametrize("S, Hkv, G, windows", [(1, 1, 1, ()), (31, 2, 4, (3,)), (512, 1, 4, ()), (513, 2, 4, (65, 600)), (1055, 1, 7, (300,))])
def test_score_reductions_add_the_tiles_in_order(S, Hkv, G, windows):
    """15, 16, 17 and more query tiles behind a column: the sums are the tiles' partials added in order, bit for bit."""
    from cold_compress_b200 import _lib, ops
    gen = torch.Generator().manual_seed(S)
    q, k, v = (torch.randn(h, S, 128, generator=gen).bfloat16().cuda() for h in (Hkv * G, Hkv, Hkv))
    y, obs = torch.empty_like(q), min(16, S)
    ws = torch.full((ops.prefill_attention_workspace(S, Hkv, G, obs, len(windows)) // 4 + 64,), float("nan"), device="cuda")
    col, seen, band = (torch.empty(n, device="cuda") for n in ((Hkv, S), (Hkv, S), (max(1, len(windows)), Hkv, S)))
    ops._prefill_attention(q, k, v, y, _lib.ATTN_NAIVE_BF16, obs, list(windows), col, seen, band if windows else None, ws)
    QB = 1 << ((128 // G).bit_length() - 1)
    tiles, pad = -(-S // QB), -(-S // 128) * 128
    at = (-ws.data_ptr() % 256) // 4
    first = (S - obs) // QB

    def part(n_tiles, lead=()):
        nonlocal at
        n = Hkv * n_tiles * pad
        for d in lead:
            n *= d
        t = ws[at:at + n].view(*lead, Hkv, n_tiles, pad)[..., :S].cpu()
        at += n
        return t

    def in_order(p, lo, hi):       # p [.., n, S]; column j takes tiles lo[j] .. hi[j] - 1
        acc = torch.zeros(p.shape[:-2] + p.shape[-1:])
        for t in range(p.shape[-2]):
            acc = torch.where((lo <= t) & (t < hi), acc + p[..., t, :], acc)
        return acc

    j = torch.arange(S)
    assert torch.equal(col.cpu(), in_order(part(tiles), j // QB, torch.tensor(tiles)))
    assert torch.equal(seen.cpu(), in_order(part(tiles - first), (j // QB - first).clamp(min=0), torch.tensor(tiles - first)))
    if windows:
        bands = part(tiles, (len(windows),))
        for i, w in enumerate(windows):
            assert torch.equal(band[i].cpu(), in_order(bands[i], j // QB, ((j + w - 1) // QB).clamp(max=tiles - 1) + 1))


@pytest.mark.parametrize("S", [1, 64, 65, 128, 129, 192, 193, 257, 321, 449])
@pytest.mark.parametrize("Hkv, G, D", [(2, 4, 128), (1, 7, 64)])
def test_scores_attention_at_every_count_of_key_blocks(S, Hkv, G, D):
    """No, one, two, three and four 64-key blocks per key half (its value and probability blocks alternate between two)."""
    from cold_compress_b200.attention_utils import prefill_attention_stats
    gen = torch.Generator().manual_seed(S)
    q, k, v = (torch.randn(1, h, S, D, generator=gen).bfloat16().cuda() for h in (Hkv * G, Hkv, Hkv))
    y, _ = prefill_attention_stats(q, k, v, obs_len=1)
    rnd = lambda x: x.bfloat16().double()
    kk, vv = (x.repeat_interleave(G, 1).double() for x in (k, v))
    s = rnd(rnd((q.double() @ kk.mT).float()).float() * (1.0 / D ** 0.5))
    s = s.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    want = rnd(s.softmax(-1).float()) @ vv
    y = y.reshape(want.shape).double()
    # a logit's two roundings may fall the other way (2^-8 of |s| <= ~5, hence 2^-6 of a weight), a weight's and y's (2^-9)
    err = (y - want).norm(dim=-1) / (rnd(s.softmax(-1).float()) @ vv.abs()).norm(dim=-1)
    assert err.max().item() <= 2.0 ** -6 + 2.0 ** -8 and ((y - want).norm() / want.norm()).item() <= 2.0 ** -8
