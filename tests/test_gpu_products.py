"""One-token products (gemv_multi, head_gemv) and the embedding under bounded norms: every split of rows and columns over warps
against 64-bit products, and weights that the launch just before has written."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(out, w, x):
    want = w.double() @ x.to(w.dtype).double()
    # K products in fp32 in some order: relative 2^-24 sqrt(K) of the terms' root sum of squares, four times that
    bound = 4 * 2.0 ** -24 * math.sqrt(w.shape[1]) * (w.double().square() @ x.to(w.dtype).double().square()).sqrt() + 1e-30
    bad = (out.double() - want).abs() > bound
    assert not bad.any(), (int(bad.sum()), bad.nonzero()[:4].flatten().tolist())


# (N, K): eight, four, two warps and one per pair of rows (by how many pairs there are and how long a row is), more rows than
# the GPU holds at once (9472 pairs ...), odd counts whose last pair or group of sixteen is partial, rows that end within, at
# and past the vectors a lane has in flight (128 and 256 of them per warp), and rows that are not whole vectors
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("N,K", [(1, 4096), (3, 8192), (590, 4096), (1183, 4096), (2367, 2048), (4735, 1016), (4735, 1024), (4737, 1032), (4737, 2048),
                                 (9471, 512), (9472, 2056), (9473, 2048), (9473, 2064), (19001, 1000), (19001, 1024), (32001, 512), (9473, 1027), (20, 515),
                                 (40000, 8)])
def test_every_split_of_a_product(N, K, dtype):
    from cold_compress_b200 import seq_ops
    gen = torch.Generator(device="cuda").manual_seed(N + K)
    w, x = (torch.randn(*s, device="cuda", generator=gen) for s in ((N, K), (1, K)))
    w, out = w.to(dtype), torch.full((1, N + 16), math.nan, device="cuda")
    seq_ops.gemv_multi([(x, w, out[:, :N])])
    _check(out[0, :N], w, x[0])
    assert out[0, N:].isnan().all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("sizes", [[(9473, 2048), (77, 512)], [(5, 512), (19001, 520), (33, 2056)], [(300, 4096), (301, 1024)], [(100, 2048), (17, 70)]])
def test_products_of_different_sizes_in_one_launch(sizes, dtype):
    from cold_compress_b200 import seq_ops
    gen = torch.Generator(device="cuda").manual_seed(len(sizes))
    jobs = [(torch.randn(1, K, device="cuda", generator=gen), torch.randn(N, K, device="cuda", generator=gen).to(dtype), torch.empty(1, N, device="cuda"))
            for N, K in sizes]
    seq_ops.gemv_multi(jobs)
    for x, w, out in jobs:
        _check(out[0], w, x[0])


def test_weights_written_by_the_launch_before():
    """A copy into the weights, then the product, with nothing between: the product's launch may start under the copy."""
    from cold_compress_b200 import seq_ops
    gen = torch.Generator(device="cuda").manual_seed(1)
    N, K, H, E = 1500, 4096, 16, 4096
    randn = lambda *s: torch.randn(*s, device="cuda", generator=gen)  # noqa: E731
    ws, x = [randn(N, K).bfloat16() for _ in range(3)], randn(1, K)
    hw, hx = [randn(H, 128, 256).bfloat16() for _ in range(3)], randn(1, H * 256)
    gains, table, tokens = [randn(2, E) for _ in range(3)], randn(8, E).bfloat16(), torch.tensor([3], dtype=torch.int32, device="cuda")
    w, head, gain, alpha = ws[0].clone(), hw[0].clone(), gains[0].clone(), torch.full((1,), 0.5, device="cuda")

    def product(i, out):
        w.copy_(ws[i])
        seq_ops.gemv_multi([(x, w, out)])

    def heads(i, out):
        head.copy_(hw[i])
        seq_ops.head_gemv(head, hx, 256, out, 128)

    def embed(i, out):
        gain.copy_(gains[i])
        seq_ops.embed_bounded(tokens, table, (alpha, gain[0], gain[1]), out)

    for call, n in ((product, N), (heads, H * 128), (embed, E)):
        want = []
        for i in range(3):
            out = torch.empty(1, n, device="cuda")
            call(i, out)
            torch.cuda.synchronize()
            call(i, out)          # the same weights again: nothing to be late
            torch.cuda.synchronize()
            want.append(out.clone())
        outs = torch.empty(300, 1, n, device="cuda")
        for step in range(300):
            call(step % 3, outs[step])
        for step in range(300):
            assert torch.equal(outs[step], want[step % 3]), (call.__name__, step)
