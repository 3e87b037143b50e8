"""One-token products: the gated unit on the way out of its product, against the product and the unit apart and against 64 bits."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("F,K", [(1, 8), (3, 5), (17, 64), (40, 33), (500, 1024), (1001, 256), (2816, 1024), (9000, 72)])
def test_gated_unit_on_the_way_out(dtype, F, K):
    from cold_compress_b200 import _lib, seq_ops
    g = torch.Generator(device=DEV).manual_seed(F + K)
    x = torch.randn(1, K, device=DEV, generator=g).to(dtype)
    w = (torch.randn(2 * F, K, device=DEV, generator=g) * K ** -0.5).to(dtype)
    fused, rows, apart = torch.empty(1, F, dtype=dtype, device=DEV), torch.empty(1, 2 * F, device=DEV), torch.empty(1, F, dtype=dtype, device=DEV)
    seq_ops.gemv_multi([(x, w, fused)], unit=_lib.ACT_SILU)
    seq_ops.gemv_multi([(x, w, rows)])
    seq_ops.gated_unit(rows, 0, F, apart, _lib.ACT_SILU)
    assert torch.equal(fused, apart)                   # the same sums, the same unit, the same rounding
    r = x.double() @ w.double().t()
    want = torch.nn.functional.silu(r[:, :F]) * r[:, F:]
    # products of unit variance: K roundings of the sum walk at random, bf16 rounds the result once
    tol = 2.0 ** -8 * want.abs() + 8 * math.sqrt(K) * 2.0 ** -24 if dtype == torch.bfloat16 else 64 * math.sqrt(K) * 2.0 ** -24 * (1 + want.abs())
    assert ((fused.double() - want).abs() <= tol).all()


def test_gated_unit_on_the_way_out_refuses():
    import ctypes as C

    from cold_compress_b200 import _lib
    lib, g = _lib.load_seq(), _lib.CcSeqGemvMulti()
    t = torch.zeros(64, device=DEV)
    g.n_jobs, g.w_dtype = 1, _lib.DT_F32
    b = g.job[0]
    b.x, b.W, b.out = (t.data_ptr(),) * 3
    b.x_dtype, b.N, b.K, b.off_up, b.pair = _lib.DT_F32, 6, 4, -1, 2
    assert lib.cc_seq_gemv_multi(C.byref(g), None) < 0 and b"way out" in lib.cc_seq_last_error()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("F,K,N", [(17, 64, 33), (500, 1024, 2001), (1001, 257, 64)])
def test_a_unit_beside_plain_products(dtype, F, K, N):
    """A launch of a unit and of plain products gives each job what a launch of its own gives it."""
    from cold_compress_b200 import _lib, seq_ops
    g = torch.Generator(device=DEV).manual_seed(F)
    x = torch.randn(1, K, device=DEV, generator=g).to(dtype)
    w, v = ((torch.randn(n, K, device=DEV, generator=g) * K ** -0.5).to(dtype) for n in (2 * F, N))
    unit, rows, alone = torch.empty(1, F, dtype=dtype, device=DEV), torch.empty(1, N, device=DEV), torch.empty(1, N, device=DEV)
    both = torch.empty_like(unit)
    seq_ops.gemv_multi([(x, w, unit)], unit=_lib.ACT_SILU)
    seq_ops.gemv_multi([(x, v, alone)])
    seq_ops.gemv_multi([(x, w, both), (x, v, rows)], unit=_lib.ACT_SILU)
    # the rows may be split over another number of warps beside other jobs: the same products, added in another order
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 64 * math.sqrt(K) * 2.0 ** -24
    assert ((both.double() - unit.double()).abs() <= tol * (1 + unit.double().abs())).all()
    assert ((rows - alone).abs() <= 64 * math.sqrt(K) * 2.0 ** -24 * (1 + alone.abs())).all()
    want = x.double() @ v.double().t()
    assert ((rows.double() - want).abs() <= 64 * math.sqrt(K) * 2.0 ** -24 * (1 + want.abs())).all()
