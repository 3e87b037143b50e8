"""When the row kernels of a prompt layer must leave a call to the tensor operations: another device, and everything that records
operations to run them again on other tensors."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def norm():
    from cold_compress_b200.model import RMSNorm
    m = RMSNorm(256).to(torch.bfloat16).cuda().requires_grad_(False)
    m.weight.copy_(torch.linspace(0.5, 1.5, 256))
    return m


def _expressions(m, x):
    f = x.float()
    return (f * torch.rsqrt(f.pow(2).mean(-1, keepdim=True) + m.eps)).type_as(x) * m.weight


def _aside(rows):
    """A contiguous tensor that does not start on a 16-byte boundary: not one for the kernels."""
    t = torch.randn(rows * 256 + 4, device="cuda").bfloat16()[4:].view(rows, 256)
    assert t.is_contiguous() and t.data_ptr() % 16 == 8
    return t


def test_tensors_of_another_device(norm, monkeypatch):
    from cold_compress_b200 import ops
    x = torch.randn(3, 256, device="cuda").bfloat16()
    assert ops.plain_rows(x, norm.weight)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 1)
    assert not ops.plain_rows(x, norm.weight)


@pytest.mark.parametrize("record", ["jit.trace", "make_fx", "compile"])
def test_what_is_recorded_runs_on_other_tensors(norm, record):
    from torch.fx.experimental.proxy_tensor import make_fx
    x, y = torch.randn(3, 256, device="cuda").bfloat16(), _aside(5)
    if record == "jit.trace":
        f = torch.jit.trace(norm, x)
    elif record == "make_fx":
        f = make_fx(norm)(x)
        y = _aside(3)
    else:
        f = torch.compile(norm, fullgraph=True, backend="eager")
    for t in (x, y):
        torch.testing.assert_close(f(t), _expressions(norm, t), rtol=2.0 ** -7, atol=0)      # a recorder may fuse operations


def test_a_single_number_and_other_widths(norm):
    x = torch.tensor(2.0, device="cuda").bfloat16()
    assert torch.equal(norm(x), _expressions(norm, x)) and norm(x).shape == (256,)
    one = torch.randn(3, 1, device="cuda").bfloat16()
    assert torch.equal(norm(one), _expressions(norm, one))
