"""Softmax and its arg-max as one launch: sizes around what a thread keeps, ties, and numbers that are none."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("V", [2, 3, 5, 31, 1000, 4097, 32000, 32003, 131072, 131075, 152064])
@pytest.mark.parametrize("scale", [1.0, 30.0])
def test_greedy_is_the_softmax_and_its_first_largest_index(V, scale):
    from cold_compress_b200 import seq_ops
    x = torch.randn(V, device=DEV, generator=torch.Generator(device=DEV).manual_seed(V)) * scale
    token, probs = seq_ops.greedy(x)
    want, gap = torch.softmax(x.double(), 0), (x.max() - x).double()
    # the difference of the logits is rounded once (2^-24 of it moves the exponential by as much), the exponential, the sum of sums and the quotient
    assert ((probs.double() - want).abs() <= 2.0 ** -24 * (gap + 24) * want + 1e-37).all()
    assert token.dtype == torch.int32 and int(token) == int(torch.argmax(probs)) and float(probs[token.long()]) == float(probs.max())


def test_greedy_ties_and_what_is_no_number():
    from cold_compress_b200 import seq_ops
    from cold_compress_b200.generation_utils import greedy
    x = torch.zeros(50000, device=DEV)
    x[[777, 778, 49999, 20000]] = 3.0
    assert int(seq_ops.greedy(x)[0]) == 777
    x[777] -= 1e-9                                     # rounds away
    assert int(seq_ops.greedy(x)[0]) == 777
    for bad in (float("nan"), float("inf")):
        y = x.clone()
        y[40000] = bad
        want = torch.softmax(y, 0)
        tok, p = seq_ops.greedy(y)
        assert torch.equal(p.isnan(), want.isnan()) and int(tok) == int(torch.argmax(want))
    y = torch.full((100,), -float("inf"), device=DEV)
    y[7] = 0.0
    tok, p = seq_ops.greedy(y)
    assert int(tok) == 7 and float(p.sum()) == 1.0
    # other types, rows that do not start on a 16-byte boundary and rows under differentiation go through tensor operations
    for row in (x.double(), x[1:], x.clone().requires_grad_(True)):
        tok, p = greedy(row.view(1, 1, -1), None)
        assert p.dtype == row.dtype and int(tok) == int(torch.argmax(p.detach()))
    tok, p = greedy(x.view(1, 1, -1), torch.tensor([5], dtype=torch.int32, device=DEV))
    assert int(tok) == 5 and p.shape == x.shape


def test_greedy_under_tracing_vmap_and_capture():
    from cold_compress_b200.generation_utils import greedy
    gen = torch.Generator(device=DEV).manual_seed(2)
    a, b = (torch.randn(1, 1, 5000, device=DEV, generator=gen) * 4 for _ in range(2))
    traced = torch.jit.trace(lambda x: greedy(x, None), (a,), check_trace=False)
    tok, p = traced(b)                                 # what was recorded runs on other logits
    assert int(tok) == int(b.argmax()) and torch.allclose(p, torch.softmax(b[0, -1], -1), rtol=1e-5, atol=0)
    many = torch.vmap(lambda x: greedy(x, None)[1])(torch.stack([a, b]))
    assert torch.equal(many, torch.softmax(torch.stack([a, b])[:, 0, -1], -1))
    held = a.clone()
    greedy(held, None)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        tok, p = greedy(held, None)
    for x in (a, b):
        held.copy_(x)
        graph.replay()
        want_tok, want = greedy(x, None)
        assert torch.equal(tok, want_tok) and torch.equal(p, want)
