"""CC_B200_PDL=0 turns programmatic dependent launch off in both libraries: the edges of a captured graph say which it was."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent
CODE = """
import ctypes as C
import torch
from cold_compress_b200 import ops, seq_ops
w, x, out = torch.randn(256, 512, device="cuda"), torch.randn(1, 512, device="cuda"), torch.empty(1, 256, device="cuda")
wb, xb, ob = torch.randn(512, 512, device="cuda").bfloat16(), torch.randn(512, device="cuda").bfloat16(), torch.empty(512, device="cuda").bfloat16()
for call in (lambda: seq_ops.gemv_multi([(x, w, out)]), lambda: ops.gemv_residual(xb, None, 1e-5, wb, None, ob, [], [], None)):
    call()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        call()
        call()
    n, before, after, data = C.c_size_t(4), (C.c_void_p * 4)(), (C.c_void_p * 4)(), (C.c_ubyte * 32)()
    assert C.CDLL("libcuda.so.1").cuGraphGetEdges_v2(C.c_void_p(g.raw_cuda_graph()), before, after, data, C.byref(n)) == 0 and n.value == 1
    print("edge", data[2])          # CUgraphEdgeData: from_port, to_port, type
"""


@pytest.mark.parametrize("value,edges", [("0", ["0", "0"]), ("1", ["1", "1"])])
def test_the_switch_reaches_both_libraries(value, edges):
    done = subprocess.run([sys.executable, "-c", CODE], cwd=ROOT, env={**os.environ, "CC_B200_PDL": value, "PYTHONPATH": str(ROOT)}, capture_output=True,
                          text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
    assert [x.split()[1] for x in done.stdout.splitlines() if x.startswith("edge")] == edges
