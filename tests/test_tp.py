"""Tensor-parallel tests.  CPU: world_size-2 gloo run of the sharding + all-reduce host logic.
GPU (needs >= 2 devices): head-sharded decode reproduces the unsharded run."""
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent


def _torchrun(n, *args, timeout=600):
    env = dict(os.environ, OMP_NUM_THREADS="2")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", f"--nproc-per-node={n}",
           "--master-addr", "127.0.0.1", "--master-port", "29517", str(ROOT / "tests" / "tp_worker.py"), *args]
    return subprocess.run(cmd, capture_output=True, text=True, timeout=timeout, env=env, cwd=ROOT)


@pytest.mark.parametrize("world", [2, 4, 8])
def test_tp_host_logic_gloo(world):
    env_cuda = os.environ.get("CUDA_VISIBLE_DEVICES")
    os.environ["CUDA_VISIBLE_DEVICES"] = ""
    try:
        r = _torchrun(world, "heavy_hitter")
    finally:
        if env_cuda is None:
            os.environ.pop("CUDA_VISIBLE_DEVICES", None)
        else:
            os.environ["CUDA_VISIBLE_DEVICES"] = env_cuda
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-3000:]
    assert r.stdout.count("tp host logic ok") == world


@pytest.mark.gpu
@pytest.mark.parametrize("strategy", ["heavy_hitter", "recent_global", "l2", "heavy_hitter_compressed",
                                      "heavy_hitter_fused", "recent_global_fused", "heavy_hitter_nccl"])
def test_tp_decode_world2(strategy):
    if torch.cuda.device_count() < 2:
        pytest.skip("needs 2 GPUs")
    r = _torchrun(2, strategy)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-3000:]
    assert r.stdout.count("tp decode ok") == 2


@pytest.mark.gpu
@pytest.mark.parametrize("strategy", ["heavy_hitter", "recent_global"])
def test_tp_decode_world4(strategy):
    """The whole-token kernel with 4 ranks (one KV head per rank): all-reduces inside the kernel over NVLink."""
    if torch.cuda.device_count() < 4:
        pytest.skip("needs 4 GPUs")
    r = _torchrun(4, strategy)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-3000:]
    assert r.stdout.count("tp decode ok") == 4


@pytest.mark.gpu
@pytest.mark.parametrize("strategy", ["heavy_hitter", "recent_global"])
def test_tp_decode_world8(strategy):
    """Eight ranks, one KV head each (the tensor-parallel layout of Llama-3-8B): the whole-token kernel's
    second round of partial-vector reads (ranks 4-7) and its 64-CTA-per-head attention stage.  Needs 8 GPUs; not run yet:
    a recorded line of the benchmark with 8 ranks is the only evidence at this world size."""
    if torch.cuda.device_count() < 8:
        pytest.skip("needs 8 GPUs")
    r = _torchrun(8, strategy)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-3000:]
    assert r.stdout.count("tp decode ok") == 8
