"""CPU: how much shared memory a kernel may be launched with (csrc/smem_limit.cuh), against a runtime that only writes down what it is asked
for: the limit belongs to a kernel on a device, all that the device has is asked for once, and a failure is not remembered."""
import re
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "cold_compress_b200" / "csrc"

PROGRAM = r"""
#include "smem_limit.cuh"
#include <assert.h>
#include <thread>
#include <vector>
static thread_local int device = 0;
static std::atomic<int> fails{0}, sets{0}, last{0};
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr a, int) { assert(a == cudaDevAttrMaxSharedMemoryPerBlockOptin); *v = 232448; return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void*) { *a = {}; a->sharedSizeBytes = 1000; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, enum cudaFuncAttribute a, int v) {
    assert(a == cudaFuncAttributeMaxDynamicSharedMemorySize);
    if (fails > 0) { --fails; return cudaErrorInvalidValue; }
    ++sets;
    last = v;
    return cudaSuccess;
}
}
static void kernel(int) {}
int main() {
    SmemLimit limit, other;
    assert(limit.allow(kernel, 4 * 1024) == cudaSuccess && sets == 0);
    assert(limit.allow(kernel, 60 * 1024) == cudaSuccess && sets == 1 && last == 232448 - 1000);
    assert(limit.allow(kernel, 200 * 1024) == cudaSuccess && sets == 1);
    device = 1;                                                        // another device knows nothing of the first
    assert(limit.allow(kernel, 60 * 1024) == cudaSuccess && sets == 2);
    device = 0;
    assert(limit.allow(kernel, 60 * 1024) == cudaSuccess && sets == 2);
    assert(other.allow(kernel, 60 * 1024) == cudaSuccess && sets == 3);
    device = 70;                                                       // past the devices that are remembered: asked for each time
    assert(limit.allow(kernel, 60 * 1024) == cudaSuccess && limit.allow(kernel, 60 * 1024) == cudaSuccess && sets == 5);
    device = 2;
    fails = 1;
    assert(limit.allow(kernel, 60 * 1024) == cudaErrorInvalidValue && limit.allow(kernel, 60 * 1024) == cudaSuccess && sets == 6);
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&, t] { device = 3 + t % 2; for (int i = 0; i < 1000; ++i) assert(limit.allow(kernel, (40 + 10 * t) * 1024) == cudaSuccess && last == 231448); });
    for (auto& t : threads) t.join();
    return 0;
}
"""


def test_the_limit_is_asked_for_once_per_kernel_and_device(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", str(CSRC), "-I/usr/local/cuda/include", "-x", "c++", str(tmp_path / "t.cpp"), "-o", str(tmp_path / "t")], check=True)
    subprocess.run([str(tmp_path / "t")], check=True, timeout=60)


def test_launchers_ask_for_it_so():
    """gemv.cu, decode_step.cu and decode_token.cu keep or plan by device themselves."""
    own = {"gemv.cu", "decode_step.cu", "decode_token.cu", "smem_limit.cuh"}
    for f in CSRC.rglob("*.cu*"):
        text = re.sub(r"//[^\n]*", "", f.read_text())
        assert f.name in own or "cudaFuncAttributeMaxDynamicSharedMemorySize" not in text, f.name
        assert not re.search(r"static (bool|size_t) configured", text), f.name
    assert "raised[i].dev == dev" in (CSRC / "gemv.cu").read_text()


def test_what_is_looked_up_once_is_there_for_every_thread():
    """A flag that says 'looked up' before the result is stored let a second thread go on without it."""
    for f in (CSRC / "prefill_attn.cu", CSRC / "seq" / "tensor_map.cuh"):
        text = f.read_text()
        body = text[text.index("EncodeTiledFn encode_fn() {"):]
        body = body[:body.index("\n}\n")]
        assert re.findall(r"\bstatic\b.*", body) and all(x.startswith("static const EncodeTiledFn fn = [] {") for x in re.findall(r"\bstatic\b.*", body)), f.name
