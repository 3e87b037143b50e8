// launch.cuh -- launches of the sequence kernels that start under their predecessor.
//
// A decode step is a chain of short launches: with programmatic stream serialisation a kernel is set up, and its weights are
// requested, while the one before it still runs.  Two rules keep that safe whatever stands in the stream:
//   * before pdl_wait() a kernel reads parameters only (weights, gains, biases: no kernel of this library writes them);
//   * dependents are released after pdl_wait(), so a kernel that reads ahead meets no kernel older than its own predecessor.
// What a predecessor may have written is read with plain loads, never through the read-only path.
#pragma once
#include <cuda_runtime.h>

namespace ccs {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait_release() {
    pdl_wait();
    pdl_release();
}

template <typename... P, typename... A>
inline cudaError_t launch_under(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

}  // namespace ccs
