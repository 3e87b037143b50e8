// launch.cuh -- launches of the sequence kernels that start under their predecessor.
//
// A decode step is a chain of short launches: with programmatic stream serialisation a kernel is set up, and its weights are
// brought into L2, while the one before it still runs.  The predecessor can be anyone's, the copy that writes the weights
// included, and its stores are visible only after pdl_wait().  So:
//   * before pdl_wait() a kernel takes no value from memory; it may ask for lines in L2 (ask_l2), which is a hint: L2 is where
//     all stores meet, and nothing depends on what a line held when it was asked for;
//   * memory is read with plain loads, never through the read-only path, whose lines may be older than this kernel's wait;
//   * dependents are released after pdl_wait(), so a kernel that starts early meets no kernel older than its own predecessor.
#pragma once
#include <cuda_runtime.h>
#include <stdlib.h>

#include "../smem_limit.cuh"

namespace ccs {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait_release() {
    pdl_wait();
    pdl_release();
}

__device__ __forceinline__ void ask_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// CC_B200_PDL=0 turns programmatic dependent launch off, here as in the main library.
inline bool pdl_enabled() {
    static const bool on = [] { const char* e = getenv("CC_B200_PDL"); return !(e && e[0] == '0'); }();
    return on;
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
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

}  // namespace ccs
