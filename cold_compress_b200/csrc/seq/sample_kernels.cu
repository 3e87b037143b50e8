// sample_kernels.cu -- the end of a decode step: probabilities of one row of logits and the token with the largest one.
//
// As tensor operations these are three launches (softmax, arg-max, conversion), the first two on a single SM.  Here a cluster of eight
// CTAs shares the row, keeps it in registers and meets three times through distributed shared memory (largest logit, sum, first index
// of the largest probability).  Bound: those exchanges; 128 KB of logits are nothing.  Back to back in a graph, 32,000 logits 4.6 us
// (20.8 as tensor operations), 128,256 7.1 (63.2).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../../include/cc_b200_seq.h"
#include "launch.cuh"

namespace ccs {

int fail(int code, const char* msg);
int cuda_check(const char* where);

namespace {

constexpr int SM_CTAS = 8, SM_THREADS = 1024, SM_WARPS = SM_THREADS / 32, SM_KEEP = 4;      // SM_KEEP: 16-byte vectors a thread keeps

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void to_cta(uint32_t* slot, uint32_t cta, uint32_t v) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(slot)), "r"(cta));
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float larger(float a, float b) { return a > b || a != a ? a : b; }      // a NaN stays

// probs = softmax(logits) in fp32, token = the first index of the largest probability (0 when they are not numbers)
__global__ void __cluster_dims__(SM_CTAS, 1, 1) __launch_bounds__(SM_THREADS) greedy_kernel(const float* logits, int V, float* probs, int32_t* token) {
    __shared__ uint32_t part[3][SM_CTAS], warps[SM_WARPS];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = blockIdx.x;
    // every CTA has started before one stores into another
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    pdl_wait_release();
    const int vecs = V / 4, each = (vecs + SM_CTAS - 1) / SM_CTAS, first = cta * each, last = min(first + each, vecs), tail = V - 4 * vecs;
    const bool tails = cta == SM_CTAS - 1 && tid < tail;      // entries behind the last whole vector
    const float4* in = reinterpret_cast<const float4*>(logits);
    float4 keep[SM_KEEP];
#pragma unroll
    for (int i = 0; i < SM_KEEP; ++i)
        if (first + tid + i * SM_THREADS < last) keep[i] = in[first + tid + i * SM_THREADS];
    // what a thread does not keep it reads again
    auto each_vec = [&](auto&& f) {
#pragma unroll
        for (int i = 0; i < SM_KEEP; ++i)
            if (first + tid + i * SM_THREADS < last) f(first + tid + i * SM_THREADS, keep[i]);
        for (int v = first + tid + SM_KEEP * SM_THREADS; v < last; v += SM_THREADS) f(v, in[v]);
    };
    const float odd = tails ? logits[4 * vecs + tid] : -INFINITY;
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");

    float m = odd;
    each_vec([&](int, const float4& x) { m = larger(larger(larger(m, x.x), larger(x.y, x.z)), x.w); });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = larger(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (lane == 0) warps[warp] = __float_as_uint(m);
    __syncthreads();
    if (warp == 0) {
        m = __uint_as_float(warps[lane]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = larger(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane < SM_CTAS) to_cta(&part[0][cta], lane, __float_as_uint(m));
    }
    cluster_sync();
    m = __uint_as_float(part[0][0]);
#pragma unroll
    for (int c = 1; c < SM_CTAS; ++c) m = larger(m, __uint_as_float(part[0][c]));

    float sum = tails ? expf(odd - m) : 0.f;
    each_vec([&](int, const float4& x) { sum += (expf(x.x - m) + expf(x.y - m)) + (expf(x.z - m) + expf(x.w - m)); });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) warps[warp] = __float_as_uint(sum);      // read by warp 0 before the barrier above: free again
    __syncthreads();
    if (warp == 0) {
        sum = __uint_as_float(warps[lane]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane < SM_CTAS) to_cta(&part[1][cta], lane, __float_as_uint(sum));
    }
    cluster_sync();
    sum = 0.f;
#pragma unroll
    for (int c = 0; c < SM_CTAS; ++c) sum += __uint_as_float(part[1][c]);

    const float top = expf(m - m) / sum;      // of the largest logit; others may round to the same
    uint32_t best = 0xffffffffu;
    auto take = [&](int i, float x) {
        const float p = expf(x - m) / sum;
        if (p == top) best = min(best, (uint32_t)i);
        return p;
    };
    float4* const out = reinterpret_cast<float4*>(probs);
    each_vec([&](int v, const float4& x) { out[v] = make_float4(take(4 * v, x.x), take(4 * v + 1, x.y), take(4 * v + 2, x.z), take(4 * v + 3, x.w)); });
    if (tails) probs[4 * vecs + tid] = take(4 * vecs + tid, odd);
    best = __reduce_min_sync(0xffffffffu, best);
    if (lane == 0) warps[warp] = best;
    __syncthreads();
    if (warp == 0) {
        best = __reduce_min_sync(0xffffffffu, warps[lane]);
        if (lane == 0) to_cta(&part[2][cta], 0, best);
    }
    cluster_sync();
    if (cta == 0 && warp == 0) {
        best = __reduce_min_sync(0xffffffffu, lane < SM_CTAS ? part[2][lane] : 0xffffffffu);
        if (lane == 0) *token = best == 0xffffffffu ? 0 : (int32_t)best;
    }
}

}  // namespace
}  // namespace ccs

using namespace ccs;

extern "C" int cc_seq_greedy(const float* logits, int32_t V, float* probs, int32_t* token, void* stream) {
    if (!logits || !probs || !token || V < 1) return fail(CC_SEQ_ERR_INVALID_ARG, "greedy: bad argument");
    if (((uintptr_t)logits | (uintptr_t)probs) & 15) return fail(CC_SEQ_ERR_INVALID_ARG, "greedy: rows on 16-byte boundaries expected");
    launch_under(greedy_kernel, dim3(SM_CTAS), dim3(SM_THREADS), 0, (cudaStream_t)stream, logits, V, probs, token);
    return cuda_check("greedy_kernel");
}
