// prompt_rows.cu -- the element-wise work of a prompt layer between its library products, one pass over memory each:
//   * RMS norm of rows                          model.py:452-457   (tensor ops: seven passes, six of them in fp32)
//   * rotation of the q and k columns of the fused projection, split into contiguous heads   model.py:507-519, 377-386
//   * silu(w1 x) * w3 x                          model.py:436-443
// with the reference's rounding points: fp32 inside, bf16 where it has bf16 tensors.  All three are bound by HBM: a thread
// moves 16 bytes per access and keeps a row's elements in registers between the norm's two looks at them.
// (8B layer, 4096 tokens: a norm about 150 -> 12 us, the rotation of q and k about 340 -> 18, the gated unit 107 -> 75.)
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "internal.h"

namespace cc {
namespace {

__device__ __forceinline__ uint4 pack8(const float* v) {
    uint4 u;
    __nv_bfloat162 p[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
    u.x = *reinterpret_cast<uint32_t*>(&p[0]);
    u.y = *reinterpret_cast<uint32_t*>(&p[1]);
    u.z = *reinterpret_cast<uint32_t*>(&p[2]);
    u.w = *reinterpret_cast<uint32_t*>(&p[3]);
    return u;
}

// One CTA per row: NV vectors of eight elements per thread stay in registers.
template <int NV>
__global__ void __launch_bounds__(256) rmsnorm_rows_kernel(const uint4* __restrict__ x, const uint4* __restrict__ w, float eps, uint4* __restrict__ out, int vecs) {
    __shared__ float red[8];
    const size_t base = (size_t)blockIdx.x * vecs;
    uint4 raw[NV];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = threadIdx.x + 256 * i;
        raw[i] = c < vecs ? x[base + c] : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        float f[8];
        unpack8(raw[i], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) ss = fmaf(f[e], f[e], ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = red[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) tot += red[i];
    const float r = rsqrtf(tot / (float)(vecs * 8) + eps);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = threadIdx.x + 256 * i;
        if (c >= vecs) continue;
        float f[8], g[8];
        unpack8(raw[i], f);
        unpack8(w[c], g);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = __bfloat162float(__float2bfloat16_rn(f[e] * r)) * g[e];
        out[base + c] = pack8(f);
    }
}

// Rows [q | k | v] of the fused projection: adjacent pairs of q and k are turned (products and their difference or sum rounded
// one by one, as separate tensor operations round them) into contiguous [S, heads, D] rows.
__global__ void __launch_bounds__(256) rope_rows_kernel(const __nv_bfloat16* __restrict__ qkv, long long ld, const uint4* __restrict__ freqs, uint4* __restrict__ q,
                                                        uint4* __restrict__ k, int S, int q_vecs, int k_vecs, int head_vecs) {
    const int per_row = q_vecs + k_vecs;
    const long long total = (long long)S * per_row;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int s = (int)(i / per_row), c = (int)(i - (long long)s * per_row);
        float x[8], f[8];
        unpack8(*reinterpret_cast<const uint4*>(qkv + s * ld + 8 * c), x);
        unpack8(freqs[(size_t)s * head_vecs + c % head_vecs], f);     // (cos, sin) of four pairs; heads start at whole vectors
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
            const float re = x[e], im = x[e + 1];
            x[e] = __fsub_rn(__fmul_rn(re, f[e]), __fmul_rn(im, f[e + 1]));
            x[e + 1] = __fadd_rn(__fmul_rn(im, f[e]), __fmul_rn(re, f[e + 1]));
        }
        const uint4 o = pack8(x);
        if (c < q_vecs) q[(size_t)s * q_vecs + c] = o;
        else k[(size_t)s * k_vecs + (c - q_vecs)] = o;
    }
}

__global__ void __launch_bounds__(256) silu_mul_kernel(const uint4* __restrict__ a, const uint4* __restrict__ b, uint4* __restrict__ out, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float x[8], y[8];
        unpack8(a[i], x);
        unpack8(b[i], y);
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = __bfloat162float(__float2bfloat16_rn(x[e] / (1.0f + expf(-x[e])))) * y[e];
        out[i] = pack8(x);
    }
}

bool aligned(const void* a, const void* b = nullptr, const void* c = nullptr, const void* d = nullptr) {
    return (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d) & 15) == 0;
}

int check(const char* where) {
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? CC_OK : set_cuda_error(e, where);
}

unsigned blocks_for(long long n) {
    const long long b = (n + 255) / 256;
    return (unsigned)(b < 148 * 32 ? b : 148 * 32);
}

}  // namespace

int rmsnorm_rows_impl(const void* x, const void* w, float eps, void* out, int rows, int dim, cudaStream_t stream) {
    if (!x || !w || !out || rows < 1 || dim < 1) return set_error(CC_ERR_INVALID_ARG, "cc_rmsnorm_rows: bad argument");
    const int vecs = dim / 8;
    if (dim % 8 || vecs > 256 * 8 || !aligned(x, w, out)) return set_error(CC_ERR_UNSUPPORTED_SHAPE, "cc_rmsnorm_rows: rows of whole 16-byte vectors, up to 16384 wide");
#define RN(NV) rmsnorm_rows_kernel<NV><<<rows, 256, 0, stream>>>((const uint4*)x, (const uint4*)w, eps, (uint4*)out, vecs)
    if (vecs <= 256) RN(1);
    else if (vecs <= 512) RN(2);
    else if (vecs <= 1024) RN(4);
    else RN(8);
#undef RN
    return check("cc_rmsnorm_rows launch");
}

int rope_rows_impl(const void* qkv, long long row_stride, const void* freqs, void* q, void* k, int S, int n_q_heads, int n_kv_heads, int head_dim, cudaStream_t stream) {
    if (!qkv || !freqs || !q || !k || S < 1 || n_q_heads < 1 || n_kv_heads < 1 || head_dim < 2) return set_error(CC_ERR_INVALID_ARG, "cc_rope_rows: bad argument");
    if (head_dim % 8 || row_stride % 8 || !aligned(qkv, freqs, q, k)) return set_error(CC_ERR_UNSUPPORTED_SHAPE, "cc_rope_rows: rows of whole 16-byte vectors");
    const int hv = head_dim / 8, qv = n_q_heads * hv, kv = n_kv_heads * hv;
    rope_rows_kernel<<<blocks_for((long long)S * (qv + kv)), 256, 0, stream>>>((const __nv_bfloat16*)qkv, row_stride, (const uint4*)freqs, (uint4*)q, (uint4*)k, S, qv, kv, hv);
    return check("cc_rope_rows launch");
}

int silu_mul_impl(const void* a, const void* b, void* out, long long n, cudaStream_t stream) {
    if (!a || !b || !out || n < 1) return set_error(CC_ERR_INVALID_ARG, "cc_silu_mul: bad argument");
    if (n % 8 || !aligned(a, b, out)) return set_error(CC_ERR_UNSUPPORTED_SHAPE, "cc_silu_mul: whole 16-byte vectors");
    silu_mul_kernel<<<blocks_for(n / 8), 256, 0, stream>>>((const uint4*)a, (const uint4*)b, (uint4*)out, n / 8);
    return check("cc_silu_mul launch");
}

}  // namespace cc
