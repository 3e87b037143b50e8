// wkv_segment_kernels.cu -- the matrix-state recurrence of cc_seq_wkv over many tokens, segments of the sequence side by side.
//
// Token after token, 4096 tokens of 32 heads of 64 are 4096 dependent steps at one warp per scheduler: the chain bounds it, not
// the arithmetic.  The decay is diagonal, so what a segment adds to the state does not depend on the state it starts from:
//   1. per segment, sum_t (k_t * w_{t+1} * ... * w_end) v_t^T and the product of its decays: products of two matrices for 16 tokens
//      at a time.  No decay is ever divided by: every factor is a product of numbers in (0, 1];
//   2. the states at the segments' starts, one after another over the segments and beside each other over the elements;
//   3. the recurrence inside every segment from its own start.
// Where a start is not finite, 2. looks at the tokens (a product of decays may underflow where no decay is zero), and where a sum is not,
// 3. walks its segment again with the bonus per row, so that infinities and NaN come out as they do token after token (4096 tokens of
// 32 heads of 64 with keys that are all NaN: 330 us).
// Rows on other than 16-byte boundaries are staged 4 bytes at a time: the same sums, so the same bits.
// One multiplication and addition per state element and token more than the plain recurrence, for segments times the parallelism:
// Back to back in a graph, 4096 tokens of 32 heads of 64 go from 405 us to 144, of 4 heads from 387 to 38, of 64 heads of 128 from
// 1663 to 1040.  Now bound by the fp32 pipe (69 % busy in 3., 50 % in 1.; 9 warps of up to 168 registers an SM).
// Against 64 bits the outputs are as far off as token after token (1.31e-7 and 1.34e-7 of their norm), with other roundings.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../../include/cc_b200_seq.h"
#include "../smem_limit.cuh"

namespace ccs {
int fail(int code, const char* msg);
int cuda_check(const char* where);
}  // namespace ccs

namespace ccw {
using ccs::cuda_check;
using ccs::fail;

typedef unsigned long long f32x2;      // a pair of fp32 values: one instruction for two operations, each rounded as the scalar one
__device__ __forceinline__ f32x2 pair(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpair(f32x2 r, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void cp_async16_or_zero(void* dst, const void* src, bool have) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(have ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4_or_zero(void* dst, const void* src, bool have) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(have ? 4 : 0) : "memory");
}
// four floats of a row, on any boundary of a float unless VEC
template <bool VEC>
__device__ __forceinline__ void stage4(float* dst, const float* src, bool have) {
    if constexpr (VEC) {
        cp_async16_or_zero(dst, src, have);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) cp_async4_or_zero(dst + i, src + i, have);
    }
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct Segments {
    float* w;       // [T, H * D] decays
    float* X;       // [n, H, D, D] what segment s - 1 adds to the state, then the state that segment s starts from
    float* P;       // [n, H, D] product of a segment's decays
    int len, n;     // tokens per segment (the last one may have fewer), segments
};

constexpr int TILE = 64, STATE_THREADS = 64, TB = 16;      // state tile, threads of the first kernel, tokens of a batch

// Decays of a segment's tokens, their product, and (but for the last segment, whose end nobody starts from) what the segment adds
// to a 64 x 64 tile of the state.  A thread first takes a channel of a batch of tokens, then 16 rows x 4 columns of the tile.
template <bool VEC>
__global__ void __launch_bounds__(STATE_THREADS, 8) wkv_segment_state_kernel(const CcSeqWkv a, const Segments g) {
    __shared__ float4 smw4[2 * 3 * TB * TILE / 4];
    __shared__ float4 decay4[TILE / 4];
    float* const sm = reinterpret_cast<float*>(smw4);
    constexpr int ROWS = TB * TILE;
    const int tid = threadIdx.x, s = blockIdx.x, h = blockIdx.y, tiles = (a.D + TILE - 1) / TILE;
    const int i0 = (int)(blockIdx.z / tiles) * TILE, j0 = (int)(blockIdx.z % tiles) * TILE;
    const bool add = s + 1 < g.n, keep = j0 == 0;
    if (!add && !keep) return;
    const size_t HD = (size_t)a.H * a.D;
    const int first = s * g.len, count = min(g.len, a.T - first);
    auto fetch = [&](int b, float* buf) {       // [raw decay | key | value] rows of TB tokens
        const int nt = min(TB, count - b * TB), x = 4 * (tid % (TILE / 4));
        const bool in = i0 + x < a.D, inv = j0 + x < a.D;
#pragma unroll
        for (int t = tid / (TILE / 4); t < TB; t += STATE_THREADS / (TILE / 4)) {
            const size_t row = (size_t)(first + b * TB + (t < nt ? t : 0)) * HD + (size_t)h * a.D;
            float* const d = buf + t * TILE + x;
            stage4<VEC>(d, a.wraw + row + (in ? i0 + x : 0), t < nt && in);
            if (!add) continue;
            stage4<VEC>(d + ROWS, a.k + row + (in ? i0 + x : 0), t < nt && in);
            stage4<VEC>(d + 2 * ROWS, a.v + row + (inv ? j0 + x : 0), t < nt && inv);
        }
        cp_async_commit();
    };
    const bool in_c = i0 + tid < a.D;
    const float w0 = in_c ? a.w0[(size_t)h * a.D + i0 + tid] : 0.f;
    const int ty = tid / 16, tx = tid % 16;
    float total = 1.f;      // product of all decays
    f32x2 acc[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int x = 0; x < 4; ++x) acc[r][x] = 0ull;
    const int nb = (count + TB - 1) / TB;
    fetch(0, sm);
    int cur = 0;
    for (int b = 0; b < nb; ++b, cur ^= 1) {
        float* const buf = sm + cur * 3 * ROWS;
        const int nt = min(TB, count - b * TB);
        if (b + 1 < nb) {
            fetch(b + 1, sm + (cur ^ 1) * 3 * ROWS);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        float* const wt = g.w + (size_t)(first + b * TB) * HD + (size_t)h * a.D + i0 + tid;
        float carry = 1.f;      // product of the decays behind a token, inside the batch
#pragma unroll 4
        for (int t = TB - 1; t >= 0; --t) {
            const float w = t < nt ? expf(-expf(buf[t * TILE + tid] + w0)) : 1.f;
            if (t < nt && in_c && keep) wt[(size_t)t * HD] = w;
            if (add) buf[ROWS + t * TILE + tid] *= carry;
            carry *= w;
        }
        total *= carry;
        reinterpret_cast<float*>(decay4)[tid] = carry;
        __syncthreads();
        if (add) {
            // the sum so far goes through the batch's decays, so that its roundings decay as they do token after token
            if (b > 0) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 dv = decay4[4 * ty + q];
                    const f32x2 d2[2] = {pair(dv.x, dv.y), pair(dv.z, dv.w)};
#pragma unroll
                    for (int e = 0; e < 2; ++e)
#pragma unroll
                        for (int x = 0; x < 4; ++x) acc[2 * q + e][x] = mul2(d2[e], acc[2 * q + e][x]);
                }
            }
#pragma unroll 4
            for (int t = 0; t < TB; ++t) {
                const float4 vv = reinterpret_cast<const float4*>(buf + 2 * ROWS + t * TILE)[tx];
                const f32x2 v2[4] = {pair(vv.x, vv.x), pair(vv.y, vv.y), pair(vv.z, vv.z), pair(vv.w, vv.w)};
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const float4 kv = reinterpret_cast<const float4*>(buf + ROWS + t * TILE)[4 * ty + q];
                    const f32x2 k2[2] = {pair(kv.x, kv.y), pair(kv.z, kv.w)};
#pragma unroll
                    for (int e = 0; e < 2; ++e)
#pragma unroll
                        for (int x = 0; x < 4; ++x) acc[2 * q + e][x] = fma2(k2[e], v2[x], acc[2 * q + e][x]);
                }
            }
        }
        __syncthreads();      // the batch is consumed
    }
    if (!add) return;
    if (keep && in_c) g.P[((size_t)s * a.H + h) * a.D + i0 + tid] = total;
    float* const X = g.X + ((size_t)(s + 1) * a.H + h) * a.D * a.D;
    const int j = j0 + 4 * tx;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        float lo[4], hi[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) unpair(acc[r][x], lo[x], hi[x]);
        const int i = i0 + 16 * ty + 2 * r;
        if (j >= a.D || i >= a.D) continue;      // rows come in pairs: D is a multiple of 4
        *reinterpret_cast<float4*>(X + (size_t)i * a.D + j) = make_float4(lo[0], lo[1], lo[2], lo[3]);
        *reinterpret_cast<float4*>(X + (size_t)(i + 1) * a.D + j) = make_float4(hi[0], hi[1], hi[2], hi[3]);
    }
}

__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= 3.402823466e38f; }
__device__ __forceinline__ bool finite(const float4& x) { return finite(x.x) && finite(x.y) && finite(x.z) && finite(x.w); }
__device__ __forceinline__ bool none_left(const float4& x) { return x.x != x.x && x.y != x.y && x.z != x.z && x.w != x.w; }
__device__ __forceinline__ float4 fma4(float p, const float4& x, const float4& y) {
    return make_float4(fmaf(p, x.x, y.x), fmaf(p, x.y, y.y), fmaf(p, x.z, y.z), fmaf(p, x.w, y.w));
}
// Four elements of a state row through segment s, where that meets numbers that are not finite: NaN stay, a sum that is not finite is
// formed again token after token, and an infinite element stays through decays whose product underflows if none of them is zero.
__device__ __forceinline__ float4 through_segment(const CcSeqWkv& a, const Segments& g, int s, size_t hi, size_t col, float4 x, const float4& add) {
    if (none_left(x)) return x;
    const size_t HD = (size_t)a.H * a.D, at = (size_t)s * g.len * HD;
    if (!finite(add)) {
#pragma unroll 8
        for (int t = 0; t < g.len; ++t) {
            const size_t row = at + (size_t)t * HD;
            const float* v = a.v + row + col;
            const float k = a.k[row + hi];
            x = fma4(g.w[row + hi], x, make_float4(k * v[0], k * v[1], k * v[2], k * v[3]));
        }
        return x;
    }
    const float p = g.P[(size_t)s * HD + hi];
    if (p != 0.f || finite(x)) return fma4(p, x, add);
    float least = 1.f;
#pragma unroll 16
    for (int t = 0; t < g.len; ++t) least = fminf(least, g.w[at + (size_t)t * HD + hi]);
    if (least == 0.f) return fma4(p, x, add);
    return make_float4(finite(x.x) ? add.x : x.x, finite(x.y) ? add.y : x.y, finite(x.z) ? add.z : x.z, finite(x.w) ? add.w : x.w);
}

// State at every segment's start, thread = four elements of a state row; the loads of sixteen segments are under way together.
__global__ void __launch_bounds__(128) wkv_segment_starts_kernel(const CcSeqWkv a, const Segments g) {
    const size_t n4 = (size_t)a.H * a.D * a.D / 4, e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n4) return;
    const size_t hi = e * 4 / a.D;      // head and row
    float4 x;
    if (((uintptr_t)a.state & 15) == 0) x = reinterpret_cast<const float4*>(a.state)[e];
    else x = make_float4(a.state[4 * e], a.state[4 * e + 1], a.state[4 * e + 2], a.state[4 * e + 3]);
    float4* X = reinterpret_cast<float4*>(g.X);
    X[e] = x;
    for (int s0 = 0; s0 + 1 < g.n; s0 += 16) {
        float4 add[16], from = x;
        float p[16];
#pragma unroll
        for (int q = 0; q < 16; ++q)
            if (s0 + q + 1 < g.n) {
                add[q] = X[(size_t)(s0 + q + 1) * n4 + e];
                p[q] = g.P[(size_t)(s0 + q) * a.H * a.D + hi];
            }
#pragma unroll
        for (int q = 0; q < 16; ++q)
            if (s0 + q + 1 < g.n) add[q] = x = fma4(p[q], x, add[q]);
        if (finite(x)) {      // what is not finite stays so: then all of them were
#pragma unroll
            for (int q = 0; q < 16; ++q)
                if (s0 + q + 1 < g.n) X[(size_t)(s0 + q + 1) * n4 + e] = add[q];
        } else {
            x = from;
#pragma unroll 1
            for (int s = s0; s < s0 + 16 && s + 1 < g.n; ++s) {
                float4* const at = X + (size_t)(s + 1) * n4 + e;
                *at = x = through_segment(a, g, s, hi, hi / a.D * a.D + e * 4 % a.D, x, *at);
            }
        }
    }
}

// A segment whose sums are not all finite, with the bonus meeting the value row by row: the outputs again, the state is the same.  Only
// the order of loading is simpler than below: one batch of tokens at a time.
template <int Dp>
__device__ __forceinline__ void wkv_segment_again(const CcSeqWkv& a, const Segments& g, float* sm) {
    constexpr int THREADS = Dp, P = Dp / 16, ROWS = TB * Dp;
    const int tid = threadIdx.x, s = blockIdx.x, h = blockIdx.y, j0 = blockIdx.z * TILE, p = tid % P, cg = tid / P, j = j0 + 4 * cg;
    const size_t HD = (size_t)a.H * a.D;
    const int first = s * g.len, count = min(g.len, a.T - first);
    const float* X = g.X + ((size_t)s * a.H + h) * a.D * a.D;
    float st[16][4];
    float* const us = sm + 3 * ROWS + TB * TILE;      // in the place of the second buffer
    for (int i = tid; i < Dp; i += THREADS) us[i] = i < a.D ? a.u[(size_t)h * a.D + i] : 0.f;
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const int i = 4 * P * (r / 4) + 4 * p + r % 4;
        const bool in = i < a.D;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (in && j < a.D) x = *reinterpret_cast<const float4*>(X + (size_t)i * a.D + j);
        st[r][0] = x.x; st[r][1] = x.y; st[r][2] = x.z; st[r][3] = x.w;
    }
    for (int t0 = 0; t0 < count; t0 += TB) {
        const int nt = min(TB, count - t0);
        const size_t at = (size_t)(first + t0) * HD + (size_t)h * a.D;
        for (int n = tid; n < TB * Dp; n += THREADS) {
            const int t = n / Dp, x = n % Dp;
            const bool in = t < nt && x < a.D;
            const size_t src = at + (in ? (size_t)t * HD + x : 0);
            sm[n] = in ? a.r[src] : 0.f;
            sm[ROWS + n] = in ? a.k[src] : 0.f;
            sm[2 * ROWS + n] = in ? g.w[src] : 0.f;
        }
        for (int n = tid; n < TB * TILE; n += THREADS) {
            const int t = n / TILE, x = n % TILE;
            sm[3 * ROWS + n] = t < nt && j0 + x < a.D ? a.v[at + (size_t)t * HD + j0 + x] : 0.f;
        }
        __syncthreads();
#pragma unroll 1
        for (int t = 0; t < nt; ++t) {
            const float* const row = sm + t * Dp;
            const float4 v = reinterpret_cast<const float4*>(sm + 3 * ROWS + t * TILE)[cg];
            float o[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const int i = 4 * P * (r / 4) + 4 * p + r % 4;
                const float rv = row[i], k = row[ROWS + i], w = row[2 * ROWS + i], kv[4] = {k * v.x, k * v.y, k * v.z, k * v.w};
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    o[x] = fmaf(rv, fmaf(us[i], kv[x], st[r][x]), o[x]);
                    st[r][x] = fmaf(w, st[r][x], kv[x]);
                }
            }
#pragma unroll
            for (int x = 0; x < 4; ++x) {
#pragma unroll
                for (int d = 1; d < P; d <<= 1) o[x] += __shfl_xor_sync(0xffffffffu, o[x], d);
                if (p == x && j < a.D) a.o[at + (size_t)t * HD + j + x] = o[x];
            }
        }
        __syncthreads();
    }
}

// The recurrence inside a segment, 64 columns of a head.  Thread = 16 rows x 4 columns: lane % P holds rows 4 P q + 4 p .. + 3 of
// P = Dp / 16 row groups, the rest of the thread number the columns.  A token's operands are 13 16-byte reads of shared memory for
// 124 pairs of fp32 operations; the row groups of a column meet by shuffles, so that tokens need no barrier.
// (168 registers, six CTAs an SM of 64 threads; asked for that many CTAs the compiler schedules the walk 3 us slower.)
template <int Dp, bool VEC>
__global__ void __launch_bounds__(Dp) wkv_segment_scan_kernel(const CcSeqWkv a, const Segments g) {
    extern __shared__ float4 smw4[];
    float* const sm = reinterpret_cast<float*>(smw4);
    constexpr int THREADS = Dp, P = Dp / 16, ROWS = TB * Dp, BUF = 3 * ROWS + TB * TILE;
    const int tid = threadIdx.x, s = blockIdx.x, h = blockIdx.y, j0 = blockIdx.z * TILE;
    const int p = tid % P, cg = tid / P, j = j0 + 4 * cg;
    const size_t HD = (size_t)a.H * a.D;
    const int first = s * g.len, count = min(g.len, a.T - first);
    auto fetch = [&](int t0, float* buf) {      // [r | k | w | v] rows of TB tokens
        const int nt = min(TB, count - t0);
        const size_t at = (size_t)(first + t0) * HD + (size_t)h * a.D;
        {
            const int x = 4 * (tid % (Dp / 4));
#pragma unroll
            for (int t = tid / (Dp / 4); t < TB; t += THREADS / (Dp / 4)) {
                const bool in = t < nt && x < a.D;
                const size_t src = at + (in ? (size_t)t * HD + x : 0);
                float* const d = buf + t * Dp + x;
                stage4<VEC>(d, a.r + src, in);
                stage4<VEC>(d + ROWS, a.k + src, in);
                stage4<VEC>(d + 2 * ROWS, g.w + src, in);
            }
        }
        const int x = 4 * (tid % (TILE / 4));
#pragma unroll
        for (int t = tid / (TILE / 4); t < TB; t += THREADS / (TILE / 4)) {
            const bool in = t < nt && j0 + x < a.D;
            stage4<VEC>(buf + 3 * ROWS + t * TILE + x, a.v + at + (in ? (size_t)t * HD + j0 + x : 0), in);
        }
        cp_async_commit();
    };
    fetch(0, sm);
    f32x2 st[8][4], u2[8];
    const float* X = g.X + ((size_t)s * a.H + h) * a.D * a.D;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int i = 4 * P * (r / 2) + 4 * p + 2 * (r % 2);
        const bool in = i < a.D;
        u2[r] = in ? pair(a.u[(size_t)h * a.D + i], a.u[(size_t)h * a.D + i + 1]) : 0ull;
        float4 lo = make_float4(0.f, 0.f, 0.f, 0.f), hi = lo;
        if (in && j < a.D) {
            lo = *reinterpret_cast<const float4*>(X + (size_t)i * a.D + j);
            hi = *reinterpret_cast<const float4*>(X + (size_t)(i + 1) * a.D + j);
        }
        st[r][0] = pair(lo.x, hi.x);
        st[r][1] = pair(lo.y, hi.y);
        st[r][2] = pair(lo.z, hi.z);
        st[r][3] = pair(lo.w, hi.w);
    }
    const bool up2 = p & 2, up1 = p & 1;
    float* out = a.o + (size_t)first * HD + (size_t)h * a.D + j + (up2 ? 2 : 0) + (up1 ? 1 : 0);
    const bool writes = p < 4 && j < a.D;
    float none = 0.f;      // NaN from the first sum on that is not finite
    int cur = 0;
    for (int t0 = 0; t0 < count; t0 += TB, cur ^= 1) {
        const float* const buf = sm + cur * BUF;
        const int nt = min(TB, count - t0);
        if (t0 + TB < count) {
            fetch(t0 + TB, sm + (cur ^ 1) * BUF);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
#pragma unroll 2
        for (int t = 0; t < nt; ++t, out += HD) {
            const float4* const r4 = reinterpret_cast<const float4*>(buf + t * Dp) + p;
            const float4 vv = reinterpret_cast<const float4*>(buf + 3 * ROWS + t * TILE)[cg];
            const f32x2 v2[4] = {pair(vv.x, vv.x), pair(vv.y, vv.y), pair(vv.z, vv.z), pair(vv.w, vv.w)};
            f32x2 acc[2][4], bonus[2];      // two chains each: half the roundings in a row
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 rv = r4[P * q], kv = r4[P * q + ROWS / 4], wv = r4[P * q + 2 * (ROWS / 4)];
                const f32x2 r2[2] = {pair(rv.x, rv.y), pair(rv.z, rv.w)}, k2[2] = {pair(kv.x, kv.y), pair(kv.z, kv.w)}, w2[2] = {pair(wv.x, wv.y), pair(wv.z, wv.w)};
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int r = 2 * q + e;
                    const f32x2 uk = mul2(u2[r], k2[e]);
                    bonus[e] = q == 0 ? mul2(r2[e], uk) : fma2(r2[e], uk, bonus[e]);
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        acc[e][x] = q == 0 ? mul2(r2[e], st[r][x]) : fma2(r2[e], st[r][x], acc[e][x]);
                        st[r][x] = fma2(w2[e], st[r][x], mul2(k2[e], v2[x]));
                    }
                }
            }
            float o[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                float lo, hi;
                unpair(add2(fma2(bonus[0], v2[x], acc[0][x]), fma2(bonus[1], v2[x], acc[1][x])), lo, hi);
                o[x] = lo + hi;
            }
            // columns meet over the row groups: half of the values is sent at each of two steps, a lane ends with one column
            float a0 = (up2 ? o[2] : o[0]) + __shfl_xor_sync(0xffffffffu, up2 ? o[0] : o[2], 2);
            const float a1 = (up2 ? o[3] : o[1]) + __shfl_xor_sync(0xffffffffu, up2 ? o[1] : o[3], 2);
            a0 = (up1 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, up1 ? a0 : a1, 1);
            if (P == 8) a0 += __shfl_xor_sync(0xffffffffu, a0, 4);
            if (writes) *out = a0;
            none = fmaf(0.f, a0, none);
        }
        __syncthreads();
    }
    float* const S = a.state + (size_t)h * a.D * a.D;
#pragma unroll
    for (int r = 0; r < 8 && s + 1 == g.n; ++r) {
        const int i = 4 * P * (r / 2) + 4 * p + 2 * (r % 2);
        if (i >= a.D || j >= a.D) continue;
        float lo[4], hi[4];
#pragma unroll
        for (int x = 0; x < 4; ++x) unpair(st[r][x], lo[x], hi[x]);
        float* const row = S + (size_t)i * a.D + j;
        if (((uintptr_t)S & 15) == 0) {      // D is a multiple of 4
            *reinterpret_cast<float4*>(row) = make_float4(lo[0], lo[1], lo[2], lo[3]);
            *reinterpret_cast<float4*>(row + a.D) = make_float4(hi[0], hi[1], hi[2], hi[3]);
        } else {
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                row[x] = lo[x];
                row[a.D + x] = hi[x];
            }
        }
    }
    if (__syncthreads_or(none != none)) wkv_segment_again<Dp>(a, g, sm);
}

// Segments: as many as give an SM six CTAs (what the scan's registers allow) over heads and column tiles, of at least 32 tokens.  Eight, so that
// a second wave evens out the first, while segments keep 100 tokens: each has a start of its own (a state to load, a batch to wait for),
// which shorter ones repeat more often than an even end is worth.  Time with six over time with eight, back to back in a graph, by the length
// that eight leave: up to 90 tokens 0.92 to 1.13, and as often below one as above (3000 tokens of 32 heads of 64 0.97, 512 of 40 of 100 0.92); at 92 to
// 99 0.98 to 1.06; at 100 1.00 to 1.12; at 110 (4096 of 32 of 64) 1.06, at 120 1.005 to 1.14, at 220 1.01 to 1.15 (9 to 128 heads of 16 to 128).
// Where six give a single segment or two and eight one more, 1.15 to 1.8 (256 to 1024 tokens of 460 to 592 heads of 64, 222 to 296 of 100 to
// 128).  Nine and twelve are slower than eight, and seven than six for most numbers of heads.
// The three launches follow one another in full: started under each other (programmatic launch) 256 tokens of 16 heads take 32 us
// instead of 20.
constexpr int MIN_LEN = 32, LONG_LEN = 100;
static Segments plan(int T, int H, int D) {
    const long long per = (long long)H * ((D + TILE - 1) / TILE);
    long long most = 8 * 148 / per;
    if (T < LONG_LEN * most) most = 6 * 148 / per;
    if (most < 1) most = 1;
    int len = (int)((T + most - 1) / most);
    if (len < MIN_LEN) len = MIN_LEN;
    return {nullptr, nullptr, nullptr, len, (T + len - 1) / len};
}
// Whether segments side by side are the faster way.  They work on whole tiles of 64 rows and columns, the other way on 8 x 16 or 32
// columns, so heads that leave much of a tile empty gain only while the GPU is not full.  Measured, this / token after token in us:
//   filled tiles (56 to 64, 100 to 128 wide), any number of heads: 256 tokens of 64 30 / 36 (64 heads), 131 / 144 (300), 141 / 177
//   (444), of 56 96 / 124 (296); 1024 of 60 482 / 578 (370), of 100 884 / 1189 (222); 256 of 104 62 / 60 (40), 300 70 / 69, 512 97 / 112;
//   others up to 74 tiles of the state: 256 tokens of 16 29 / 45 (74 heads), 37 / 45 (96), 48 / 45 (128); of 32 29 / 32, 37 / 32, 48 / 33;
//   of 48 30 / 42 (74), 61 / 55 (160); of 72 30 / 39 (18), 45 / 39 (28), 66 / 47 (48); of 96 31 / 38 (18), 39 / 38 (20), 68 / 45 (48).
static bool pays(int T, int H, int D) {
    const int tiles = (D + TILE - 1) / TILE;
    if (D <= TILE ? D >= 56 : D >= 100) return D <= TILE || D == 2 * TILE || T >= 384;
    return (long long)H * tiles * tiles <= 74;
}
static uint64_t workspace_floats(const Segments& g, int T, int H, int D) {
    return ((uint64_t)T * H * D + 3) / 4 * 4 + (uint64_t)g.n * H * D * D + (uint64_t)g.n * H * D;
}

template <int Dp, bool VEC>
static int launch_scan(const CcSeqWkv* a, const Segments& g, cudaStream_t st) {
    const size_t smem = 2 * sizeof(float) * (3 * TB * Dp + TB * TILE);
    static SmemLimit limit;
    if (limit.allow(wkv_segment_scan_kernel<Dp, VEC>, smem) != cudaSuccess) return cuda_check("wkv_segments: shared memory");
    wkv_segment_scan_kernel<Dp, VEC><<<dim3(g.n, a->H, (a->D + TILE - 1) / TILE), Dp, smem, st>>>(*a, g);
    return cuda_check("wkv_segment_scan_kernel");
}

}  // namespace ccw

using namespace ccw;

extern "C" {

uint64_t cc_seq_wkv_segments_workspace(int32_t T, int32_t H, int32_t D) {
    if (T < 1 || H < 1 || D < 1 || D > 128 || D % 4 != 0) return 0;
    const Segments g = plan(T, H, D);
    return g.n < 2 || !pays(T, H, D) ? 0 : sizeof(float) * workspace_floats(g, T, H, D);
}

int cc_seq_wkv_segments(const CcSeqWkv* a, void* workspace, uint64_t workspace_bytes, void* stream) {
    if (!a || !a->r || !a->k || !a->v || !a->wraw || !a->w0 || !a->u || !a->state || !a->o || a->decayed)
        return fail(CC_SEQ_ERR_INVALID_ARG, "wkv_segments: bad argument");
    const uint64_t need = cc_seq_wkv_segments_workspace(a->T, a->H, a->D);
    if (need == 0) return fail(CC_SEQ_ERR_UNSUPPORTED_SHAPE, "wkv_segments: heads of multiples of 4 up to 128, at least two segments");
    if (!workspace || workspace_bytes < need) return fail(CC_SEQ_ERR_INVALID_ARG, "wkv_segments: workspace too small");
    if ((uintptr_t)workspace & 15) return fail(CC_SEQ_ERR_INVALID_ARG, "wkv_segments: the workspace starts on a 16-byte boundary");
    cudaStream_t st = (cudaStream_t)stream;
    Segments g = plan(a->T, a->H, a->D);
    g.w = (float*)workspace;
    g.X = g.w + ((uint64_t)a->T * a->H * a->D + 3) / 4 * 4;
    g.P = g.X + (uint64_t)g.n * a->H * a->D * a->D;
    const int tiles = (a->D + TILE - 1) / TILE;
    const bool vec = (((uintptr_t)a->r | (uintptr_t)a->k | (uintptr_t)a->v | (uintptr_t)a->wraw) & 15) == 0;
    const dim3 grid(g.n, a->H, tiles * tiles);
    if (vec) wkv_segment_state_kernel<true><<<grid, STATE_THREADS, 0, st>>>(*a, g);
    else wkv_segment_state_kernel<false><<<grid, STATE_THREADS, 0, st>>>(*a, g);
    int rc = cuda_check("wkv_segment_state_kernel");
    if (rc) return rc;
    const uint64_t n4 = (uint64_t)a->H * a->D * a->D / 4;
    wkv_segment_starts_kernel<<<(unsigned)((n4 + 127) / 128), 128, 0, st>>>(*a, g);
    rc = cuda_check("wkv_segment_starts_kernel");
    if (rc) return rc;
    if (vec) return a->D <= 64 ? launch_scan<64, true>(a, g, st) : launch_scan<128, true>(a, g, st);
    return a->D <= 64 ? launch_scan<64, false>(a, g, st) : launch_scan<128, false>(a, g, st);
}

}  // extern "C"
