// seq_kernels.cu -- position-addressed sequence kernels behind include/cc_b200_seq.h (libcc_b200_seq.so).
//
// Arithmetic rule of this file: positions, angles, norms, attention scores, softmax weights, the weighted value sum
// and the residual stream are fp32 whatever the storage type of activations, weights and cache rows (fp32 or bf16);
// expf / logf / sinf / cosf / sqrtf are the accurate versions (no fast-math).  Results of the attention kernels depend on
// the key positions a query sees, never on which launch, chunk or slot brought a key: keys are addressed by
// position (slot = position mod capacity, checked against the slot's recorded position).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <string.h>

#include "../../../include/cc_b200_seq.h"
#include "launch.cuh"
#include "tensor_map.cuh"

namespace ccs {

static thread_local char g_err[512] = "";
// fail() and cuda_check() are shared with the other files of this library (declared there by hand)
int fail(int code, const char* msg) {
    strncpy(g_err, msg, sizeof(g_err) - 1);
    g_err[sizeof(g_err) - 1] = 0;
    return code;
}
int cuda_check(const char* where) {
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) return CC_SEQ_OK;
    snprintf(g_err, sizeof(g_err), "%s: %s", where, cudaGetErrorString(e));
    return CC_SEQ_ERR_CUDA;
}

__device__ __forceinline__ float ldf(const float* p, size_t i) { return p[i]; }
__device__ __forceinline__ float ldf(const __nv_bfloat16* p, size_t i) { return __bfloat162float(p[i]); }
__device__ __forceinline__ void stf(float* p, size_t i, float v) { p[i] = v; }
__device__ __forceinline__ void stf(__nv_bfloat16* p, size_t i, float v) { p[i] = __float2bfloat16_rn(v); }

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// ------------------------------------------------------------------------------------------------ embedding
template <typename WT, typename AT>
__global__ void embed_kernel(const int32_t* __restrict__ tokens, const int32_t* __restrict__ input_pos,
                             int32_t* prev_token, const WT* __restrict__ embed, const WT* __restrict__ bigram,
                             const float* __restrict__ inv_freq, float* __restrict__ x, AT* __restrict__ x_act, int T,
                             int E, float scale, int buckets, int mul_prev, int mul_cur) {
    const int t = blockIdx.x;
    const int p = input_pos[0] + t;
    const int tok = tokens[t];
    long long row = -1;
    if (bigram != nullptr) {
        if (p == 0) {
            row = buckets;
        } else {
            const long long prev = t > 0 ? tokens[t - 1] : prev_token[0];
            row = (prev * (long long)mul_prev + (long long)tok * (long long)mul_cur) % (long long)buckets;
            if (row < 0) row += buckets;
        }
    }
    const float pf = (float)p;
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        float v = ldf(embed, (size_t)tok * E + e) * scale;
        if (row >= 0) v += ldf(bigram, (size_t)row * E + e);
        const float ang = pf * inv_freq[e >> 1];
        v += (e & 1) ? cosf(ang) : sinf(ang);
        x[(size_t)t * E + e] = v;
        if (x_act != nullptr) stf(x_act, (size_t)t * E + e, v);
    }
    if (t == 0) {  // every thread of this block has read the old state above
        __syncthreads();
        if (threadIdx.x == 0) prev_token[0] = tokens[T - 1];
    }
}

// ------------------------------------------------------------------------------------------------ q/k/v preparation
template <typename IT, typename OT>
__global__ void qkv_prepare_kernel(const IT* __restrict__ qkv, const float* __restrict__ bias,
                                   const int32_t* __restrict__ input_pos, const float* __restrict__ mix_lambda,
                                   const OT* __restrict__ v_first, float* __restrict__ q_out, OT* __restrict__ k_out,
                                   OT* __restrict__ v_out, int T, int H, int G, int Dk, int Dv, float eps, int unit_norm,
                                   float gain_coef, int gain_every) {
    const int t = blockIdx.x;
    const int N = (H + G) * Dk + G * Dv;
    const IT* row = qkv + (size_t)t * N;
    const int p = input_pos[0] + t;
    float gain = 1.0f;
    if (gain_every > 0) gain = 1.0f + gain_coef * logf((float)((p + 1) / gain_every + 1));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
    for (int hh = warp; hh < H + G; hh += nwarp) {
        const int off = hh * Dk;
        float ss = 0.f;
        for (int d = lane; d < Dk; d += 32) {
            float v = ldf(row, off + d);
            if (bias != nullptr) v += bias[off + d];
            ss += v * v;
        }
        ss = warp_sum(ss);
        const float r = unit_norm ? 1.0f / sqrtf(ss / (float)Dk + eps) : 1.0f;
        for (int d = lane; d < Dk; d += 32) {
            float v = ldf(row, off + d);
            if (bias != nullptr) v += bias[off + d];
            if (hh < H) q_out[((size_t)t * H + hh) * Dk + d] = v * r * gain;
            else stf(k_out, ((size_t)t * G + (hh - H)) * Dk + d, v * r);
        }
    }
    const int voff = (H + G) * Dk, NV = G * Dv;
    const float lam = v_first != nullptr ? mix_lambda[0] : 0.f;
    for (int i = threadIdx.x; i < NV; i += blockDim.x) {
        float v = ldf(row, voff + i);
        if (bias != nullptr) v += bias[voff + i];
        if (v_first != nullptr) v = (1.0f - lam) * v + lam * ldf(v_first, (size_t)t * NV + i);
        stf(v_out, (size_t)t * NV + i, v);
    }
}

// ------------------------------------------------------------------------------------------------ chunk attention
constexpr int BQ = 64, BK = 32, ATT_THREADS = 256;

// Slot of position j: the first keep_first positions own the first slots for good, the others share a ring over the
// rest of the cache (keep_first == 0: slot = j mod L).
__device__ __forceinline__ int slot_of(const CcSeqAttn& a, int j) {
    return j < a.keep_first ? j : a.keep_first + (j - a.keep_first) % (a.L - a.keep_first);
}

__device__ __forceinline__ int key_source(const CcSeqAttn& a, int j, int p0) {
    // >= 0: cache slot, -1: not a key, <= -2: row -(s + 2) of the chunk
    if (j >= p0) return -(j - p0) - 2;
    const int slot = slot_of(a, j);
    return a.pos[slot] == j ? slot : -1;
}

// What the design does to a scaled score before the softmax: a tanh soft cap, then a penalty that grows with the
// logarithm of the distance between query i and key j, with two numbers per query head.
__device__ __forceinline__ float shape_score(const CcSeqAttn& a, float s, int h, int dist) {
    if (a.softcap > 0.f) s = a.softcap * tanhf(s / a.softcap);
    if (a.dist_a != nullptr) s -= a.dist_a[h] * log1pf(a.dist_b[h] * (float)dist);
    return s;
}

// Stages `rows` rows of `width` elements (global, row r at src(r), or zeros when src(r) == nullptr) into fp32 shared
// memory rows of `stride` floats (a multiple of 4, dst 16-byte aligned).  16-byte loads and stores when the rows allow
// it, element loads otherwise.
template <typename CT, typename SrcFn>
__device__ __forceinline__ void stage_rows(float* dst, int stride, int rows, int width, SrcFn src, int tid, int nthreads) {
    constexpr int VEC = 16 / (int)sizeof(CT);
    if (width % VEC == 0) {
        constexpr int U = 4;   // loads in flight per thread
        const int per_row = width / VEC, total = rows * per_row;
        for (int base = tid; base < total; base += nthreads * U) {
            uint4 u[U];
            int off[U];
#pragma unroll
            for (int e = 0; e < U; ++e) {
                const int idx = base + e * nthreads;
                off[e] = -1;
                u[e] = make_uint4(0u, 0u, 0u, 0u);
                if (idx < total) {
                    const int r = idx / per_row, c = (idx - r * per_row) * VEC;
                    off[e] = r * stride + c;
                    const CT* p = src(r);
                    if (p != nullptr) u[e] = __ldg(reinterpret_cast<const uint4*>(p + c));
                }
            }
#pragma unroll
            for (int e = 0; e < U; ++e) {
                if (off[e] < 0) continue;
                const CT* e8 = reinterpret_cast<const CT*>(&u[e]);
                float4* d4 = reinterpret_cast<float4*>(dst + off[e]);   // stride and column are multiples of 4 floats
#pragma unroll
                for (int i = 0; i < VEC / 4; ++i)
                    d4[i] = make_float4(ldf(e8, 4 * i), ldf(e8, 4 * i + 1), ldf(e8, 4 * i + 2), ldf(e8, 4 * i + 3));
            }
        }
    } else {
        for (int idx = tid; idx < rows * width; idx += nthreads) {
            const int r = idx / width, c = idx - r * width;
            const CT* p = src(r);
            dst[r * stride + c] = p == nullptr ? 0.f : ldf(p, c);
        }
    }
}


// Row stride (floats) of a shared-memory tile read with 16-byte loads by lanes that hold different rows: a multiple
// of 4 whose quarter is odd, so that eight rows fall into eight different 16-byte bank groups.
__host__ __device__ inline int vec_stride(int width) {
    const int w4 = (width + 3) / 4;
    return 4 * (w4 | 1);
}

// CTA = 64 consecutive queries of one query head; key tiles of 32 positions.  Thread (ty, tx) of the 16 x 16 grid owns
// score rows 4 ty .. 4 ty + 3 x columns tx, tx + 16 and output rows 4 ty .. x value columns 64 c + 4 tx .. 4 tx + 3.
// All shared-memory operands are read with 16-byte loads: q, k along the head dimension, P along the keys, V along
// the value columns; 32 (scores) and 64 DV4 (values) FMAs per 6 and 4 + 4 DV4 loads.
template <typename CT, typename YT, int DV4>
__global__ void __launch_bounds__(ATT_THREADS) attn_chunk_kernel(const CcSeqAttn a) {
    extern __shared__ float4 sm4[];
    float* sm = reinterpret_cast<float*>(sm4);
    const int Dk = a.Dk, Dv = a.Dv, Dkp = vec_stride(Dk), Dk4 = (Dk + 3) / 4;
    constexpr int DVW = 64 * DV4, SP = BK + 4;
    float* Qs = sm;
    float* Ks = Qs + BQ * Dkp;
    float* Vs = Ks + BK * Dkp;
    float* Ss = Vs + BK * DVW;
    int* ksrc = (int*)(Ss + BQ * SP);
    int* kpos = ksrc + BK;

    const int qb = blockIdx.x, h = blockIdx.y, g = h / (a.H / a.G);
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int p0 = a.input_pos[0];
    const int i0 = qb * BQ;
    const int nq = min(BQ, a.T - i0);
    const CT* kc = (const CT*)a.k_cache;
    const CT* vc = (const CT*)a.v_cache;
    const CT* kn = (const CT*)a.k_new;
    const CT* vn = (const CT*)a.v_new;

    // padding columns are zero for the whole kernel (the tile loads below never touch them)
    for (int idx = tid; idx < (BQ + BK) * (Dkp - Dk); idx += ATT_THREADS) {
        const int r = idx / (Dkp - Dk), c = Dk + idx - r * (Dkp - Dk);
        Qs[r * Dkp + c] = 0.f;   // Ks follows Qs with the same stride
    }
    for (int idx = tid; idx < BK * (DVW - Dv); idx += ATT_THREADS) {
        const int r = idx / (DVW - Dv), c = Dv + idx - r * (DVW - Dv);
        Vs[r * DVW + c] = 0.f;
    }
    stage_rows<float>(Qs, Dkp, BQ, Dk, [&](int r) -> const float* {
        return r < nq ? a.q + ((size_t)(i0 + r) * a.H + h) * Dk : nullptr;
    }, tid, ATT_THREADS);
    const int j_hi = p0 + i0 + nq - 1;
    const int j_lo = a.block > 0 ? ((p0 + i0) / a.block) * a.block : (a.window > 0 ? max(0, p0 + i0 - a.window + 1) : 0);

    float m[4], l[4], O[4][4 * DV4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        if (a.sink_mode == CC_SINK_LEARNED) { m[r] = a.sink[h]; l[r] = 1.f; }
        else if (a.sink_mode == CC_SINK_ZERO) { m[r] = 0.f; l[r] = 1.f; }
        else { m[r] = -INFINITY; l[r] = 0.f; }
#pragma unroll
        for (int c = 0; c < 4 * DV4; ++c) O[r][c] = 0.f;
    }

    // the keys of this CTA in order: the kept first positions that lie below the window, then j_lo .. j_hi
    const int kx = a.window > 0 ? min(a.keep_first, j_lo) : 0;
    const int n_keys = kx + (j_hi - j_lo + 1);
    for (int ut = 0; ut < n_keys; ut += BK) {
        __syncthreads();  // the previous tile is consumed
        const int nk = min(BK, n_keys - ut);
        if (tid < BK) {
            const int u = ut + tid, j = u < kx ? u : j_lo + (u - kx);
            kpos[tid] = j;
            ksrc[tid] = tid < nk ? key_source(a, j, p0) : -1;
        }
        __syncthreads();
        stage_rows<CT>(Ks, Dkp, BK, Dk, [&](int r) -> const CT* {
            const int s = ksrc[r];
            return s >= 0 ? kc + ((size_t)g * a.L + s) * Dk : (s <= -2 ? kn + ((size_t)(-s - 2) * a.G + g) * Dk : nullptr);
        }, tid, ATT_THREADS);
        stage_rows<CT>(Vs, DVW, BK, Dv, [&](int r) -> const CT* {
            const int s = ksrc[r];
            return s >= 0 ? vc + ((size_t)g * a.L + s) * Dv : (s <= -2 ? vn + ((size_t)(-s - 2) * a.G + g) * Dv : nullptr);
        }, tid, ATT_THREADS);
        __syncthreads();

        float s[4][2];
#pragma unroll
        for (int r = 0; r < 4; ++r) s[r][0] = s[r][1] = 0.f;
        const float4* q4 = reinterpret_cast<const float4*>(Qs + (ty * 4) * Dkp);
        const float4* k4 = reinterpret_cast<const float4*>(Ks + tx * Dkp);
        const int rs4 = Dkp / 4;
#pragma unroll 2
        for (int d = 0; d < Dk4; ++d) {
            float4 qv[4], kv[2];
#pragma unroll
            for (int r = 0; r < 4; ++r) qv[r] = q4[r * rs4 + d];
            kv[0] = k4[d];
            kv[1] = k4[16 * rs4 + d];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    s[r][c] = fmaf(qv[r].x, kv[c].x, s[r][c]);
                    s[r][c] = fmaf(qv[r].y, kv[c].y, s[r][c]);
                    s[r][c] = fmaf(qv[r].z, kv[c].z, s[r][c]);
                    s[r][c] = fmaf(qv[r].w, kv[c].w, s[r][c]);
                }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int qi = ty * 4 + r;
            const int i = p0 + i0 + qi;
            float mx = -INFINITY;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int col = tx + 16 * c;
                const int j = kpos[col];
                const bool ok = qi < nq && col < nk && ksrc[col] != -1 && j <= i &&
                                (a.window == 0 || i - j < a.window || j < a.keep_first) &&
                                (a.block == 0 || j >= (i / a.block) * a.block);
                s[r][c] = ok ? shape_score(a, s[r][c] * a.scale, h, i - j) : -INFINITY;
                mx = fmaxf(mx, s[r][c]);
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float m_new = fmaxf(m[r], mx);
            const float corr = (m[r] == -INFINITY) ? 0.f : expf(m[r] - m_new);
            float rsum = 0.f;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const float pr = (s[r][c] == -INFINITY) ? 0.f : expf(s[r][c] - m_new);
                rsum += pr;
                Ss[qi * SP + tx + 16 * c] = pr;
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) rsum += __shfl_xor_sync(0xffffffffu, rsum, o);
            l[r] = l[r] * corr + rsum;
            m[r] = m_new;
#pragma unroll
            for (int c = 0; c < 4 * DV4; ++c) O[r][c] *= corr;
        }
        __syncwarp();
        const float4* p4 = reinterpret_cast<const float4*>(Ss + (ty * 4) * SP);
        const float4* v4 = reinterpret_cast<const float4*>(Vs) + tx;
#pragma unroll 2
        for (int kq = 0; kq < BK / 4; ++kq) {
            float4 pv[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) pv[r] = p4[r * (SP / 4) + kq];
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
#pragma unroll
                for (int c = 0; c < DV4; ++c) {
                    const float4 vv = v4[(kq * 4 + kk) * (DVW / 4) + 16 * c];
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const float pk = kk == 0 ? pv[r].x : kk == 1 ? pv[r].y : kk == 2 ? pv[r].z : pv[r].w;
                        O[r][4 * c + 0] = fmaf(pk, vv.x, O[r][4 * c + 0]);
                        O[r][4 * c + 1] = fmaf(pk, vv.y, O[r][4 * c + 1]);
                        O[r][4 * c + 2] = fmaf(pk, vv.z, O[r][4 * c + 2]);
                        O[r][4 * c + 3] = fmaf(pk, vv.w, O[r][4 * c + 3]);
                    }
                }
            }
        }
    }
    YT* y = (YT*)a.y;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int qi = ty * 4 + r;
        if (qi >= nq) continue;
        const float inv = l[r] > 0.f ? 1.0f / l[r] : 0.f;
#pragma unroll
        for (int c = 0; c < 4 * DV4; ++c) {
            const int col = 64 * (c / 4) + 4 * tx + (c & 3);
            if (col < Dv) stf(y, ((size_t)(i0 + qi) * a.H + h) * Dv + col, O[r][c] * inv);
        }
    }
}

// ------------------------------------------------------------------------------------------------ decode attention
constexpr int KS = 128;           // keys per tile of the one-token kernel
constexpr int DEC_THREADS = 128;  // one thread per key
#ifndef CC_DEC_MAX_SPLITS
#define CC_DEC_MAX_SPLITS 64
#endif
constexpr int DEC_MAX_SPLITS = CC_DEC_MAX_SPLITS;  // runs of tiles per key/value head: bounds the partials the last CTA combines

__host__ __device__ inline int dec_k_stride(int Dk) {
    const int d4 = (Dk + 3) & ~3;
    return d4 + ((8 - (d4 & 31)) & 31);
}

__host__ __device__ inline int decode_max_splits(int L, int window) {
    const long long maxkeys = window > 0 ? (window < L + 1 ? window : L + 1) : (long long)L + 1;
    const long long tiles = (maxkeys + KS - 1) / KS;
    return (int)(tiles < DEC_MAX_SPLITS ? tiles : DEC_MAX_SPLITS);
}

// the most keys a query can see besides the limit of the cache: its window, or its block
__host__ __device__ inline int attn_reach(const CcSeqAttn& a) {
    return a.block > 0 ? a.block : (a.window > 0 ? a.window + a.keep_first : 0);
}

template <typename CT>
__device__ __forceinline__ void append_row(const CcSeqAttn& a, int g, int t, int p, int tid, int nthreads) {
    const int slot = slot_of(a, p);
    CT* kc = (CT*)a.k_cache;
    CT* vc = (CT*)a.v_cache;
    const CT* kn = (const CT*)a.k_new;
    const CT* vn = (const CT*)a.v_new;
    for (int d = tid; d < a.Dk; d += nthreads) kc[((size_t)g * a.L + slot) * a.Dk + d] = kn[((size_t)t * a.G + g) * a.Dk + d];
    for (int d = tid; d < a.Dv; d += nthreads) vc[((size_t)g * a.L + slot) * a.Dv + d] = vn[((size_t)t * a.G + g) * a.Dv + d];
    if (tid == 0) {
        if (a.mask != nullptr) a.mask[(size_t)g * a.L + slot] = 1;
        if (g == 0) {
            const int old = a.pos[slot];
            a.pos[slot] = p;
            if (old < 0 && a.cache_cts != nullptr) atomicAdd(a.cache_cts, 1);
        }
    }
}

// One CTA = a run of KS-key tiles of one key/value head, all R = H / G query heads of the group.  Per tile: one thread
// per key reads its K row straight from global memory with 16-byte loads (all in flight at once; consecutive keys are
// consecutive rows, so a warp's loads cover whole lines) and dots it with the R query rows held in shared memory
// (broadcast float4 reads); online softmax per query head; then one thread per value column walks the tile's V rows
// (coalesced across the columns).  A head's keys are cut into at most DEC_MAX_SPLITS runs; partial (max, sum, weighted
// values) go to the workspace; the last CTA of the head to arrive combines them in split order and, when asked,
// appends the new row.
template <typename CT, typename YT, int RMAX>
__global__ void __launch_bounds__(DEC_THREADS) attn_decode_kernel(const CcSeqAttn a) {
    extern __shared__ float4 smd4[];
    float* sm = reinterpret_cast<float*>(smd4);
    constexpr int VEC = 16 / (int)sizeof(CT);
    const int R = a.H / a.G, Dk = a.Dk, Dv = a.Dv;
    const int Dq = (Dk + 7) & ~7;   // q rows zero-padded to whole vectors
    float* qs = sm;               // [R, Dq]
    float* Ps = qs + R * Dq;      // [R, KS]
    int* ksrc = (int*)(Ps + R * KS);
    __shared__ int s_last;
    __shared__ float s_M[16], s_L[16], s_corr[16];

    const int sp = blockIdx.x, g = blockIdx.y, tid = threadIdx.x;
    const int p = a.input_pos[0];
    const int j_lo = a.block > 0 ? (p / a.block) * a.block : (a.window > 0 ? max(0, p - a.window + 1) : 0);
    const int kx = a.window > 0 ? min(a.keep_first, j_lo) : 0;   // kept first positions below the window
    const int n = kx + (p - j_lo + 1);
    const int n_tiles = (n + KS - 1) / KS;
    const int tiles_per = (n_tiles + DEC_MAX_SPLITS - 1) / DEC_MAX_SPLITS;
    const int nsplit = (n_tiles + tiles_per - 1) / tiles_per;
    if (sp >= nsplit) return;
    const int NS = decode_max_splits(a.L, attn_reach(a));
    int* counters = (int*)a.workspace;
    float* part_m = (float*)(counters + ((a.G + 3) & ~3));
    float* part_l = part_m + (size_t)a.G * NS * R;
    float* part_o = part_l + (size_t)a.G * NS * R;

    const CT* kc = (const CT*)a.k_cache;
    const CT* vc = (const CT*)a.v_cache;
    const CT* kn = (const CT*)a.k_new;
    const CT* vn = (const CT*)a.v_new;
    for (int i = tid; i < R * Dq; i += DEC_THREADS) {
        const int r = i / Dq, d = i - r * Dq;
        qs[i] = d < Dk ? a.q[((size_t)g * R + r) * Dk + d] : 0.f;
    }
    if (tid < 16) { s_M[tid] = -INFINITY; s_L[tid] = 0.f; }
    const int warp = tid >> 5, lane = tid & 31;
    float oacc[2][RMAX];   // value columns tid and tid + DEC_THREADS
#pragma unroll
    for (int r = 0; r < RMAX; ++r) oacc[0][r] = oacc[1][r] = 0.f;
    const bool vec_rows = (Dk % VEC) == 0;
    // value phase with 16-byte loads when the rows allow it and R x VEC accumulators fit in registers
    constexpr int VR = RMAX * VEC <= 64 ? RMAX : 1;
    const int ncg = Dv / VEC;
    const bool vec_values = RMAX * VEC <= 64 && Dv % VEC == 0 && ncg <= DEC_THREADS;
    const int nkg = vec_values ? DEC_THREADS / ncg : 1;
    const int kg = vec_values ? tid / ncg : 0, cg = vec_values ? tid - kg * ncg : 0;
    float vacc[VR][VEC];
#pragma unroll
    for (int r = 0; r < VR; ++r)
#pragma unroll
        for (int x = 0; x < VEC; ++x) vacc[r][x] = 0.f;

    const int tile_end = min(n_tiles, (sp + 1) * tiles_per);
    for (int tile = sp * tiles_per; tile < tile_end; ++tile) {
        const int u0 = tile * KS;
        const int nk = min(KS, n - u0);
        __syncthreads();   // the previous tile is consumed (first pass: qs and the running maxima are written)
        const int jk = u0 + tid < kx ? u0 + tid : j_lo + (u0 + tid - kx);
        const int src = tid < nk ? key_source(a, jk, p) : -1;
        ksrc[tid] = src;
        {   // scores: one thread per key
            float acc[RMAX];
#pragma unroll
            for (int r = 0; r < RMAX; ++r) acc[r] = 0.f;
            if (src != -1) {
                const CT* krow = src >= 0 ? kc + ((size_t)g * a.L + src) * Dk : kn + (size_t)g * Dk;
                if (vec_rows) {
                    const uint4* k16 = reinterpret_cast<const uint4*>(krow);
                    const float4* q4 = reinterpret_cast<const float4*>(qs);
                    const int nv = Dk / VEC, q4_row = Dq / 4;
#pragma unroll 8
                    for (int i = 0; i < nv; ++i) {
                        const uint4 u = __ldg(k16 + i);
                        const CT* e = reinterpret_cast<const CT*>(&u);
                        float kf[VEC];
#pragma unroll
                        for (int x = 0; x < VEC; ++x) kf[x] = ldf(e, x);
#pragma unroll
                        for (int r = 0; r < RMAX; ++r)
                            if (r < R) {
#pragma unroll
                                for (int x4 = 0; x4 < VEC / 4; ++x4) {
                                    const float4 qv = q4[r * q4_row + i * (VEC / 4) + x4];
                                    acc[r] = fmaf(qv.x, kf[4 * x4 + 0], acc[r]);
                                    acc[r] = fmaf(qv.y, kf[4 * x4 + 1], acc[r]);
                                    acc[r] = fmaf(qv.z, kf[4 * x4 + 2], acc[r]);
                                    acc[r] = fmaf(qv.w, kf[4 * x4 + 3], acc[r]);
                                }
                            }
                    }
                } else {
                    for (int d = 0; d < Dk; ++d) {
                        const float kv = ldf(krow, d);
#pragma unroll
                        for (int r = 0; r < RMAX; ++r)
                            if (r < R) acc[r] = fmaf(qs[r * Dq + d], kv, acc[r]);
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < RMAX; ++r)
                if (r < R) Ps[r * KS + tid] = src != -1 ? shape_score(a, acc[r] * a.scale, g * R + r, p - jk) : -INFINITY;
        }
        __syncthreads();
        for (int r = warp; r < R; r += DEC_THREADS / 32) {
            float mx = -INFINITY;
            for (int k = lane; k < KS; k += 32) mx = fmaxf(mx, Ps[r * KS + k]);
            mx = warp_max(mx);
            const float m_old = s_M[r];
            const float m_new = fmaxf(m_old, mx);
            float sum = 0.f;
            for (int k = lane; k < KS; k += 32) {
                const float sv = Ps[r * KS + k];
                const float pr = sv == -INFINITY ? 0.f : expf(sv - m_new);
                Ps[r * KS + k] = pr;
                sum += pr;
            }
            sum = warp_sum(sum);
            if (lane == 0) {
                const float corr = m_old == -INFINITY ? 0.f : expf(m_old - m_new);
                s_corr[r] = corr;
                s_L[r] = s_L[r] * corr + sum;
                s_M[r] = m_new;
            }
        }
        __syncthreads();
        if (vec_values) {
            // thread (kg, cg): keys kg, kg + nkg, ... of the tile x the VEC value columns of group cg, 16-byte loads
            if (kg < nkg) {
#pragma unroll
                for (int r = 0; r < VR; ++r)
                    if (r < R) {
                        const float cr = s_corr[r];
#pragma unroll
                        for (int x = 0; x < VEC; ++x) vacc[r][x] *= cr;
                    }
                const CT* vbase = vc + (size_t)g * a.L * Dv + cg * VEC;
                const CT* vnew = vn + (size_t)g * Dv + cg * VEC;
#pragma unroll 4
                for (int k = kg; k < nk; k += nkg) {
                    const int s = ksrc[k];
                    if (s == -1) continue;
                    const uint4 u = __ldg(reinterpret_cast<const uint4*>(s >= 0 ? vbase + (size_t)s * Dv : vnew));
                    const CT* e = reinterpret_cast<const CT*>(&u);
                    float vf[VEC];
#pragma unroll
                    for (int x = 0; x < VEC; ++x) vf[x] = ldf(e, x);
#pragma unroll
                    for (int r = 0; r < VR; ++r)
                        if (r < R) {
                            const float pw = Ps[r * KS + k];
#pragma unroll
                            for (int x = 0; x < VEC; ++x) vacc[r][x] = fmaf(pw, vf[x], vacc[r][x]);
                        }
                }
            }
        } else {
    #pragma unroll
            for (int cc = 0; cc < 2; ++cc) {
                const int c = tid + cc * DEC_THREADS;
                if (c >= Dv) break;
    #pragma unroll
                for (int r = 0; r < RMAX; ++r)
                    if (r < R) oacc[cc][r] *= s_corr[r];
                const CT* vbase = vc + (size_t)g * a.L * Dv + c;
                const CT* vnew = vn + (size_t)g * Dv + c;
    #pragma unroll 2
                for (int k = 0; k < KS; k += 4) {
                    if (k >= nk) break;
                    float v[4];
    #pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int s = ksrc[k + i];   // -1 beyond nk as well
                        v[i] = s >= 0 ? ldf(vbase, (size_t)s * Dv) : (s <= -2 ? ldf(vnew, 0) : 0.f);
                    }
    #pragma unroll
                    for (int r = 0; r < RMAX; ++r)
                        if (r < R) {
                            const float4 pw = *reinterpret_cast<const float4*>(Ps + r * KS + k);
                            oacc[cc][r] = fmaf(pw.x, v[0], oacc[cc][r]);
                            oacc[cc][r] = fmaf(pw.y, v[1], oacc[cc][r]);
                            oacc[cc][r] = fmaf(pw.z, v[2], oacc[cc][r]);
                            oacc[cc][r] = fmaf(pw.w, v[3], oacc[cc][r]);
                        }
                }
            }
    
        }
    }
    if (vec_values) {   // sum the key groups' partial value sums: red[kg][r][c] -> column c of this thread
        __syncthreads();
        float* red = Ps + R * KS + KS;   // behind the key sources
        if (kg < nkg) {
#pragma unroll
            for (int r = 0; r < VR; ++r)
                if (r < R) {
#pragma unroll
                    for (int x = 0; x < VEC; ++x) red[((size_t)kg * R + r) * Dv + cg * VEC + x] = vacc[r][x];
                }
        }
        __syncthreads();
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
            const int c = tid + cc * DEC_THREADS;
            if (c >= Dv) break;
#pragma unroll
            for (int r = 0; r < RMAX; ++r)
                if (r < R) {
                    float t = 0.f;
                    for (int q = 0; q < nkg; ++q) t += red[((size_t)q * R + r) * Dv + c];
                    oacc[cc][r] = t;
                }
        }
    }
    const size_t pbase = ((size_t)g * NS + sp) * R;
    if (tid < R) { part_m[pbase + tid] = s_M[tid]; part_l[pbase + tid] = s_L[tid]; }
#pragma unroll
    for (int cc = 0; cc < 2; ++cc) {
        const int c = tid + cc * DEC_THREADS;
        if (c >= Dv) break;
#pragma unroll
        for (int r = 0; r < RMAX; ++r)
            if (r < R) part_o[(pbase + r) * Dv + c] = oacc[cc][r];
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = (atomicAdd(&counters[g], 1) == nsplit - 1);
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // the last CTA of this head: every other CTA of the head has finished reading; combine in split order
    // (partials are read with ld.global.cg: other SMs wrote them, so L1 is bypassed)
    YT* y = (YT*)a.y;
    __shared__ float s_inv[16], s_max[16];
    float* wgt = Ps;   // [R, KS] weights of up to KS splits at a time (reuses the probability tile)
    for (int r = warp; r < R; r += DEC_THREADS / 32) {
        const int h = g * R + r;
        float M = -INFINITY;
        if (a.sink_mode == CC_SINK_LEARNED) M = a.sink[h];
        else if (a.sink_mode == CC_SINK_ZERO) M = 0.f;
        const float sinkv = M;
        for (int s = lane; s < nsplit; s += 32) M = fmaxf(M, __ldcg(part_m + ((size_t)g * NS + s) * R + r));
        M = warp_max(M);
        float Lsum = 0.f;
        for (int s = lane; s < nsplit; s += 32) {
            const size_t b = ((size_t)g * NS + s) * R + r;
            const float ms = __ldcg(part_m + b);
            Lsum += __ldcg(part_l + b) * (ms == -INFINITY ? 0.f : expf(ms - M));
        }
        Lsum = warp_sum(Lsum);
        if (a.sink_mode != CC_SINK_NONE) Lsum += expf(sinkv - M);
        if (lane == 0) { s_inv[r] = Lsum > 0.f ? 1.0f / Lsum : 0.f; s_max[r] = M; }
    }
    for (int c0 = 0; c0 < Dv; c0 += DEC_THREADS) {
        const int c = c0 + tid;
        float acc[RMAX];
#pragma unroll
        for (int r = 0; r < RMAX; ++r) acc[r] = 0.f;
        for (int s0 = 0; s0 < nsplit; s0 += KS) {   // splits in order, KS at a time
            const int ns = min(KS, nsplit - s0);
            __syncthreads();
            for (int i = tid; i < R * ns; i += DEC_THREADS) {
                const int r = i / ns, s = i - r * ns;
                const float ms = __ldcg(part_m + ((size_t)g * NS + s0 + s) * R + r);
                wgt[r * KS + s] = ms == -INFINITY ? 0.f : expf(ms - s_max[r]);
            }
            __syncthreads();
            if (c < Dv) {
#pragma unroll 8
                for (int s = 0; s < ns; ++s) {
                    const float* po = part_o + (((size_t)g * NS + s0 + s) * R) * Dv + c;
#pragma unroll
                    for (int r = 0; r < RMAX; ++r)
                        if (r < R) acc[r] = fmaf(__ldcg(po + (size_t)r * Dv), wgt[r * KS + s], acc[r]);
                }
            }
        }
        if (c < Dv) {
#pragma unroll
            for (int r = 0; r < RMAX; ++r)
                if (r < R) stf(y, (size_t)(g * R + r) * Dv + c, acc[r] * s_inv[r]);
        }
    }
    if (tid == 0) counters[g] = 0;
    if (a.append) append_row<CT>(a, g, 0, p, tid, DEC_THREADS);
}

// ---- the same for rows of whole 16-byte vectors and up to 8 query heads per key/value head
// A run of VT-key tiles per CTA; the key and value rows of a tile are all requested at once (cp.async, the next tile under
// this one) before anything is known about their slots, which are checked meanwhile.  Scores: eight lanes per key, four keys
// at a time, the query rows read from shared memory once for the four.  Values: a thread owns a 16-byte column group and
// every nkg-th key.  Two fp32 operations per instruction in both.  Partials and their combination as above, 16 bytes a load
// and 16 loads in flight.
// Bound: issue slots and the chain of dependent round trips (lookup and rows, partials, counter, combination), not the rows'
// bandwidth.  8 layers, 32 / 8 heads of 128, 4096 positions in a graph: 32 us a layer on the kernel above (a thread walks a
// row, values are read after the scores), 27 with rows requested at once, 18 with 256 threads, 128-key tiles, paired operations and ring
// places without a division per row.
constexpr int VD_THREADS = 256, VD_MAX_SPLITS = 64, VD_RMAX = 8;

// tiles of VT keys that a head can have at most, and the runs they are cut into: as many CTAs over the heads as the GPU holds at once
inline long long vd_tiles(int L, int reach, int VT) {
    const long long maxkeys = reach > 0 && reach <= L ? reach : (long long)L + 1;
    return (maxkeys + VT - 1) / VT;
}
inline int vd_splits(long long tiles, int G, int per_sm) {
    long long most = 148 * per_sm / G;
    if (most < 1) most = 1;
    if (most > VD_MAX_SPLITS) most = VD_MAX_SPLITS;
    return (int)(tiles < most ? tiles : most);
}

__device__ __forceinline__ void cp_async16_or_zero(void* dst, const void* src, bool have) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(have ? 16 : 0) : "memory");
}

// pairs of fp32 values: one instruction for two operations, each rounded as the scalar one
typedef unsigned long long f32x2;
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
// the elements of a 16-byte vector as pairs
__device__ __forceinline__ void as_pairs(const uint4& u, f32x2 (&v)[2], const float*) {
    v[0] = pair(__uint_as_float(u.x), __uint_as_float(u.y));
    v[1] = pair(__uint_as_float(u.z), __uint_as_float(u.w));
}
__device__ __forceinline__ void as_pairs(const uint4& u, f32x2 (&v)[4], const __nv_bfloat16*) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = pair(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
}

template <typename CT, typename YT, int RMAX, int VT>
__global__ void __launch_bounds__(VD_THREADS, RMAX <= 4 ? 2 : 1) attn_decode_rows_kernel(const CcSeqAttn a, int buffers, int NS) {
    extern __shared__ float4 smd4[];
    constexpr int VEC = 16 / (int)sizeof(CT), VP = VEC / 2, WARPS = VD_THREADS / 32, KEYS = VT / WARPS, KI = KEYS / 4;
    const int R = a.H / a.G, Dk = a.Dk, Dv = a.Dv, kc16 = Dk / VEC, vc16 = Dv / VEC;
    const int k_row = kc16 + 1, k_tile = VT * k_row, v_tile = VT * vc16;         // 16-byte units; one of padding per key row
    uint4* const ks = reinterpret_cast<uint4*>(smd4);                            // [buffers][VT][k_row]
    uint4* const vs = ks + buffers * k_tile;                                     // [buffers][VT][vc16]
    float* const qs = reinterpret_cast<float*>(vs + buffers * v_tile);           // [R][Dk]
    float* const Ps = qs + RMAX * Dk;                                            // [RMAX][VT]
    __shared__ int s_live[2][VT];
    __shared__ float s_M[RMAX], s_L[RMAX], s_corr[RMAX], s_inv[RMAX];
    __shared__ int s_last;

    pdl_wait_release();
    const int sp = blockIdx.x, g = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int p = a.input_pos[0];
    const int j_lo = a.block > 0 ? (p / a.block) * a.block : (a.window > 0 ? max(0, p - a.window + 1) : 0);
    const int kx = a.window > 0 ? min(a.keep_first, j_lo) : 0;
    const int n = kx + (p - j_lo + 1);
    const int n_tiles = (n + VT - 1) / VT, nsplit = min(n_tiles, NS);      // runs of n_tiles / nsplit tiles, or of one more
    if (sp >= nsplit) return;
    const int tile0 = (int)((long long)sp * n_tiles / nsplit), tile_end = (int)((long long)(sp + 1) * n_tiles / nsplit), ring = a.L - a.keep_first;
    // copies: thread = column c of rows row, row + step, ...
    const int k_step = VD_THREADS / kc16, k_first = tid / kc16, k_col = tid - k_first * kc16;
    const int v_step = VD_THREADS / vc16, v_first = tid / vc16, v_col = tid - v_first * vc16;
    const CT* const kc = (const CT*)a.k_cache + (size_t)g * a.L * Dk + k_col * VEC;
    const CT* const vc = (const CT*)a.v_cache + (size_t)g * a.L * Dv + v_col * VEC;
    const CT* const kn = (const CT*)a.k_new + (size_t)g * Dk + k_col * VEC;
    const CT* const vn = (const CT*)a.v_new + (size_t)g * Dv + v_col * VEC;

    auto fetch = [&](int tile) {
        const int b = buffers > 1 ? (tile - tile0) & 1 : 0, u0 = tile * VT;
        // beside the kept first positions a tile's slots are one or two runs of the ring (rings of at least a tile)
        const int j0 = u0 < kx ? 0 : j_lo + (u0 - kx);
        const bool plain = u0 >= kx && j0 >= a.keep_first && ring >= VT;
        const int r0 = plain ? (j0 - a.keep_first) % ring : 0;
        auto position = [&](int row) { return u0 + row < kx ? u0 + row : j_lo + (u0 + row - kx); };
        auto slot = [&](int row) {
            if (!plain) return slot_of(a, position(row));
            const int r = r0 + row;
            return a.keep_first + (r >= ring ? r - ring : r);
        };
        const int rows = min(VT, n - u0), last = p - (u0 < kx ? 0 : j0);      // row of the token itself, in a tile beside the kept ones
        if (k_first < k_step) {
#pragma unroll 4
            for (int row = k_first; row < VT; row += k_step) {
                const bool have = row < rows, mine = plain ? row == last : position(row) == p;
                cp_async16_or_zero(ks + b * k_tile + row * k_row + k_col, have && !mine ? kc + (size_t)slot(row) * Dk : kn, have);
            }
        }
        if (v_first < v_step) {
#pragma unroll 4
            for (int row = v_first; row < VT; row += v_step) {
                const bool have = row < rows, mine = plain ? row == last : position(row) == p;
                cp_async16_or_zero(vs + b * v_tile + row * vc16 + v_col, have && !mine ? vc + (size_t)slot(row) * Dv : vn, have);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (tid < VT) {
            const int j = position(tid);
            s_live[(tile - tile0) & 1][tid] = tid < rows && (j == p || a.pos[slot(tid)] == j);
        }
    };
    fetch(tile0);
    for (int i = tid; i < R * Dk; i += VD_THREADS) qs[i] = a.q[(size_t)g * R * Dk + i];
    if (tid < RMAX) { s_M[tid] = -INFINITY; s_L[tid] = 0.f; }
    const int nkg = v_step, kg = v_first, cg = v_col;     // value phase: key groups x column groups
    f32x2 acc[RMAX][VP];
#pragma unroll
    for (int r = 0; r < RMAX; ++r)
#pragma unroll
        for (int x = 0; x < VP; ++x) acc[r][x] = 0ull;

    for (int tile = tile0; tile < tile_end; ++tile) {
        const int b = buffers > 1 ? (tile - tile0) & 1 : 0, u0 = tile * VT;
        const int* live = s_live[(tile - tile0) & 1];
        if (buffers > 1 && tile + 1 < tile_end) {
            fetch(tile + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        {   // scores: keys KEYS warp + 4 i + lane / 8
            const int part = lane & 7, k0 = KEYS * warp + (lane >> 3);
            f32x2 sc[KI][RMAX];
#pragma unroll
            for (int i = 0; i < KI; ++i)
#pragma unroll
                for (int r = 0; r < RMAX; ++r) sc[i][r] = 0ull;
            for (int c = part; c < kc16; c += 8) {
                f32x2 kf[KI][VP];
#pragma unroll
                for (int i = 0; i < KI; ++i) as_pairs(ks[b * k_tile + (k0 + 4 * i) * k_row + c], kf[i], (const CT*)nullptr);
#pragma unroll
                for (int r = 0; r < RMAX; ++r)
                    if (r < R) {
#pragma unroll
                        for (int x4 = 0; x4 < VEC / 4; ++x4) {
                            const float4 qv = *reinterpret_cast<const float4*>(qs + r * Dk + c * VEC + 4 * x4);
                            const f32x2 q0 = pair(qv.x, qv.y), q1 = pair(qv.z, qv.w);
#pragma unroll
                            for (int i = 0; i < KI; ++i) sc[i][r] = fma2(q1, kf[i][2 * x4 + 1], fma2(q0, kf[i][2 * x4], sc[i][r]));
                        }
                    }
            }
#pragma unroll
            for (int i = 0; i < KI; ++i) {
                const int k = k0 + 4 * i, j = u0 + k < kx ? u0 + k : j_lo + (u0 + k - kx);
                const bool ok = live[k] != 0;
                float mine = 0.f;      // lane `part` of the key closes query head `part`
#pragma unroll
                for (int r = 0; r < RMAX; ++r) {
                    if (r >= R) break;
                    float s0, s1;
                    unpair(sc[i][r], s0, s1);
                    s0 += s1;
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
                    mine = part == r ? s0 : mine;
                }
                if (part < R) Ps[part * VT + k] = ok ? shape_score(a, mine * a.scale, g * R + part, p - j) : -INFINITY;
            }
        }
        __syncthreads();
        for (int r = warp; r < R; r += WARPS) {
            float sv[VT / 32], mx = -INFINITY, sum = 0.f;
#pragma unroll
            for (int q = 0; q < VT / 32; ++q) mx = fmaxf(mx, sv[q] = Ps[r * VT + lane + 32 * q]);
            const float m_old = s_M[r], m_new = fmaxf(m_old, warp_max(mx));
#pragma unroll
            for (int q = 0; q < VT / 32; ++q) {
                const float w = sv[q] == -INFINITY ? 0.f : expf(sv[q] - m_new);
                Ps[r * VT + lane + 32 * q] = w;
                sum += w;
            }
            sum = warp_sum(sum);
            if (lane == 0) {
                const float corr = m_old == -INFINITY ? 0.f : expf(m_old - m_new);
                s_corr[r] = corr;
                s_L[r] = s_L[r] * corr + sum;
                s_M[r] = m_new;
            }
        }
        __syncthreads();
        if (kg < nkg) {
            if (tile > tile0) {
#pragma unroll
                for (int r = 0; r < RMAX; ++r)
                    if (r < R) {
                        const float cr = s_corr[r];
#pragma unroll
                        for (int x = 0; x < VP; ++x) acc[r][x] = fma2(acc[r][x], pair(cr, cr), 0ull);
                    }
            }
#pragma unroll 4
            for (int k = kg; k < VT; k += nkg) {
                if (!live[k]) continue;
                f32x2 vf[VP];
                as_pairs(vs[b * v_tile + k * vc16 + cg], vf, (const CT*)nullptr);
#pragma unroll
                for (int r = 0; r < RMAX; ++r)
                    if (r < R) {
                        const float w = Ps[r * VT + k];
#pragma unroll
                        for (int x = 0; x < VP; ++x) acc[r][x] = fma2(pair(w, w), vf[x], acc[r][x]);
                    }
            }
        }
        __syncthreads();      // the tile is consumed: its buffers may be filled again
        if (buffers == 1 && tile + 1 < tile_end) fetch(tile + 1);
    }
    // the key groups' sums meet in group order: red[kg][r][c], over the tiles
    float* const red = reinterpret_cast<float*>(ks);
    if (kg < nkg) {
#pragma unroll
        for (int r = 0; r < RMAX; ++r)
            if (r < R) {
#pragma unroll
                for (int x = 0; x < VP; ++x) {
                    float s0, s1;
                    unpair(acc[r][x], s0, s1);
                    *reinterpret_cast<float2*>(red + ((size_t)kg * R + r) * Dv + cg * VEC + 2 * x) = make_float2(s0, s1);
                }
            }
    }
    __syncthreads();
    int* counters = (int*)a.workspace;
    float* part_m = (float*)(counters + ((a.G + 3) & ~3));
    float* part_l = part_m + (size_t)a.G * NS * R;
    float* part_o = (float*)(((uintptr_t)(part_l + (size_t)a.G * NS * R) + 15) & ~(uintptr_t)15);
    YT* y = (YT*)a.y + (size_t)g * R * Dv;
    auto sink_of = [&](int r) { return a.sink_mode == CC_SINK_LEARNED ? a.sink[g * R + r] : a.sink_mode == CC_SINK_ZERO ? 0.f : -INFINITY; };
    if (nsplit == 1) {
        if (tid < R) {
            const float sk = sink_of(tid), M = fmaxf(s_M[tid], sk);
            const float w = s_M[tid] == -INFINITY ? 0.f : expf(s_M[tid] - M);
            const float L = s_L[tid] * w + (a.sink_mode != CC_SINK_NONE ? expf(sk - M) : 0.f);
            s_inv[tid] = L > 0.f ? w / L : 0.f;
        }
        __syncthreads();
        for (int i = tid; i < R * Dv; i += VD_THREADS) {
            float t = 0.f;
            for (int q = 0; q < nkg; ++q) t += red[(size_t)q * R * Dv + i];
            stf(y, i, t * s_inv[i / Dv]);
        }
        if (a.append) append_row<CT>(a, g, 0, p, tid, VD_THREADS);
        return;
    }
    const size_t pbase = ((size_t)g * NS + sp) * R;
    for (int i = tid; i < R * Dv; i += VD_THREADS) {
        float t = 0.f;
        for (int q = 0; q < nkg; ++q) t += red[(size_t)q * R * Dv + i];
        part_o[pbase * Dv + i] = t;
    }
    if (tid < R) { part_m[pbase + tid] = s_M[tid]; part_l[pbase + tid] = s_L[tid]; }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(&counters[g], 1) == nsplit - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // the last CTA of the head: every other one has finished reading; combine in split order
    static_assert(VD_MAX_SPLITS <= VT, "the weights of the splits take the place of a tile's");
    float* const wgt = Ps;     // [R][VT]
    for (int r = warp; r < R; r += WARPS) {
        const float sk = sink_of(r);
        const float* pm = part_m + (size_t)g * NS * R + r;
        const float m0 = lane < nsplit ? __ldcg(pm + (size_t)lane * R) : -INFINITY, m1 = lane + 32 < nsplit ? __ldcg(pm + (size_t)(lane + 32) * R) : -INFINITY;
        const float* pl = part_l + (size_t)g * NS * R + r;
        const float l0 = lane < nsplit ? __ldcg(pl + (size_t)lane * R) : 0.f, l1 = lane + 32 < nsplit ? __ldcg(pl + (size_t)(lane + 32) * R) : 0.f;
        const float M = fmaxf(sk, warp_max(fmaxf(m0, m1)));
        const float w0 = m0 == -INFINITY ? 0.f : expf(m0 - M), w1 = m1 == -INFINITY ? 0.f : expf(m1 - M);
        wgt[r * VT + lane] = w0;
        wgt[r * VT + lane + 32] = w1;
        float L = warp_sum(l0 * w0 + l1 * w1);
        if (a.sink_mode != CC_SINK_NONE) L += expf(sk - M);
        if (lane == 0) s_inv[r] = L > 0.f ? 1.0f / L : 0.f;
    }
    __syncthreads();
    const float4* po = reinterpret_cast<const float4*>(part_o + (size_t)g * NS * R * Dv);     // Dv is a multiple of 4
    const int quads = R * Dv / 4;
    for (int i = tid; i < quads; i += VD_THREADS) {
        const int r = i / (Dv / 4);
        const float* w = wgt + r * VT;
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 16
        for (int s = 0; s < nsplit; ++s) {
            const float4 v = __ldcg(po + (size_t)s * quads + i);
            t.x = fmaf(w[s], v.x, t.x);
            t.y = fmaf(w[s], v.y, t.y);
            t.z = fmaf(w[s], v.z, t.z);
            t.w = fmaf(w[s], v.w, t.w);
        }
        const float inv = s_inv[r];
        stf(y, 4 * i + 0, t.x * inv);
        stf(y, 4 * i + 1, t.y * inv);
        stf(y, 4 * i + 2, t.z * inv);
        stf(y, 4 * i + 3, t.w * inv);
    }
    if (tid == 0) counters[g] = 0;
    if (a.append) append_row<CT>(a, g, 0, p, tid, VD_THREADS);
}

// ---- bf16 rows of that kind: both products on the tensor cores (mma.sync), fp32 queries and weights in three exact bf16 parts
// Truncation takes 8 of the 24 significant bits at a time, so the three parts of a number add up to it exactly and every product
// of a part with a bf16 key or value is exact; the sums are fp32.  An MMA cuts off what it adds below the last bit of the largest
// term, so those of the large part start from zero and are added up, rounded, outside.  Scores: 16 keys x 8 query heads per MMA, the three parts of q
// into one accumulator.  Values: 8 columns per MMA, two parts of the weights in the two halves of its 16 rows, the third in a
// second one; a warp owns columns, so no sums meet across warps.  Sums that are not finite (an infinite key or value meets parts
// that are zero) are formed again key by key with fp32 multiplications, where such operands give what they give.
// The keys of a tile are waited for alone, its values land under the scores and the softmax.  The last CTA of a head asks for all
// partial sums before it knows their weights, and stores the new row under them.
// Bound: the chain of dependent waits: position, keys, scores, softmax, values, partials and their counter, combination.  8 layers of 32 / 8
// heads of 128, 4096 positions in a graph: 143 us on the kernel above, 109 here, 106 since tiles come as boxes and slots' positions are
// compared after the query has been read.  Against 64 bits (fp32 results, scores of size 4): 2.1e-7 of the norm, 2.4e-7 above.
constexpr int MD_THREADS = 256, MD_WARPS = MD_THREADS / 32, MD_AHEAD = 17, MD_KEYS = 128;      // MD_KEYS: keys of a tile

__device__ __forceinline__ uint32_t smem_at(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_at(p)) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_at(p)) : "memory");
}
__device__ __forceinline__ void ldsm2(uint32_t (&r)[2], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(smem_at(p)) : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the parts of x, largest first
__device__ __forceinline__ void three_parts(float x, __nv_bfloat16 (&o)[3]) {
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const uint32_t top = __float_as_uint(x) & 0xffff0000u;
        o[i] = __ushort_as_bfloat16((unsigned short)(top >> 16));
        x -= __uint_as_float(top);
    }
}
__device__ __forceinline__ void md_bar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_at(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void md_bar_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_at(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void md_bar_arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_at(bar)) : "memory"); }
// a row of whole 16-byte vectors into shared memory; the barrier counts its bytes
__device__ __forceinline__ void md_copy_row(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_at(dst)), "l"(src), "r"(bytes),
                 "r"(smem_at(bar)) : "memory");
}
// 128 rows x 64 columns, swizzled, into shared memory
__device__ __forceinline__ void md_copy_box(void* dst, const CUtensorMap* tm, int column, int row, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_at(dst)), "l"(tm),
                 "r"(smem_at(bar)), "r"(column), "r"(row) : "memory");
}
// bounded: a copy that does not arrive ends the wait, not the kernel, whose results are then no numbers
__device__ __forceinline__ bool md_bar_wait(uint64_t* bar, uint32_t parity) {
    for (uint32_t n = 0; n < (1u << 22); ++n) {
        uint32_t done;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(done) : "r"(smem_at(bar)), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}
__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= 3.402823466e38f; }

struct MdLayout {
    int KU, k_row, v_row;                                   // 16-byte units: padded key row, strides (odd: rows on different banks)
    size_t vs, qs, qb, ps, pb, total;                       // byte offsets
};
// boxes: tiles as boxes of 64 columns, rows of 128 bytes one after another, 16-byte units swizzled by the row
__host__ __device__ inline MdLayout md_layout(int R, int Dk, int Dv, int buffers, bool boxes) {
    constexpr int VT = MD_KEYS;
    MdLayout l;
    l.KU = 2 * ((Dk + 15) / 16);
    l.k_row = boxes ? l.KU : l.KU + 1;
    l.v_row = boxes ? Dv / 8 : (Dv / 8) | 1;
    l.vs = (size_t)buffers * VT * l.k_row * 16;
    l.qs = l.vs + ((size_t)buffers * VT * l.v_row + 1) * 16;        // one more: the second half of an odd last tile is read
    l.qb = l.qs + ((size_t)R * Dk * 4 + 15) / 16 * 16;
    l.ps = l.qb + (size_t)3 * 8 * (l.KU + 1) * 16;
    l.pb = l.ps + (size_t)8 * VT * 4;
    l.total = l.pb + (size_t)3 * 8 * (VT + 8) * 2 + (boxes ? 1024 : 0);      // and the way to a multiple of 1024
    static_assert(MD_KEYS * 3 >= MD_THREADS, "the groups' sums of the combination take the keys' place, three units a row at least");
    return l;
}

template <typename YT, bool BOX>
__global__ void __launch_bounds__(MD_THREADS, 2) attn_decode_mma_kernel(const CcSeqAttn a, int buffers, int NS, const __grid_constant__ CUtensorMap k_map,
                                                                        const __grid_constant__ CUtensorMap v_map) {
    extern __shared__ float4 smd4[];
    typedef __nv_bfloat16 CT;
    constexpr int VT = MD_KEYS;
    uint8_t* const sm = reinterpret_cast<uint8_t*>(smd4) + (BOX ? (1024 - (smem_at(smd4) & 1023)) & 1023 : 0);
    const int R = a.H / a.G, Dk = a.Dk, Dv = a.Dv, kc16 = Dk / 8, vc16 = Dv / 8;
    const MdLayout lay = md_layout(R, Dk, Dv, buffers, BOX);
    const int KU = lay.KU, k_row = lay.k_row, v_row = lay.v_row, qb_row = 8 * (KU + 1);      // qb_row in elements
    uint4* const ks = reinterpret_cast<uint4*>(sm);                                 // [buffers][VT][k_row]
    uint4* const vs = reinterpret_cast<uint4*>(sm + lay.vs);                        // [buffers][VT][v_row]
    float* const qs = reinterpret_cast<float*>(sm + lay.qs);                        // [R][Dk]
    CT* const qb = reinterpret_cast<CT*>(sm + lay.qb);                              // [3][8][qb_row] parts of q, zero beyond R and Dk
    float* const Ps = reinterpret_cast<float*>(sm + lay.ps);                        // [8][VT]
    CT* const pb = reinterpret_cast<CT*>(sm + lay.pb);                              // [3][8][VT + 8] parts of the weights, zero beyond R
    // 16-byte unit c of a row of a tile
    auto unit = [](uint4* t, int row, int c, int stride) { return BOX ? t + (c >> 3) * 8 * VT + row * 8 + ((c ^ row) & 7) : t + row * stride + c; };
    __shared__ int s_live[2][VT];
    __shared__ float s_M[8], s_L[8], s_corr[8], s_inv[8];
    __shared__ int s_last;
    __shared__ volatile int s_lost;
    __shared__ __align__(8) uint64_t bars[2][2];      // [buffer][keys, values]

    const int sp = blockIdx.x, g = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        s_lost = 0;
        for (int i = 0; i < 4; ++i) md_bar_init(&bars[i >> 1][i & 1], MD_THREADS / 2);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < 3 * 8 * (VT + 8) / 8; i += MD_THREADS) reinterpret_cast<uint4*>(pb)[i] = make_uint4(0, 0, 0, 0);
    if (!BOX && KU > kc16)
        for (int i = tid; i < buffers * VT; i += MD_THREADS) ks[i * k_row + kc16] = make_uint4(0, 0, 0, 0);
    if (tid < 8) { s_M[tid] = -INFINITY; s_L[tid] = 0.f; s_corr[tid] = 0.f; s_inv[tid] = 0.f; }
    if (BOX && tid < 2) asm volatile("prefetch.tensormap [%0];" ::"l"(tid ? &v_map : &k_map) : "memory");
    pdl_wait_release();
    const int p = a.input_pos[0];
    const int j_lo = a.block > 0 ? (p / a.block) * a.block : (a.window > 0 ? max(0, p - a.window + 1) : 0);
    const int kx = a.window > 0 ? min(a.keep_first, j_lo) : 0;
    const int n = kx + (p - j_lo + 1);
    const int n_tiles = (n + VT - 1) / VT, nsplit = min(n_tiles, NS);      // runs of n_tiles / nsplit tiles, or of one more
    if (sp >= nsplit) return;
    const int tile0 = (int)((long long)sp * n_tiles / nsplit), tile_end = (int)((long long)(sp + 1) * n_tiles / nsplit);
    __syncthreads();      // the barriers and the zeros stand
    // The first half of the CTA asks for keys, the second for values, a thread per row: a whole tile is under way at once, where 16
    // copies of 16 bytes per thread waited for one another (8 layers of 8 heads x 4096 positions of 128 + 128: 117 us, 109).
    static_assert(MD_THREADS == 2 * VT, "a thread per row");
    const bool value = tid >= MD_THREADS / 2;
    const int ht = tid & (MD_THREADS / 2 - 1), D = value ? Dv : Dk, stride = value ? v_row : k_row;
    const CT* const fresh_row = value ? (const CT*)a.v_new + (size_t)g * Dv : (const CT*)a.k_new + (size_t)g * Dk;
    const CT* const cached = (value ? (const CT*)a.v_cache : (const CT*)a.k_cache) + (size_t)g * a.L * D;
    int held = 0;
    auto fetch = [&](int tile) {
        const int b = buffers > 1 ? (tile - tile0) & 1 : 0, u0 = tile * VT, rows = min(VT, n - u0);
        uint64_t* const bar = &bars[b][value];
        uint4* const dst = (value ? vs : ks) + b * VT * stride;
        auto position = [&](int row) { return u0 + row < kx ? u0 + row : j_lo + (u0 + row - kx); };
        auto source = [&](int row) {
            const int j = position(row);
            return j == p ? fresh_row : cached + (size_t)slot_of(a, j) * D;
        };
        if constexpr (BOX) {
            // One run of slots, but for the token itself, which is put over what was fetched in its place: boxes.  Otherwise (at the end
            // of a ring, or beside kept positions) rows by asynchronous copies of 16 bytes, neighbouring lanes in neighbouring bytes, that
            // arrive at the same barrier.  One such tile a head sets the time of all: 8 layers in a graph, us a layer by a row per thread through
            // registers / by these, 32 / 8 heads of 128, windows of 1000 behind 1128 positions 11.8 / 9.5, of 1000 and 4 kept 11.8 / 9.5, of 4096 and 128
            // kept 16.0 / 13.1, 8 / 2 heads of 256 15.6 / 11.2 (a bulk copy per row, all tiles so: 10.5, 10.5, 13.5, 12.0).
            const int ring = a.L - a.keep_first, j0 = position(0), r0 = j0 >= a.keep_first ? (j0 - a.keep_first) % ring : ring;
            const int old = rows - (u0 + rows == n ? 1 : 0);           // rows that the cache holds
            if (u0 >= kx && r0 + old <= ring) {
                if (ht == 0 && old > 0) {
                    md_bar_expect(bar, (uint32_t)VT * D * 2);
                    for (int c = 0; c < D; c += 64) md_copy_box(dst + c * (VT / 8), value ? &v_map : &k_map, c, g * a.L + a.keep_first + r0, bar);
                } else {
                    md_bar_arrive(bar);
                }
            } else {
                // a warp's 32 rows, 16 bytes a lane of rows one after another, all under way together
                const unsigned long long mine = ht < rows ? (unsigned long long)source(ht) : 0ull;
                const int units = D / 8, down = 32 / units, right = 32 - down * units;      // units: 8, 16, 24 or 32
                int r = lane / units, c = lane - r * units;
#pragma unroll 4
                for (int i = 0; i < units; ++i) {
                    const unsigned long long from = __shfl_sync(0xffffffffu, mine, r);
                    if (from != 0ull)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_at(unit(dst, (ht & ~31) + r, c, stride))), "l"(from + 16 * c) : "memory");
                    r += down;
                    c += right;
                    if (c >= units) { c -= units; ++r; }
                }
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_at(bar)) : "memory");
            }
        } else if (ht < rows) {
            md_bar_expect(bar, (uint32_t)D * 2);
            md_copy_row(dst + ht * stride, source(ht), (uint32_t)D * 2, bar);
        } else {
            md_bar_arrive(bar);
        }
        if (value && !BOX) {      // no position: whatever lay there must not meet a weight of zero
            if (ht >= rows)
                for (int c = 0; c < vc16; ++c) dst[ht * stride + c] = make_uint4(0, 0, 0, 0);
        }
        // whether the key's slot holds its position: asked for here, looked at by mark()
        const int j = position(ht);
        held = ht < rows ? j : j - 1;
        if (!value && ht < rows && j != p) held = a.pos[slot_of(a, j)];
    };
    auto mark = [&](int tile) {
        const int u = tile * VT + ht, j = u < kx ? u : j_lo + (u - kx);
        if (!value) s_live[(tile - tile0) & 1][ht] = held == j;
    };
    fetch(tile0);
    // boxes: the token's own row goes over what was fetched for it, and values without a position that meet a weight of zero become zero
    uint4 own = make_uint4(0, 0, 0, 0);
    if (BOX && ht < D / 8 && tile_end == n_tiles) own = reinterpret_cast<const uint4*>(fresh_row)[ht];
    auto finish = [&](int tile, uint4* t) {                  // the half of the CTA whose rows they are, before a barrier of the CTA
        const int rows = n - tile * VT;
        if (ht < D / 8) *unit(t, rows - 1, ht, stride) = own;
        if (value)
            for (int r = rows + ht / 8; r < ((rows + 15) & ~15); r += MD_THREADS / 16)      // of the 16 that a step of the product takes
                for (int c = ht & 7; c < D / 8; c += 8) *unit(t, r, c, stride) = make_uint4(0, 0, 0, 0);
    };
    const bool q16 = ((uintptr_t)a.q & 15) == 0;
    for (int i = 4 * tid; i < 8 * KU * 8; i += 4 * MD_THREADS) {      // four columns of a query row
        const int r = i / (KU * 8), d = i - r * (KU * 8);
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < R && d < Dk) {                                            // Dk is a multiple of 8
            const float* const at = a.q + ((size_t)g * R + r) * Dk + d;
            x = q16 ? *reinterpret_cast<const float4*>(at) : make_float4(at[0], at[1], at[2], at[3]);
            *reinterpret_cast<float4*>(qs + r * Dk + d) = x;
        }
        __align__(8) CT part[3][4];
        CT three[3];
        const float e[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            three_parts(e[c], three);
#pragma unroll
            for (int q = 0; q < 3; ++q) part[q][c] = three[q];
        }
#pragma unroll
        for (int q = 0; q < 3; ++q) *reinterpret_cast<uint2*>(qb + (q * 8 + r) * qb_row + d) = *reinterpret_cast<const uint2*>(part[q]);
    }
    mark(tile0);
    const int row_r = lane >> 2, col2 = (lane & 3) * 2;      // of an accumulator
    float acc[2][2][2];                                      // [pair of column tiles][tile][column]: head row_r
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int t = 0; t < 2; ++t) acc[i][t][0] = acc[i][t][1] = 0.f;

    for (int tile = tile0; tile < tile_end; ++tile) {
        const int b = buffers > 1 ? (tile - tile0) & 1 : 0, u0 = tile * VT;
        const int* live = s_live[(tile - tile0) & 1];
        const uint32_t turn = (buffers > 1 ? (tile - tile0) >> 1 : tile - tile0) & 1;
        if (buffers > 1 && tile + 1 < tile_end) {
            fetch(tile + 1);
            mark(tile + 1);
        }
        bool landed = md_bar_wait(&bars[b][0], turn);
        uint4* const kt = ks + b * VT * k_row;
        if (BOX && !value && tile == n_tiles - 1) finish(tile, kt);
        __syncthreads();
        for (int mt = warp; mt < VT / 16; mt += MD_WARPS) {
            float d[2][4], small[2][4];      // sums of even and odd steps; of the two smaller parts
#pragma unroll
            for (int e = 0; e < 4; ++e) d[0][e] = d[1][e] = small[0][e] = small[1][e] = 0.f;
#pragma unroll 4
            for (int k = 0; k < KU / 2; ++k) {
                uint32_t ka[4];
                ldsm4(ka, unit(kt, 16 * mt + (lane & 15), 2 * k + (lane >> 4), k_row));
                float step[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int q = 2; q >= 0; --q) {
                    uint32_t bq[2];
                    ldsm2(bq, qb + (q * 8 + (lane & 7)) * qb_row + 16 * k + ((lane >> 3) & 1) * 8);
                    mma16816(q > 0 ? small[q - 1] : step, ka[0], ka[1], ka[2], ka[3], bq[0], bq[1]);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (k & 1) d[1][e] += step[e];
                    else d[0][e] += step[e];
                }
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int k = 16 * mt + row_r + 8 * (e >> 1), r = col2 + (e & 1), j = u0 + k < kx ? u0 + k : j_lo + (u0 + k - kx);
                if (r >= R) continue;
                float s = (d[0][e] + d[1][e]) + (small[0][e] + small[1][e]);
                if (!finite(s) && live[k]) {
                    s = 0.f;
                    for (int c = 0; c < Dk; ++c) s = fmaf(qs[r * Dk + c], __bfloat162float(reinterpret_cast<const CT*>(unit(kt, k, c >> 3, k_row))[c & 7]), s);
                }
                Ps[r * VT + k] = live[k] ? shape_score(a, s * a.scale, g * R + r, p - j) : -INFINITY;
            }
        }
        __syncthreads();
        if (warp < R) {
            const int r = warp;
            float sv[VT / 32], mx = -INFINITY, sum = 0.f;
#pragma unroll
            for (int q = 0; q < VT / 32; ++q) mx = fmaxf(mx, sv[q] = Ps[r * VT + lane + 32 * q]);
            const float m_old = s_M[r], m_new = fmaxf(m_old, warp_max(mx));
#pragma unroll
            for (int q = 0; q < VT / 32; ++q) {
                const float w = sv[q] == -INFINITY ? 0.f : expf(sv[q] - m_new);
                CT part[3];
                three_parts(w, part);
                Ps[r * VT + lane + 32 * q] = w;
#pragma unroll
                for (int i = 0; i < 3; ++i) pb[(i * 8 + r) * (VT + 8) + lane + 32 * q] = part[i];
                sum += w;
            }
            sum = warp_sum(sum);
            if (lane == 0) {
                const float corr = m_old == -INFINITY ? 0.f : expf(m_old - m_new);
                s_corr[r] = corr;
                s_L[r] = s_L[r] * corr + sum;
                s_M[r] = m_new;
            }
        }
        landed = md_bar_wait(&bars[b][1], turn) && landed;
        uint4* const vt = vs + b * VT * v_row;
        if (BOX && value && tile == n_tiles - 1) finish(tile, vt);
        if (!landed) s_lost = 1;
        __syncthreads();
        const bool lost = s_lost;                                // read by all between two barriers without a wait in between
        const float corr = s_corr[row_r];
        const int steps = min(VT, n - u0 + 15) >> 4;             // further rows have no position
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int np = warp + MD_WARPS * i;
            if (16 * np >= Dv) break;
            float d[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, odd[2][2] = {{0.f, 0.f}, {0.f, 0.f}}, small[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll 4
            for (int k = 0; k < steps; ++k) {
                uint32_t pa[4], pc[2], vb[4];
                ldsm4(pa, pb + (((lane >> 3) & 1) * 8 + (lane & 7)) * (VT + 8) + 16 * k + (lane >> 4) * 8);
                ldsm2(pc, pb + (16 + (lane & 7)) * (VT + 8) + 16 * k + ((lane >> 3) & 1) * 8);
                ldsm4_t(vb, unit(vt, 16 * k + (lane & 15), 2 * np + (lane >> 4), v_row));
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    float step[4] = {0.f, 0.f, 0.f, 0.f};
                    mma16816(small[t], pc[0], 0u, pc[1], 0u, vb[2 * t], vb[2 * t + 1]);
                    mma16816(step, pa[0], pa[1], pa[2], pa[3], vb[2 * t], vb[2 * t + 1]);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        if (k & 1) odd[t][e] += step[e];
                        else d[t][e] += step[e];
                        d[t][2 + e] += step[2 + e];
                    }
                }
            }
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int c = 16 * np + 8 * t + col2 + e;
                    float sum = (d[t][e] + odd[t][e]) + (d[t][2 + e] + small[t][e]);
                    if (!finite(sum) && row_r < R && c < Dv) {
                        sum = 0.f;
                        for (int k = 0; k < VT; ++k)
                            if (live[k]) sum = fmaf(Ps[row_r * VT + k], __bfloat162float(reinterpret_cast<const CT*>(unit(vt, k, c >> 3, v_row))[c & 7]), sum);
                    }
                    acc[i][t][e] = tile > tile0 ? fmaf(acc[i][t][e], corr, sum) : sum;
                }
        }
        if (lost) {           // a copy did not arrive: those under way end before the CTA goes on
            for (int i = 0; i < 2; ++i) {
                md_bar_wait(&bars[b][i], turn);
                if (buffers > 1 && tile + 1 < tile_end) md_bar_wait(&bars[b ^ 1][i], ((tile + 1 - tile0) >> 1) & 1);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int t = 0; t < 2; ++t) acc[i][t][0] = acc[i][t][1] = NAN;
            break;
        }
        if (tile + 1 == tile_end) break;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // reads before the copies that follow
        __syncthreads();      // the tile is consumed: its buffers may be filled again
        if (buffers == 1) {
            fetch(tile + 1);
            mark(tile + 1);
        }
    }
    int* counters = (int*)a.workspace;
    float* part_m = (float*)(counters + ((a.G + 3) & ~3));
    float* part_l = part_m + (size_t)a.G * NS * R;
    float* part_o = (float*)(((uintptr_t)(part_l + (size_t)a.G * NS * R) + 15) & ~(uintptr_t)15);
    YT* y = (YT*)a.y + (size_t)g * R * Dv;
    auto sink_of = [&](int r) { return a.sink_mode == CC_SINK_LEARNED ? a.sink[g * R + r] : a.sink_mode == CC_SINK_ZERO ? 0.f : -INFINITY; };
    // this thread's values: f(head, column, value, value of the next column)
    auto each_pair = [&](auto&& f) {
        if (row_r >= R) return;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int c = 16 * (warp + MD_WARPS * i) + 8 * t + col2;
                if (c < Dv) f(row_r, c, acc[i][t][0], acc[i][t][1]);
            }
    };
    if (nsplit == 1) {
        if (tid < R) {
            const float sk = sink_of(tid), M = fmaxf(s_M[tid], sk);
            const float w = s_M[tid] == -INFINITY ? 0.f : expf(s_M[tid] - M);
            const float L = s_L[tid] * w + (a.sink_mode != CC_SINK_NONE ? expf(sk - M) : 0.f);
            s_inv[tid] = L > 0.f ? w / L : 0.f;
        }
        __syncthreads();
        each_pair([&](int r, int c, float v0, float v1) {
            stf(y, (size_t)r * Dv + c, v0 * s_inv[r]);
            stf(y, (size_t)r * Dv + c + 1, v1 * s_inv[r]);
        });
        if (a.append) append_row<CT>(a, g, 0, p, tid, MD_THREADS);
        return;
    }
    const size_t pbase = ((size_t)g * NS + sp) * R;
    each_pair([&](int r, int c, float v0, float v1) { *reinterpret_cast<float2*>(part_o + (pbase + r) * Dv + c) = make_float2(v0, v1); });
    if (tid < R) { part_m[pbase + tid] = s_M[tid]; part_l[pbase + tid] = s_L[tid]; }
    __syncthreads();
    if (tid == 0) {      // releases what the whole CTA stored before the barrier, and acquires what the others did
        int before;
        asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;" : "=r"(before) : "l"(counters + g) : "memory");
        s_last = before == nsplit - 1;
    }
    __syncthreads();
    if (!s_last) return;
    // the last CTA of the head: every other one has finished reading
    static_assert(VD_MAX_SPLITS <= VT, "the weights of the splits take the place of a tile's");
    float* const wgt = Ps;     // [R][VT]
    const float4* po = reinterpret_cast<const float4*>(part_o + (size_t)g * NS * R * Dv);     // Dv is a multiple of 8
    const int quads = R * Dv / 4, groups = quads >= MD_THREADS ? 1 : min(8, MD_THREADS / quads);
    const int grp = groups > 1 ? tid / quads : 0, first = groups > 1 ? tid - grp * quads : tid;
    // asked for together: maxima and sums, the new row and its slot, the first partial sums
    const int hr = min(warp, R - 1);
    const float* pm = part_m + (size_t)g * NS * R + hr;
    const float* pl = part_l + (size_t)g * NS * R + hr;
    const float m0 = lane < nsplit ? __ldcg(pm + (size_t)lane * R) : -INFINITY, m1 = lane + 32 < nsplit ? __ldcg(pm + (size_t)(lane + 32) * R) : -INFINITY;
    const float l0 = lane < nsplit ? __ldcg(pl + (size_t)lane * R) : 0.f, l1 = lane + 32 < nsplit ? __ldcg(pl + (size_t)(lane + 32) * R) : 0.f;
    const int at = slot_of(a, p);
    const bool stores = a.append && tid < kc16 + vc16, key = tid < kc16;
    uint4 fresh = make_uint4(0, 0, 0, 0);
    int old = 0;
    if (stores) fresh = key ? reinterpret_cast<const uint4*>((const CT*)a.k_new + (size_t)g * Dk)[tid] : reinterpret_cast<const uint4*>((const CT*)a.v_new + (size_t)g * Dv)[tid - kc16];
    if (a.append && tid == 0 && g == 0) old = a.pos[at];
    float4 v[MD_AHEAD];
#pragma unroll
    for (int u = 0; u < MD_AHEAD; ++u)
        if (grp < groups && first < quads && grp + u * groups < nsplit) v[u] = __ldcg(po + (size_t)(grp + u * groups) * quads + first);
    if (warp < R) {
        const float sk = sink_of(hr), M = fmaxf(sk, warp_max(fmaxf(m0, m1)));
        const float w0 = m0 == -INFINITY ? 0.f : expf(m0 - M), w1 = m1 == -INFINITY ? 0.f : expf(m1 - M);
        wgt[hr * VT + lane] = w0;
        wgt[hr * VT + lane + 32] = w1;
        float L = warp_sum(l0 * w0 + l1 * w1);
        if (a.sink_mode != CC_SINK_NONE) L += expf(sk - M);
        if (lane == 0) s_inv[hr] = L > 0.f ? 1.0f / L : 0.f;
    }
    if (stores) {      // every CTA of the head has read its rows, and none of another head reads these
        if (key) reinterpret_cast<uint4*>((CT*)a.k_cache + ((size_t)g * a.L + at) * Dk)[tid] = fresh;
        else reinterpret_cast<uint4*>((CT*)a.v_cache + ((size_t)g * a.L + at) * Dv)[tid - kc16] = fresh;
        if (tid == 0) {
            if (a.mask != nullptr) a.mask[(size_t)g * a.L + at] = 1;
            if (g == 0) {
                a.pos[at] = p;
                if (old < 0 && a.cache_cts != nullptr) atomicAdd(a.cache_cts, 1);
            }
        }
    }
    if (tid == 0) counters[g] = 0;
    __syncthreads();
    // splits of a group in order, then the groups in order
    float4* const met = reinterpret_cast<float4*>(sm);      // [groups][quads], over the keys
    for (int i = first; i < quads && grp < groups; i += MD_THREADS) {
        const float* w = wgt + (i / (Dv / 4)) * VT;
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        auto add = [&](int s, const float4& x) {
            t.x = fmaf(w[s], x.x, t.x);
            t.y = fmaf(w[s], x.y, t.y);
            t.z = fmaf(w[s], x.z, t.z);
            t.w = fmaf(w[s], x.w, t.w);
        };
        if (i == first) {
#pragma unroll
            for (int u = 0; u < MD_AHEAD; ++u)
                if (grp + u * groups < nsplit) add(grp + u * groups, v[u]);
        }
#pragma unroll 16
        for (int s = grp + (i == first ? MD_AHEAD * groups : 0); s < nsplit; s += groups) add(s, __ldcg(po + (size_t)s * quads + i));
        if (groups == 1) {
            const float inv = s_inv[i / (Dv / 4)];
            stf(y, 4 * i + 0, t.x * inv);
            stf(y, 4 * i + 1, t.y * inv);
            stf(y, 4 * i + 2, t.z * inv);
            stf(y, 4 * i + 3, t.w * inv);
        } else {
            met[grp * quads + i] = t;
        }
    }
    if (groups == 1) return;
    __syncthreads();
    if (tid < quads) {
        float4 t = met[tid];
        for (int q = 1; q < groups; ++q) {
            const float4 x = met[q * quads + tid];
            t.x += x.x; t.y += x.y; t.z += x.z; t.w += x.w;
        }
        const float inv = s_inv[tid / (Dv / 4)];
        stf(y, 4 * tid + 0, t.x * inv);
        stf(y, 4 * tid + 1, t.y * inv);
        stf(y, 4 * tid + 2, t.z * inv);
        stf(y, 4 * tid + 3, t.w * inv);
    }
}

template <typename CT>
__global__ void cache_append_kernel(const CcSeqAttn a, int t_first) {
    const int t = t_first + blockIdx.x, g = blockIdx.y;
    const int p = a.input_pos[0] + t;
    // a row whose slot a later row of the same chunk takes is not written (kept first positions never are)
    if (p >= a.keep_first && p + (a.L - a.keep_first) <= a.input_pos[0] + a.T - 1) return;
    append_row<CT>(a, g, t, p, threadIdx.x, blockDim.x);
}

// The same for rows of whole 16-byte vectors, launched under the attention before it: thread = vector x of the key row and then of the
// value row, of ROWS (token, head) rows that lie blockDim.y apart and are under way together; positions and marks by a thread
// per mark, neighbouring tokens in neighbouring threads, new slots counted by the warp.
// Bound: HBM and the launch.  Measured in a chain of launches, with a row per thread whose first thread stores its marks / so, us: 2 tokens of 8
// heads of 128 + 128 bf16 1.65 / 1.65, 64 4.9 / 1.65, 1001 12.7 / 3.3, 4096 of one head 16 / 3.1, of 8 19.5 / 5.75.
template <typename CT, int ROWS>
__global__ void __launch_bounds__(256) cache_append_rows_kernel(const CcSeqAttn a, int t_first) {
    pdl_wait_release();
    constexpr int VEC = 16 / (int)sizeof(CT);
    const int c = threadIdx.x, kc16 = a.Dk / VEC, p0 = a.input_pos[0];
    const bool key = c < kc16;
    const int D = key ? a.Dk : a.Dv, e = (key ? c : c - kc16) * VEC;
    auto kept = [&](int p) { return p < a.keep_first || p + (a.L - a.keep_first) > p0 + a.T - 1; };      // no later row takes its slot
    const CT* const src = (key ? (const CT*)a.k_new : (const CT*)a.v_new) + e;
    CT* const dst = (key ? (CT*)a.k_cache : (CT*)a.v_cache) + e;
    uint4 x[ROWS];
    long long to[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        const unsigned row = (blockIdx.x * ROWS + i) * blockDim.y + threadIdx.y, n = row / (unsigned)a.G;
        const int t = t_first + (int)n, g = (int)(row - n * (unsigned)a.G);
        to[i] = -1;
        if (t < a.T && kept(p0 + t)) {
            to[i] = ((long long)g * a.L + slot_of(a, p0 + t)) * D;
            x[i] = *reinterpret_cast<const uint4*>(src + ((size_t)t * a.G + g) * D);
        }
    }
#pragma unroll
    for (int i = 0; i < ROWS; ++i)
        if (to[i] >= 0) *reinterpret_cast<uint4*>(dst + to[i]) = x[i];
    const unsigned threads = blockDim.x * blockDim.y, tid = threadIdx.y * blockDim.x + c, tokens = a.T - t_first, marks = tokens * (unsigned)a.G;
    for (unsigned long long first = (unsigned long long)blockIdx.x * threads; first < marks; first += (unsigned long long)gridDim.x * threads) {
        const unsigned i = (unsigned)first + tid, g = i / tokens;
        const int t = t_first + (int)(i - g * tokens), p = p0 + t;
        bool fresh = false;
        if (i < marks && kept(p)) {
            const int slot = slot_of(a, p);
            if (a.mask != nullptr) a.mask[(size_t)g * a.L + slot] = 1;
            if (g == 0) {
                fresh = a.pos[slot] < 0;
                a.pos[slot] = p;
            }
        }
        const unsigned here = __activemask(), some = __ballot_sync(here, fresh);
        if (some != 0 && (tid & 31) == __ffs(here) - 1 && a.cache_cts != nullptr) atomicAdd(a.cache_cts, __popc(some));
    }
}

// ------------------------------------------------------------------------------------------------ post-sum norm
template <typename YT, typename AT>
__global__ void residual_norm_kernel(float* __restrict__ x, const YT* __restrict__ y, const float* __restrict__ w,
                                     float alpha, float eps, AT* __restrict__ x_act, int E) {
    __shared__ float red[32];
    const size_t base = (size_t)blockIdx.x * E;
    float ss = 0.f;
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        float s = alpha * x[base + e];
        if (y != nullptr) s += ldf(y, base + e);
        ss += s * s;
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x < 32) {
        float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
        v = warp_sum(v);
        if (threadIdx.x == 0) red[0] = v;
    }
    __syncthreads();
    const float r = 1.0f / sqrtf(red[0] / (float)E + eps);
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        float s = alpha * x[base + e];
        if (y != nullptr) s += ldf(y, base + e);
        const float v = s * r * (1.0f + w[e]);
        x[base + e] = v;
        if (x_act != nullptr) stf(x_act, base + e, v);
    }
}

// ------------------------------------------------------------------------------------------------ clamped gated unit
template <typename IT, typename OT>
__global__ void clamped_glu_kernel(const IT* __restrict__ gu, OT* __restrict__ out, float limit, float slope, int T,
                                   int F) {
    const size_t n = (size_t)T * F;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t t = i / F, f = i - t * F;
        const float g = fminf(ldf(gu, t * 2 * F + f), limit);
        const float u = fminf(fmaxf(ldf(gu, t * 2 * F + F + f), -limit), limit);
        stf(out, i, g * (1.0f / (1.0f + expf(-slope * g))) * (u + 1.0f));
    }
}

// ------------------------------------------------------------------------------------------------ one-token products
constexpr int GEMV_THREADS = 256, GEMV_ROWS = 8;   // one row per warp: small CTAs, many row streams in flight per SM
// (measured on a B200 at widths 2048 / 4096: 8 rows per CTA 0.435 / 0.801 ms per token, 16: 0.456 / 0.796, 32: 0.58 / 0.96;
// requesting a row's first vectors before the input is staged did not pay: 0.427 / 0.830)

__device__ __forceinline__ float block_sum(float v, float* red) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.f;
    if (threadIdx.x < 32) {
        t = warp_sum(t);
        if (threadIdx.x == 0) red[0] = t;
    }
    __syncthreads();
    t = red[0];
    __syncthreads();
    return t;
}

__device__ __forceinline__ float round_like(float v, const float*) { return v; }
__device__ __forceinline__ float round_like(float v, const __nv_bfloat16*) { return __bfloat162float(__float2bfloat16_rn(v)); }

// One row of W against the staged input: 16-byte loads, four in flight per lane.
template <typename WT>
__device__ __forceinline__ float row_dot(const WT* __restrict__ w, const float* __restrict__ xs, int K, int lane) {
    constexpr int VEC = 16 / (int)sizeof(WT);
    float acc = 0.f;
    if (K % VEC == 0) {
        const uint4* w16 = reinterpret_cast<const uint4*>(w);
        const int nv = K / VEC;
#pragma unroll 4
        for (int i = lane; i < nv; i += 32) {
            const uint4 u = __ldg(w16 + i);
            const WT* e = reinterpret_cast<const WT*>(&u);
            const float4* x4 = reinterpret_cast<const float4*>(xs + i * VEC);
#pragma unroll
            for (int q = 0; q < VEC / 4; ++q) {
                const float4 xv = x4[q];
                acc = fmaf(ldf(e, 4 * q + 0), xv.x, acc);
                acc = fmaf(ldf(e, 4 * q + 1), xv.y, acc);
                acc = fmaf(ldf(e, 4 * q + 2), xv.z, acc);
                acc = fmaf(ldf(e, 4 * q + 3), xv.w, acc);
            }
        }
    } else {
        for (int k = lane; k < K; k += 32) acc = fmaf(ldf(w, k), xs[k], acc);
    }
    return warp_sum(acc);
}

template <typename WT, typename XT, typename OT>
__global__ void __launch_bounds__(GEMV_THREADS) gemv_kernel(const CcSeqGemv g) {
    extern __shared__ float4 smg4[];
    float* xs = reinterpret_cast<float*>(smg4);   // [K] the product's input, rounded as the weights are
    __shared__ float red[32];
    const int K = g.K, N = g.N, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const XT* x = (const XT*)g.x;
    const WT* W = (const WT*)g.W;
    float rin = 1.f;
    if (g.in_norm_w != nullptr) {
        float ss = 0.f;
        for (int k = tid; k < K; k += GEMV_THREADS) { const float v = ldf(x, k); ss += v * v; }
        rin = 1.0f / sqrtf(block_sum(ss, red) / (float)K + g.eps);
    }
    for (int k = tid; k < K; k += GEMV_THREADS) {
        float v = ldf(x, k);
        if (g.in_norm_w != nullptr) v = v * rin * (1.0f + g.in_norm_w[k]);
        xs[k] = round_like(v, W);
    }
    float rres = 1.f;
    if (g.mode == CC_GEMV_RESIDUAL && g.res_norm_w != nullptr) {
        float ss = 0.f;
        for (int n = tid; n < N; n += GEMV_THREADS) { const float v = g.res[n]; ss += v * v; }
        rres = 1.0f / sqrtf(block_sum(ss, red) / (float)N + g.eps);
    }
    __syncthreads();
    for (int i = 0; i < GEMV_ROWS / (GEMV_THREADS / 32); ++i) {
        const int n = blockIdx.x * GEMV_ROWS + i * (GEMV_THREADS / 32) + warp;
        if (n >= N) break;
        float acc = row_dot<WT>(W + (size_t)n * K, xs, K, lane);
        if (g.mode == CC_GEMV_GLU) {
            const float up = row_dot<WT>(W + (size_t)(N + n) * K, xs, K, lane);
            if (lane == 0) {
                const float gt = fminf(acc, g.limit);
                const float u = fminf(fmaxf(up, -g.limit), g.limit);
                stf((OT*)g.out, n, gt * (1.0f / (1.0f + expf(-g.slope * gt))) * (u + 1.0f));
            }
            continue;
        }
        if (lane != 0) continue;
        if (g.bias != nullptr) acc += g.bias[n];
        if (g.mode == CC_GEMV_RESIDUAL) {
            float r = g.res[n];
            if (g.res_norm_w != nullptr) r = r * rres * (1.0f + g.res_norm_w[n]);
            acc = g.alpha * r + acc;
        }
        stf((OT*)g.out, n, acc);
    }
}

template <typename WT, typename XT, typename OT>
static int launch_gemv(const CcSeqGemv* g, cudaStream_t st) {
    const size_t smem = sizeof(float) * (size_t)((g->K + 3) & ~3);
    auto kern = gemv_kernel<WT, XT, OT>;
    static SmemLimit limit;
    const cudaError_t e = limit.allow(kern, smem);
    if (e != cudaSuccess) return fail(CC_SEQ_ERR_CUDA, cudaGetErrorString(e));
    kern<<<(g->N + GEMV_ROWS - 1) / GEMV_ROWS, GEMV_THREADS, smem, st>>>(*g);
    return cuda_check("gemv_kernel");
}

// ------------------------------------------------------------------------------------------------ host side
bool attn_tc_serves(const CcSeqAttn* a);              // attn_tc_kernels.cu: bf16 rows on the tensor cores
int attn_tc(const CcSeqAttn* a, cudaStream_t st);

static int check_attn(const CcSeqAttn* a) {
    if (!a || !a->q || !a->k_new || !a->v_new || !a->k_cache || !a->v_cache || !a->pos || !a->input_pos || !a->y)
        return fail(CC_SEQ_ERR_INVALID_ARG, "attention: NULL pointer");
    if (a->T < 1 || a->H < 1 || a->G < 1 || a->H % a->G || a->Dk < 1 || a->Dv < 1 || a->L < 1 || a->window < 0)
        return fail(CC_SEQ_ERR_INVALID_ARG, "attention: bad sizes");
    if (a->Dk > 256 || a->Dv > 256) return fail(CC_SEQ_ERR_UNSUPPORTED_SHAPE, "attention: head sizes above 256");
    if (a->keep_first < 0 || (a->keep_first > 0 && a->L <= a->keep_first) || a->softcap < 0.f || (a->dist_a && !a->dist_b))
        return fail(CC_SEQ_ERR_INVALID_ARG, "attention: bad kept-first count, soft cap or distance penalty");
    // rows that are read only (no fill mask: not a cache) may be fewer than the window: a missing position is not a key
    if (a->window > 0 && a->mask && a->L < a->window + a->keep_first)
        return fail(CC_SEQ_ERR_INVALID_ARG, "attention: cache capacity below the window plus the kept first positions");
    if (a->block < 0 || (a->block > 0 && (a->window > 0 || a->L < a->block)))
        return fail(CC_SEQ_ERR_INVALID_ARG, "attention: a block mask needs a cache of at least one block and no window");
    if (a->sink_mode == CC_SINK_LEARNED && !a->sink) return fail(CC_SEQ_ERR_INVALID_ARG, "attention: sink missing");
    return CC_SEQ_OK;
}

template <typename CT, typename YT, int DV4>
static int launch_chunk(const CcSeqAttn* a, cudaStream_t st) {
    const int Dkp = vec_stride(a->Dk);
    const size_t smem = sizeof(float) * ((size_t)(BQ + BK) * Dkp + (size_t)BK * 64 * DV4 + (size_t)BQ * (BK + 4)) + sizeof(int) * 2 * BK;
    auto kern = attn_chunk_kernel<CT, YT, DV4>;
    static SmemLimit limit;
    const cudaError_t e = limit.allow(kern, smem);
    if (e != cudaSuccess) return fail(CC_SEQ_ERR_CUDA, cudaGetErrorString(e));
    dim3 grid((a->T + BQ - 1) / BQ, a->H);
    kern<<<grid, ATT_THREADS, smem, st>>>(*a);
    return cuda_check("attn_chunk_kernel");
}

template <typename CT, typename YT>
static int dispatch_chunk(const CcSeqAttn* a, cudaStream_t st) {
    const int need = (a->Dv + 63) / 64;
    if (need <= 1) return launch_chunk<CT, YT, 1>(a, st);
    if (need <= 2) return launch_chunk<CT, YT, 2>(a, st);
    if (need <= 3) return launch_chunk<CT, YT, 3>(a, st);
    return launch_chunk<CT, YT, 4>(a, st);
}

template <typename CT, typename YT, int RMAX>
static int launch_decode_r(const CcSeqAttn* a, cudaStream_t st) {
    const int R = a->H / a->G;
    const int vecw = 16 / (int)sizeof(CT);
    const size_t red = (RMAX * vecw <= 64 && a->Dv % vecw == 0 && a->Dv / vecw <= DEC_THREADS) ? (size_t)(DEC_THREADS / (a->Dv / vecw)) * R * a->Dv : 0;
    const size_t smem = sizeof(float) * ((size_t)R * ((a->Dk + 7) & ~7) + (size_t)R * KS + red) + sizeof(int) * KS;
    auto kern = attn_decode_kernel<CT, YT, RMAX>;
    static SmemLimit limit;
    const cudaError_t e = limit.allow(kern, smem);
    if (e != cudaSuccess) return fail(CC_SEQ_ERR_CUDA, cudaGetErrorString(e));
    dim3 grid(decode_max_splits(a->L, attn_reach(*a)), a->G);
    kern<<<grid, DEC_THREADS, smem, st>>>(*a);
    return cuda_check("attn_decode_kernel");
}

// Rows of whole 16-byte vectors on 16-byte boundaries, up to 8 query heads per key/value head, tiles that fit the shared memory
static bool decode_rows_serves(const CcSeqAttn* a) {
    const int size = a->cache_dtype == CC_DT_BF16 ? 2 : 4;
    const uintptr_t all = (uintptr_t)a->k_new | (uintptr_t)a->v_new | (uintptr_t)a->k_cache | (uintptr_t)a->v_cache | (uintptr_t)a->workspace;
    return a->Dk * size % 16 == 0 && a->Dv * size % 16 == 0 && a->Dk * size <= 512 && a->Dv * size <= 512 && (all & 15) == 0 && a->H / a->G <= VD_RMAX;
}

template <typename CT, typename YT, int RMAX>
static int launch_decode_rows(const CcSeqAttn* a, cudaStream_t st) {
    // Two CTAs per SM, one where eight query heads' registers leave room for no more: tiles of 128 keys if one fits a CTA's share of
    // the shared memory (the bf16 rows that come here, of at most 144 columns, always do), of 64 otherwise, and a second buffer for runs
    // of more than one tile only if it fits too.  Runs of 5500 / 12000 / 32000 positions with a second buffer and one CTA per SM
    // where two were counted on, and as it is now, in us: fp32 32 / 8 heads of 128 45.7 / 65.2 / 141.7 and 27.9 / 48.9 / 105.1; fp32 16 / 16
    // of 64 39.3 / 66.2 / 145.8 and 22.0 / 39.3 / 88.6.
    const int vc16 = a->Dv * (int)sizeof(CT) / 16, per_sm = RMAX <= 4 ? 2 : 1;
    const size_t share = (per_sm == 2 ? 111 : 223) * 1024;
    const size_t red = sizeof(float) * (size_t)(VD_THREADS / vc16) * (a->H / a->G) * a->Dv;
    auto bytes = [&](int buffers, int VT) {
        const size_t tiles = (size_t)buffers * VT * (sizeof(CT) * (size_t)(a->Dk + a->Dv) + 16);
        return (tiles > red ? tiles : red) + sizeof(float) * RMAX * (size_t)(a->Dk + VT);
    };
    const int VT = sizeof(CT) == 2 || bytes(1, 128) <= share ? 128 : 64;
    const long long tiles = vd_tiles(a->L, attn_reach(*a), VT);
    const int NS = vd_splits(tiles, a->G, per_sm), buffers = tiles > NS && bytes(2, VT) <= share ? 2 : 1;
    const size_t smem = bytes(buffers, VT);
    auto kern = attn_decode_rows_kernel<CT, YT, RMAX, 128>;
    if constexpr (sizeof(CT) == 4) {
        if (VT == 64) kern = attn_decode_rows_kernel<CT, YT, RMAX, 64>;
    }
    static SmemLimit limits[2];
    const cudaError_t e = limits[VT == 64].allow(kern, smem);
    if (e != cudaSuccess) return fail(CC_SEQ_ERR_CUDA, cudaGetErrorString(e));
    launch_under(kern, dim3(NS, a->G), dim3(VD_THREADS), smem, st, *a, buffers, NS);
    return cuda_check("attn_decode_rows_kernel");
}

// One or two query heads per key head leave most of an MMA's eight columns empty: where narrow rows make the tiles' work count (several
// tiles per CTA), the kernel above is ahead.  us a layer, this kernel and that one, tiles per run in brackets:
//   one query head of 64 + 64, 16 heads: [1] 10.6 / 10.5 and 10.8 / 12.3, [1.8] 17.2 / 16.9, [3.5] 26.6 / 25.5, [5.2] 35.8 / 33.9;
//   of 72 + 72: [1.8] 16.6 / 16.9, [2.6] 22.3 / 22.2, [5.2] 37.6 / 36.7; 32 heads [3.6] 27.8 / 28.8, [10] 63.7 / 62.8; of 80 + 80 [5.2]
//   38.1 / 38.2, of 96 + 96 40.0 / 41.0;
//   two of 32 + 32, 16 key heads: [1.8] 15.8 / 15.8, [2.6] 20.0 / 19.2, [5.2] 33.8 / 31.5; 32 key heads [10] 58.3 / 53.4;
//   of 24 + 40: 32 key heads [3.6] 24.6 / 25.6, [5.2] 33.8 / 34.2, [10] 58.2 / 56.0; of 48 + 32 [5.2] 35.4 / 33.4; of 48 + 48 36.2 / 40.0,
//   of 64 + 64 [2.6] 21.5 / 22.2, [5.2] 37.9 / 37.3;
//   three of 32 + 32, 32 key heads [10] 58.6 / 61.6; four 58.7 / 65.9.
static bool decode_mma_serves(const CcSeqAttn* a) {
    const long long tiles = vd_tiles(a->L, attn_reach(*a), MD_KEYS), runs = vd_splits(tiles, a->G, 2);
    const int R = a->H / a->G, D = a->Dk + a->Dv, widest = a->Dk > a->Dv ? a->Dk : a->Dv;
    if (R == 1 && widest <= 64) return tiles <= runs;
    if (R == 2 && widest <= 32) return tiles <= 2 * runs;
    if ((R == 1 && D <= 144) || (R == 2 && D <= 80)) return tiles <= 4 * runs;
    return true;
}
template <typename YT>
static int launch_decode_mma(const CcSeqAttn* a, cudaStream_t st) {
    const int reach = attn_reach(*a), R = a->H / a->G;
    // Tiles as boxes of one TMA copy per 64 columns where rows are whole boxes wide, by a copy per row otherwise.  8 layers with L2 flushed
    // before, us by rows / by boxes: 32 / 8 heads of 128, 300 positions 90 / 80, 4096 119 / 117, 12000 229 / 215; 16 / 4 at 1000 92 / 84, in a
    // window of 1000 92 / 84.  (The rows asked for in L2 ahead of the wait, by the position that memory held then, gave 104 at 4096 and 203
    // at 12000; but no value is taken from memory there.)
    const long long rows = (long long)a->G * a->L;
    CUtensorMap k_map = {}, v_map = {};
    const bool boxes = a->Dk % 64 == 0 && a->Dv % 64 == 0 && rows >= MD_KEYS && rows < (1ll << 31) - MD_KEYS && map_rows(&k_map, a->k_cache, rows, a->Dk) &&
                       map_rows(&v_map, a->v_cache, rows, a->Dv);
    auto bytes = [&](int buffers) { return md_layout(R, a->Dk, a->Dv, buffers, boxes).total; };
    const size_t half = 111 * 1024, all = 223 * 1024;
    // Two CTAs per SM where a tile fits half of the shared memory, one otherwise (rows of 256 + 256 fit it whole).  8 / 2 heads of
    // 256, 300 / 2000 / 4096 / 8000 positions, us a layer: two CTAs with tiles of 64 keys 12.0 / 16.3 / 27.2 / 29.3, one of 128
    // 13.0 / 13.4 / 17.9 / 25.2.
    const int per_sm = bytes(1) <= half ? 2 : 1;
    const long long tiles = vd_tiles(a->L, reach, MD_KEYS);
    const int NS = vd_splits(tiles, a->G, per_sm), buffers = tiles > NS && bytes(2) <= (per_sm == 2 ? half : all) ? 2 : 1;
    const size_t smem = bytes(buffers);
    auto kern = boxes ? attn_decode_mma_kernel<YT, true> : attn_decode_mma_kernel<YT, false>;
    static SmemLimit limits[2];
    const cudaError_t e = limits[boxes].allow(kern, smem);
    if (e != cudaSuccess) return fail(CC_SEQ_ERR_CUDA, cudaGetErrorString(e));
    launch_under(kern, dim3(NS, a->G), dim3(MD_THREADS), smem, st, *a, buffers, NS, k_map, v_map);
    return cuda_check("attn_decode_mma_kernel");
}

template <typename CT, typename YT>
static int launch_decode(const CcSeqAttn* a, cudaStream_t st) {
    const int R = a->H / a->G;
    if (decode_rows_serves(a)) {
        if constexpr (sizeof(CT) == 2) {
            if (decode_mma_serves(a)) return launch_decode_mma<YT>(a, st);
            return R <= 1 ? launch_decode_rows<CT, YT, 1>(a, st) : launch_decode_rows<CT, YT, 2>(a, st);
        } else {
            if (R <= 1) return launch_decode_rows<CT, YT, 1>(a, st);
            if (R <= 2) return launch_decode_rows<CT, YT, 2>(a, st);
            if (R <= 4) return launch_decode_rows<CT, YT, 4>(a, st);
            return launch_decode_rows<CT, YT, 8>(a, st);
        }
    }
    if (R <= 1) return launch_decode_r<CT, YT, 1>(a, st);
    if (R <= 2) return launch_decode_r<CT, YT, 2>(a, st);
    if (R <= 4) return launch_decode_r<CT, YT, 4>(a, st);
    if (R <= 8) return launch_decode_r<CT, YT, 8>(a, st);
    if (R <= 16) return launch_decode_r<CT, YT, 16>(a, st);
    return fail(CC_SEQ_ERR_UNSUPPORTED_SHAPE, "attention_decode: more than 16 query heads per key/value head");
}

#define CCS_DISPATCH2(d0, d1, CALL)                                                              \
    do {                                                                                         \
        if ((d0) == CC_DT_F32 && (d1) == CC_DT_F32) return CALL(float, float);                   \
        if ((d0) == CC_DT_F32 && (d1) == CC_DT_BF16) return CALL(float, __nv_bfloat16);          \
        if ((d0) == CC_DT_BF16 && (d1) == CC_DT_F32) return CALL(__nv_bfloat16, float);          \
        if ((d0) == CC_DT_BF16 && (d1) == CC_DT_BF16) return CALL(__nv_bfloat16, __nv_bfloat16); \
        return fail(CC_SEQ_ERR_INVALID_ARG, "unknown element type");                             \
    } while (0)

}  // namespace ccs

using namespace ccs;

extern "C" {

int cc_seq_abi_version(void) { return CC_SEQ_ABI_VERSION; }
const char* cc_seq_last_error(void) { return g_err; }

int cc_seq_embed(const int32_t* tokens, const int32_t* input_pos, int32_t* prev_token, const void* embed,
                 const void* bigram, const float* inv_freq, float* x, void* x_act, int32_t T, int32_t E, float scale,
                 int32_t buckets, int32_t mul_prev, int32_t mul_cur, int32_t table_dtype, int32_t act_dtype, void* stream) {
    if (!tokens || !input_pos || !prev_token || !embed || !inv_freq || !x || T < 1 || E < 1 || (bigram && buckets < 1))
        return fail(CC_SEQ_ERR_INVALID_ARG, "embed: bad argument");
    cudaStream_t st = (cudaStream_t)stream;
#define CALL(WT, AT)                                                                                                  \
    (embed_kernel<WT, AT><<<T, 128, 0, st>>>(tokens, input_pos, prev_token, (const WT*)embed, (const WT*)bigram,      \
                                             inv_freq, x, (AT*)x_act, T, E, scale, buckets, mul_prev, mul_cur),       \
     cuda_check("embed_kernel"))
    CCS_DISPATCH2(table_dtype, act_dtype, CALL);
#undef CALL
}

int cc_seq_qkv_prepare(const void* qkv, int32_t in_dtype, const float* bias, const int32_t* input_pos,
                       const float* mix_lambda, const void* v_first, float* q_out, void* k_out, void* v_out,
                       int32_t out_dtype, int32_t T, int32_t H, int32_t G, int32_t Dk, int32_t Dv, float eps,
                       int32_t unit_norm, float gain_coef, int32_t gain_every, void* stream) {
    if (!qkv || !input_pos || !q_out || !k_out || !v_out || T < 1 || H < 1 || G < 1 || Dk < 1 || Dv < 1 ||
        (v_first && !mix_lambda))
        return fail(CC_SEQ_ERR_INVALID_ARG, "qkv_prepare: bad argument");
    cudaStream_t st = (cudaStream_t)stream;
#define CALL(IT, OT)                                                                                                   \
    (qkv_prepare_kernel<IT, OT><<<T, 128, 0, st>>>((const IT*)qkv, bias, input_pos, mix_lambda, (const OT*)v_first,    \
                                                   q_out, (OT*)k_out, (OT*)v_out, T, H, G, Dk, Dv, eps, unit_norm,     \
                                                   gain_coef, gain_every),                                             \
     cuda_check("qkv_prepare_kernel"))
    CCS_DISPATCH2(in_dtype, out_dtype, CALL);
#undef CALL
}

int cc_seq_attention(const CcSeqAttn* a, void* stream) {
    int rc = check_attn(a);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    if (attn_tc_serves(a)) return attn_tc(a, st);
#define CALL(CT, YT) dispatch_chunk<CT, YT>(a, st)
    CCS_DISPATCH2(a->cache_dtype, a->y_dtype, CALL);
#undef CALL
}

uint64_t cc_seq_decode_workspace(int32_t H, int32_t G, int32_t Dv, int32_t L, int32_t window) {
    const uint64_t narrow = (uint64_t)decode_max_splits(L, window), wide = (uint64_t)vd_splits(vd_tiles(L, window, 64), G < 1 ? 1 : G, 2);
    const uint64_t NS = narrow > wide ? narrow : wide;       // either kernel may serve the call
    return sizeof(int) * (uint64_t)((G + 3) & ~3) + sizeof(float) * NS * (uint64_t)H * (2 + (uint64_t)Dv) + 16;
}

int cc_seq_attention_decode(const CcSeqAttn* a, void* stream) {
    int rc = check_attn(a);
    if (rc) return rc;
    if (a->T != 1) return fail(CC_SEQ_ERR_INVALID_ARG, "attention_decode: one token per call");
    if (!a->workspace || a->workspace_bytes < cc_seq_decode_workspace(a->H, a->G, a->Dv, a->L, attn_reach(*a)))
        return fail(CC_SEQ_ERR_INVALID_ARG, "attention_decode: workspace missing or too small");
    cudaStream_t st = (cudaStream_t)stream;
#define CALL(CT, YT) launch_decode<CT, YT>(a, st)
    CCS_DISPATCH2(a->cache_dtype, a->y_dtype, CALL);
#undef CALL
}

int cc_seq_cache_append(const CcSeqAttn* a, void* stream) {
    if (!a || !a->k_new || !a->v_new || !a->k_cache || !a->v_cache || !a->pos || !a->input_pos || a->T < 1 || a->L < 1)
        return fail(CC_SEQ_ERR_INVALID_ARG, "cache_append: bad argument");
    cudaStream_t st = (cudaStream_t)stream;
    if (a->keep_first < 0 || a->L <= a->keep_first) return fail(CC_SEQ_ERR_INVALID_ARG, "cache_append: bad kept-first count");
    const int t_first = (a->keep_first == 0 && a->T > a->L) ? a->T - a->L : 0;   // with kept positions every row's CTA decides
    const int size = a->cache_dtype == CC_DT_BF16 ? 2 : 4, vecs = a->Dk * size % 16 || a->Dv * size % 16 ? 0 : (a->Dk + a->Dv) * size / 16;
    const uintptr_t all = (uintptr_t)a->k_new | (uintptr_t)a->v_new | (uintptr_t)a->k_cache | (uintptr_t)a->v_cache;
    const long long rows = (long long)(a->T - t_first) * a->G;
    if ((a->cache_dtype == CC_DT_F32 || a->cache_dtype == CC_DT_BF16) && vecs > 0 && vecs <= 256 && (all & 15) == 0 && a->G > 0 && rows < (1ll << 30)) {
        const dim3 block(vecs, 256 / vecs);
        auto launch = [&](auto kern, unsigned rows_each) {
            launch_under(kern, dim3((unsigned)((rows + rows_each * block.y - 1) / (rows_each * block.y))), block, 0, st, *a, t_first);
        };
        // A row per thread until that takes 24 CTAs an SM, four from there on.  One / four, us: 8 heads of 128 at 1001 tokens (6.8 CTAs an SM) 3.3
        // / 4.1, at 3000 (20) 4.85 / 5.65, at 4096 (28) 5.95 / 5.75; 64 heads of 64 at 256 (7) 3.2 / 3.6, at 1001 (27) 5.95 / 5.75, at 4096 25.8 / 22.
        const bool one = rows <= (long long)block.y * 148 * 24;
        if (size == 2) one ? launch(cache_append_rows_kernel<__nv_bfloat16, 1>, 1) : launch(cache_append_rows_kernel<__nv_bfloat16, 4>, 4);
        else one ? launch(cache_append_rows_kernel<float, 1>, 1) : launch(cache_append_rows_kernel<float, 4>, 4);
        return cuda_check("cache_append_rows_kernel");
    }
    dim3 grid(a->T - t_first, a->G);
    if (a->cache_dtype == CC_DT_F32) cache_append_kernel<float><<<grid, 64, 0, st>>>(*a, t_first);
    else if (a->cache_dtype == CC_DT_BF16) cache_append_kernel<__nv_bfloat16><<<grid, 64, 0, st>>>(*a, t_first);
    else return fail(CC_SEQ_ERR_INVALID_ARG, "cache_append: unknown element type");
    return cuda_check("cache_append_kernel");
}

int cc_seq_residual_norm(float* x, const void* y, int32_t y_dtype, const float* w, float alpha, float eps, void* x_act,
                         int32_t act_dtype, int32_t T, int32_t E, void* stream) {
    if (!x || !w || T < 1 || E < 1) return fail(CC_SEQ_ERR_INVALID_ARG, "residual_norm: bad argument");
    cudaStream_t st = (cudaStream_t)stream;
#define CALL(YT, AT)                                                                                                \
    (residual_norm_kernel<YT, AT><<<T, 256, 0, st>>>(x, (const YT*)y, w, alpha, eps, (AT*)x_act, E),                \
     cuda_check("residual_norm_kernel"))
    CCS_DISPATCH2(y_dtype, act_dtype, CALL);
#undef CALL
}

int cc_seq_clamped_glu(const void* gu, void* out, int32_t io_dtype, int32_t out_dtype, float limit, float slope,
                       int32_t T, int32_t F, void* stream) {
    if (!gu || !out || T < 1 || F < 1) return fail(CC_SEQ_ERR_INVALID_ARG, "clamped_glu: bad argument");
    cudaStream_t st = (cudaStream_t)stream;
    const size_t n = (size_t)T * F;
    const int blocks = (int)((n + 255) / 256 < 148 * 16 ? (n + 255) / 256 : 148 * 16);
#define CALL(IT, OT)                                                                                    \
    (clamped_glu_kernel<IT, OT><<<blocks, 256, 0, st>>>((const IT*)gu, (OT*)out, limit, slope, T, F),   \
     cuda_check("clamped_glu_kernel"))
    CCS_DISPATCH2(io_dtype, out_dtype, CALL);
#undef CALL
}

int cc_seq_gemv(const CcSeqGemv* g, void* stream) {
    if (!g || !g->x || !g->W || !g->out || g->N < 1 || g->K < 1 || (g->mode == CC_GEMV_RESIDUAL && !g->res) ||
        g->mode < CC_GEMV_PLAIN || g->mode > CC_GEMV_GLU)
        return fail(CC_SEQ_ERR_INVALID_ARG, "gemv: bad argument");
    if (g->in_norm_w && g->x_dtype != CC_DT_F32) return fail(CC_SEQ_ERR_INVALID_ARG, "gemv: a normed input is an fp32 sum");
    if (g->mode != CC_GEMV_GLU && g->out_dtype != CC_DT_F32) return fail(CC_SEQ_ERR_INVALID_ARG, "gemv: fp32 output expected");
    if ((size_t)g->K * 4 > 200 * 1024) return fail(CC_SEQ_ERR_UNSUPPORTED_SHAPE, "gemv: input longer than 51200");
    cudaStream_t st = (cudaStream_t)stream;
    const bool wb = g->w_dtype == CC_DT_BF16, xb = g->x_dtype == CC_DT_BF16, ob = g->out_dtype == CC_DT_BF16;
    if (wb && xb && ob) return launch_gemv<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16>(g, st);
    if (wb && xb && !ob) return launch_gemv<__nv_bfloat16, __nv_bfloat16, float>(g, st);
    if (wb && !xb && ob) return launch_gemv<__nv_bfloat16, float, __nv_bfloat16>(g, st);
    if (wb && !xb && !ob) return launch_gemv<__nv_bfloat16, float, float>(g, st);
    if (!wb && !xb && !ob) return launch_gemv<float, float, float>(g, st);
    return fail(CC_SEQ_ERR_INVALID_ARG, "gemv: unsupported combination of element types");
}

}  // extern "C"
