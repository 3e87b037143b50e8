// attn_tc_kernels.cu -- attention of a prompt portion over position-addressed bf16 rows on the tensor cores
// (cc_seq_attention for bf16 caches; the fp32 FMA kernel of seq_kernels.cu serves fp32 caches and odd row widths).
//
// Scores and softmax weights stay 32-bit: a bf16 x bf16 product is exact in fp32, so an fp32 operand is cut into
// three bf16 parts that add up to it EXACTLY (truncation takes 8 of the 24 significant bits at a time) and multiplied
// part by part: S = (q1 + q2 + q3) K^T and (p1 + p2 + p3) V, smallest part first.  The tensor core truncates where an FMA
// rounds, so an accumulator lives for one tile of 128 keys only; the sum over the tiles is an fp32 FMA in registers
// that also applies the softmax's rescaling.
//
// Bound: tensor pipe and the shared memory it reads: 2 x 24 MMAs of 128 x 128 x 16 per 128 x 128 scores at head size 128,
// 107 cycles each with both operands in shared memory (scores) and 74 with the weights in tensor memory (values) by stamps of the
// SM's clock, where the pipe itself needs 64 (ncu: tensor pipe 49 % active, issue slots 38 %); together 4350 of the
// 4400 to 5000 cycles that a tile takes (long prompts / short ones); the other pipes need ~10 instructions per score beside them.  Layout that
// follows: the query parts stay in shared memory (96 KB) and the weight parts go to tensor memory, over the scores they came
// from, as the A operand.  Sixteen warps of softmax, four threads per row.
//
// Measured on a B200: 4096 tokens, 32 / 8 heads of 128, learned sinks, 6.17 ms on the FMA kernel -> 0.449 ms (306 TFLOP/s of
// the attention, 3 times that on the tensor pipe; eight warps of softmax 0.012 ms more); 1001 tokens behind 3333 in a window of 1024,
// 16 / 4 heads, 0.435 ms -> 0.070 ms.  Error of fp32 outputs against 64 bits on the same inputs, here / on the FMA kernel: scores of a
// few units 0.2-0.6e-6 / 0.3-1.7e-6; of hundreds 0.9-1.8e-6 / 2.3-6.3e-6; all of a row's scores moved by 300 1.3-3.0e-5 / 3.7-7.0e-5, by
// 8000 0.6-1.3e-3 / 1.1-2.2e-3 (what their rounding to fp32 leaves).  Larger here only where one key takes all the weight, 0.7e-7.
// Descriptors formed ahead of the loop changed nothing.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../../include/cc_b200_seq.h"
#include "launch.cuh"

namespace ccs {

int fail(int code, const char* msg);
int cuda_check(const char* where);

namespace {

typedef __nv_bfloat16 bf16;

constexpr int BM = 128, BN = 128;             // score tile: rows = (query, query head of the group) pairs, keys
constexpr int TILE_BYTES = 128 * 128;         // 128 rows x 64 bf16, 128-byte swizzled
constexpr int SOFT_THREADS = 512;             // four threads per row (32 keys and a quarter of the value columns each)
constexpr int THREADS = SOFT_THREADS + 128;   // + MMA warp, K warp, V warp, one warp without work
constexpr int RING = 8;                       // tiles in flight, for the marks of their live keys
constexpr int TM_O = 256, TM_P3 = 384, TM_COLS = 512;   // tensor memory: scores 2 x 128 | tile result 128 | third part 2 x 64
constexpr float LOG2E = 1.4426950408889634f;
constexpr uint32_t WAIT_LIMIT = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done != 0;
}
// Bounded: a wait that runs out raises `failed`; every later wait of the CTA then gives up at once, the kernel runs to its
// end and stores NaN.
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, volatile int* failed) {
    if (mbar_try(bar, parity)) return;
    for (uint32_t n = 0; !mbar_try(bar, parity); ++n)
        if (n >= WAIT_LIMIT || *failed) { *failed = 1; return; }
}
// What was started is waited for also after another wait has run out: its shared and its tensor memory go to another CTA.
__device__ __forceinline__ void mbar_wait_out(uint32_t bar, uint32_t parity) {
    for (uint32_t n = 0; n < WAIT_LIMIT && !mbar_try(bar, parity); ++n) {}
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async;" ::: "memory"); }
// shared-memory matrix descriptor, 128-byte swizzle, descriptor version 1 (sm_100)
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) |
           (1ull << 46) | (2ull << 61);
}
// bf16 x bf16 -> fp32, M = 128, A K-major, B K-major or MN-major
__device__ __forceinline__ uint32_t idesc(int N, bool b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
}
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t id, uint32_t acc) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                 ::"r"(d), "l"(a), "l"(b), "r"(id), "r"(acc) : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t id, uint32_t acc) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
                 ::"r"(d), "r"(a), "l"(b), "r"(id), "r"(acc) : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 32 lanes x 32 consecutive columns -> registers; the caller waits with tmem_wait_ld
__device__ __forceinline__ void tmem_ld32(uint32_t t, float* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]),
          "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]), "=f"(v[17]), "=f"(v[18]),
          "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]), "=f"(v[23]), "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]),
          "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
        : "r"(t) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t t, float* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]),
          "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15])
        : "r"(t) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st16(uint32_t t, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n"
        ::"r"(t), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
          "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool have) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(have ? 16 : 0) : "memory");
}
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// pairs of fp32 values: one instruction for two additions or multiply-adds, each rounded as the scalar one
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
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// the high halves of two fp32 words as a bf16 pair (a in the low half)
__device__ __forceinline__ uint32_t high_pair(float a, float b) { return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632); }
// minus the part of x that a bf16 holds
__device__ __forceinline__ float minus_high(float x) { return __uint_as_float((__float_as_uint(x) & 0xffff0000u) ^ 0x80000000u); }
// two fp32 values as three bf16 pairs whose sums are the values
__device__ __forceinline__ void split3(float a, float b, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    p1 = high_pair(a, b);
    unpair(add2(pair(a, b), pair(minus_high(a), minus_high(b))), a, b);
    p2 = high_pair(a, b);
    unpair(add2(pair(a, b), pair(minus_high(a), minus_high(b))), a, b);
    p3 = high_pair(a, b);
}
__device__ __forceinline__ void st_out(float* p, size_t i, float v) { p[i] = v; }
__device__ __forceinline__ void st_out(bf16* p, size_t i, float v) { p[i] = __float2bfloat16_rn(v); }

struct Keys {   // the keys of one CTA in order: the kept first positions below the window, then j_lo, j_lo + 1, ...
    int p0, kx, j_lo, n;
    __device__ __forceinline__ int at(int u) const { return u < kx ? u : j_lo + (u - kx); }
};

// Where the 128 keys of one tile come from.  Positions below p0 sit in cache slots (the kept first ones in slots of their
// own, the others in a ring), the others are rows of the portion; both are runs of equally spaced rows.
struct TileRows {
    int j0;          // position of key 0, when the tile lies beside the kept first positions
    int ring, r0;    // ring length, and place of j0 in it
    uint32_t live[4];
    bool run;        // all live keys are the tile's first ones and lie in one run of rows
    size_t first;    // ... that starts here (row), in the portion or in the cache
    bool fresh;
};

__device__ __forceinline__ int slot_in(const CcSeqAttn& a, const Keys& ks, const TileRows& t, int u0, int row) {
    const int u = u0 + row;
    if (u < ks.kx) return u;
    if (u0 < ks.kx) {
        const int j = ks.at(u);
        return j < a.keep_first ? j : a.keep_first + (j - a.keep_first) % t.ring;
    }
    if (t.j0 + row < a.keep_first) return t.j0 + row;
    int r = t.r0 + row;
    if (t.r0 < 0) r = (t.j0 + row - a.keep_first) % t.ring;        // a short ring, or the tile straddles the kept positions
    else if (r >= t.ring) r -= t.ring;
    return a.keep_first + r;
}

// The 32 lanes look the tile's 128 keys up: a key is live when it is within the portion, or its slot holds its position.
__device__ __forceinline__ TileRows look_up(const CcSeqAttn& a, const Keys& ks, int n, int lane) {
    TileRows t;
    const int u0 = n * BN;
    t.ring = a.L - a.keep_first;
    t.j0 = ks.at(u0);
    t.r0 = t.ring >= BN && t.j0 >= a.keep_first ? (t.j0 - a.keep_first) % t.ring : -1;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int row = 32 * q + lane, u = u0 + row, j = ks.at(u);
        bool live = u < ks.n;
        if (live && j < ks.p0) live = a.pos[slot_in(a, ks, t, u0, row)] == j;
        t.live[q] = __ballot_sync(0xffffffffu, live);
    }
    const int rows = min(BN, ks.n - u0), j1 = t.j0 + rows - 1;
    uint32_t want[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) want[q] = rows >= 32 * q + 32 ? 0xffffffffu : rows <= 32 * q ? 0u : (1u << (rows - 32 * q)) - 1u;
    const bool all = t.live[0] == want[0] && t.live[1] == want[1] && t.live[2] == want[2] && t.live[3] == want[3];
    t.fresh = t.j0 >= ks.p0;
    t.run = all && u0 >= ks.kx && (t.fresh || (j1 < ks.p0 && t.r0 >= 0 && t.r0 + rows <= t.ring));
    t.first = t.fresh ? (size_t)(t.j0 - ks.p0) * a.G : (size_t)(a.keep_first + t.r0);
    return t;
}

// One warp copies the rows of a tile into the swizzled layout: lane = 16-byte column lane % 16 of rows lane / 16, + 2, + 4, ...
// Dead rows and columns up to the padded width become zero.  A tile that is one run of rows costs three instructions per
// copy (a row lookup per copy made this warp the slowest part of the kernel: 0.67 against 0.49 ms for 4096 tokens).
__device__ __forceinline__ void copy_tile(uint32_t dst, const CcSeqAttn& a, const Keys& ks, const TileRows& t, int n, int g, int width,
                                          const void* cache, const void* fresh, int chunks, int chunks_padded, int lane) {
    const int c = lane & 15, hi = lane >> 4;
    if (c >= chunks_padded) return;
    const bool col = c < chunks;
    const bf16* const cb = (const bf16*)cache + (size_t)g * a.L * width + 8 * c;
    const bf16* const fb = (const bf16*)fresh + (size_t)g * width + 8 * c;
    const uint32_t at = dst + (c >> 3) * TILE_BYTES + hi * 128;
    uint32_t sw[4];   // row 2 i + hi: the swizzle repeats every four i
#pragma unroll
    for (int i = 0; i < 4; ++i) sw[i] = at + ((((c & 7) ^ (2 * i + hi)) & 7) << 4);
    if (t.run) {
        const int step = t.fresh ? a.G * width : width;
        const bf16* src = (t.fresh ? fb : cb) + t.first * width + (size_t)hi * step;
        const int rows = min(BN, ks.n - n * BN);
        if (rows == BN && col) {
#pragma unroll 16
            for (int i = 0; i < 64; ++i, src += 2 * step) cp_async16(sw[i & 3] + 256 * i, src, true);
        } else {
#pragma unroll 4
            for (int i = 0; i < 64; ++i, src += 2 * step) {
                const bool have = col && 2 * i + hi < rows;
                cp_async16(sw[i & 3] + 256 * i, have ? (const void*)src : fresh, have);
            }
        }
        return;
    }
    const int u0 = n * BN;
    if (u0 >= ks.kx && (t.fresh || t.r0 >= 0)) {
        // up to three runs: slots up to the ring's end, slots from its start, rows of the portion
        const int nc = max(0, min(BN, ks.p0 - t.j0)), w1 = min(nc, t.ring - t.r0), fresh_step = a.G * width;
        const bf16* const r1 = cb + (ptrdiff_t)(a.keep_first + t.r0) * width;
        const bf16* const r2 = r1 - (ptrdiff_t)t.ring * width;
        const bf16* const r3 = fb + (ptrdiff_t)(t.j0 - ks.p0) * fresh_step;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t live = t.live[q] >> hi;
#pragma unroll 8
            for (int i = 0; i < 16; ++i) {
                const int row = 32 * q + 2 * i + hi;
                const bool have = col && (live >> (2 * i) & 1u);
                const bf16* src = row < nc ? (row < w1 ? r1 : r2) + row * width : r3 + (ptrdiff_t)row * fresh_step;
                cp_async16(sw[i & 3] + 256 * (16 * q + i), have ? (const void*)src : fresh, have);
            }
        }
        return;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint32_t live = t.live[q] >> hi;
#pragma unroll 1
        for (int i = 0; i < 16; ++i) {
            const int row = 32 * q + 2 * i + hi, j = ks.at(u0 + row);
            const bool have = col && (live >> (2 * i) & 1u);
            const bf16* src = (const bf16*)fresh;
            if (have) src = j >= ks.p0 ? fb + (size_t)(j - ks.p0) * a.G * width : cb + (size_t)slot_in(a, ks, t, u0, row) * width;
            cp_async16(sw[i & 3] + 256 * (16 * q + i), src, have);
        }
    }
}

struct Small {
    uint64_t bars[13];          // k full[2], v full[2], scores[2], weights[2], product[2], result read, queries, everything done
    uint32_t tmem;
    int failed;
    float max[4][BM];           // row maxima over a quarter of a tile's keys; the sums' meeting place at the end
    uint32_t live[RING][BN / 32];   // bit of key u % 32 of the tile: a slot holds it
    uint32_t redo[BM / 32];         // bit of row u % 32: its sums are not finite
};

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ float shaped(const CcSeqAttn& a, float x, int h, int dist) {
    if (a.softcap > 0.f) x = a.softcap * tanhf(x / a.softcap);
    if (a.dist_a != nullptr) x -= a.dist_a[h] * log1pf(a.dist_b[h] * (float)max(0, dist));
    return x;
}

// One (query, head) row again by a warp, key by key on the FMA pipe, for rows whose sums above are not finite: three parts of an
// operand times an infinity give NaN where the operand itself gives an infinity, and a weight of zero times a value row that
// this row does not see gives NaN too.  Here a key that is not seen takes no part and operands are whole, so a score of minus
// infinity is a weight of zero and an infinity stays one.  Ends as soon as the denominator is NaN: then everything is.
template <typename YT, bool SHAPED>
__device__ __forceinline__ void row_again(const CcSeqAttn& a, const Keys& ks, int t, int h, int g, int lane) {
    const int i = ks.p0 + t, Dk = a.Dk, Dv = a.Dv, ring = a.L - a.keep_first, i_block = a.block > 0 ? (i / a.block) * a.block : 0;
    const float* const q = a.q + ((size_t)t * a.H + h) * Dk;
    float m = -INFINITY, l = 0.f, o[4] = {0.f, 0.f, 0.f, 0.f};      // value columns 4 lane .. 4 lane + 3
    if (a.sink_mode == CC_SINK_LEARNED) { m = a.sink[h]; l = 1.f; }
    else if (a.sink_mode == CC_SINK_ZERO) { m = 0.f; l = 1.f; }
#pragma unroll 1
    for (int u0 = 0; u0 < ks.n && l == l; u0 += 32) {
        const int j = ks.at(u0 + lane), slot = j < a.keep_first ? j : a.keep_first + (j - a.keep_first) % ring;
        const bool seen = u0 + lane < ks.n && j <= i && (a.window == 0 || i - j < a.window || j < a.keep_first) && j >= i_block && (j >= ks.p0 || a.pos[slot] == j);
        const size_t row = j >= ks.p0 ? (size_t)(j - ks.p0) * a.G + g : (size_t)g * a.L + slot;
        float s = -INFINITY;
        if (seen) {
            const bf16* const k = (const bf16*)(j >= ks.p0 ? a.k_new : a.k_cache) + row * Dk;
            s = 0.f;
#pragma unroll 4
            for (int d = 0; d < Dk; d += 8) {      // rows are whole 16-byte vectors
                const uint4 u = *reinterpret_cast<const uint4*>(k + d);
                const bf16* const e = reinterpret_cast<const bf16*>(&u);
                float qv[8];
                *reinterpret_cast<float4*>(qv) = *reinterpret_cast<const float4*>(q + d);
                *reinterpret_cast<float4*>(qv + 4) = *reinterpret_cast<const float4*>(q + d + 4);
#pragma unroll
                for (int x = 0; x < 8; ++x) s = fmaf(qv[x], __bfloat162float(e[x]), s);
            }
            s *= a.scale;
            if (SHAPED) s = shaped(a, s, h, i - j);
        }
        const float m_new = fmaxf(m, warp_max(s)), corr = m == -INFINITY ? 0.f : expf(m - m_new), w = s == -INFINITY ? 0.f : expf(s - m_new);
        l = l * corr + warp_sum(w);
        m = m_new;
#pragma unroll
        for (int c = 0; c < 4; ++c) o[c] *= corr;
        const uint32_t all = __ballot_sync(0xffffffffu, seen);
        const unsigned long long mine = (unsigned long long)((const bf16*)(j >= ks.p0 ? a.v_new : a.v_cache) + row * Dv);
#pragma unroll 8
        for (int k = 0; k < 32; ++k) {
            const float wk = __shfl_sync(0xffffffffu, w, k);
            const bf16* const vr = (const bf16*)__shfl_sync(0xffffffffu, mine, k);
            uint2 u = make_uint2(0u, 0u);      // a key that is not seen: zero times zero
            if ((all >> k & 1u) && 4 * lane < Dv) u = *reinterpret_cast<const uint2*>(vr + 4 * lane);
            const bf16* const v = reinterpret_cast<const bf16*>(&u);
#pragma unroll
            for (int c = 0; c < 4; ++c) o[c] = fmaf(wk, __bfloat162float(v[c]), o[c]);
        }
    }
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    if (4 * lane < Dv)
#pragma unroll
        for (int c = 0; c < 4; ++c) st_out((YT*)a.y + ((size_t)t * a.H + h) * Dv, 4 * lane + c, l == l ? o[c] * inv : NAN);
}

// NO: value columns per thread (a quarter of the padded value width).  SHAPED: soft cap, distance penalty, or a scale that is not
// positive.
template <typename YT, int NO, bool SHAPED>
__global__ void __launch_bounds__(THREADS, 1) attn_tc_kernel(const CcSeqAttn a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];   // operand tiles, then Small

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int R = a.H / a.G, Dk = a.Dk, Dv = a.Dv;
    const int n_rows = a.T * R, n_tiles = (n_rows + BM - 1) / BM;
    const int g = blockIdx.x % a.G, tile = n_tiles - 1 - (int)blockIdx.x / a.G;   // longest rows first
    const int f0 = tile * BM, f1 = min(f0 + BM, n_rows) - 1;
    const int dh = (Dk + 63) / 64, ksteps = (Dk + 15) / 16;
    const uint32_t q_part = dh * TILE_BYTES, sQ = smem_u32(smem_raw), sK = sQ + 3 * q_part, sV = sK + 2 * q_part;
    const uint32_t v_tile = ((Dv + 63) / 64) * TILE_BYTES;
    Small& sm = *reinterpret_cast<Small*>(smem_raw + 5 * q_part + 2 * v_tile);
    volatile int* const failed = &sm.failed;
    const uint32_t bar = smem_u32(sm.bars);
    const uint32_t K_FULL = bar, V_FULL = bar + 16, S_DONE = bar + 32, P_DONE = bar + 48, PV_DONE = bar + 64, O_READ = bar + 80, Q_FULL = bar + 88, DONE = bar + 96;

    if (tid < BM / 32) sm.redo[tid] = 0;
    if (tid == 0) {
        *failed = 0;
        for (int b = 0; b < 2; ++b) {
            mbar_init(K_FULL + 8 * b, 32);
            mbar_init(V_FULL + 8 * b, 32);
            mbar_init(S_DONE + 8 * b, 1);
            mbar_init(P_DONE + 8 * b, SOFT_THREADS / 32);
            mbar_init(PV_DONE + 8 * b, 1);
        }
        mbar_init(O_READ, SOFT_THREADS / 32);
        mbar_init(Q_FULL, SOFT_THREADS);
        mbar_init(DONE, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem)), "r"(TM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = sm.tmem;
    const int q_chunks = 2 * ksteps;
    pdl_wait_release();

    Keys ks;
    ks.p0 = a.input_pos[0];
    const int i_first = ks.p0 + f0 / R, i_last = ks.p0 + f1 / R;
    ks.j_lo = a.block > 0 ? (i_first / a.block) * a.block : (a.window > 0 ? max(0, i_first - a.window + 1) : 0);
    ks.kx = a.window > 0 ? min(a.keep_first, ks.j_lo) : 0;
    ks.n = ks.kx + (i_last - ks.j_lo + 1);
    const int N = (ks.n + BN - 1) / BN;

    if (warp >= SOFT_THREADS / 32) {
        // 640 threads x 96 registers at launch = 61440 >= 512 x 104 + 128 x 56
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp == SOFT_THREADS / 32) {
            if (lane == 0) {
                const uint32_t id_s = idesc(BN, false), id_v = idesc((Dv + 15) & ~15, true);
                auto scores = [&](int n) {
                    const int b = n & 1;
                    mbar_wait(K_FULL + 8 * b, (n >> 1) & 1, failed);
                    fence_after();
                    uint32_t acc = 0;
                    for (int s = 2; s >= 0; --s)
                        for (int k = 0; k < ksteps; ++k, acc = 1) {
                            const uint32_t off = (k >> 2) * TILE_BYTES + (k & 3) * 32;
                            mma_ss(tmem + b * BN, smem_desc(sQ + s * q_part + off, 16, 1024), smem_desc(sK + b * q_part + off, 16, 1024), id_s, acc);
                        }
                    mma_commit(S_DONE + 8 * b);
                };
                mbar_wait(Q_FULL, 0, failed);
                scores(0);
                for (int n = 0; n < N; ++n) {
                    const int b = n & 1;
                    if (n + 1 < N) scores(n + 1);   // its columns held the weights of tile n - 1, whose product is ahead of it in the pipe
                    mbar_wait(P_DONE + 8 * b, (n >> 1) & 1, failed);
                    mbar_wait(V_FULL + 8 * b, (n >> 1) & 1, failed);
                    if (n > 0) mbar_wait(O_READ, (n - 1) & 1, failed);
                    fence_after();
                    uint32_t acc = 0;
                    for (int s = 2; s >= 0; --s)
#pragma unroll
                        for (int k = 0; k < BN / 16; ++k, acc = 1) {
                            const uint32_t part = k >> 1, kk = (k & 1) * 8;      // 16 keys of a thread's 32
                            const uint32_t at = s < 2 ? tmem + b * BN + part * 32 + s * 16 + kk : tmem + TM_P3 + b * 64 + part * 16 + kk;
                            mma_ts(tmem + TM_O, at, smem_desc(sV + b * v_tile + k * 2048, TILE_BYTES, 1024), id_v, acc);
                        }
                    mma_commit(PV_DONE + 8 * b);
                }
                mma_commit(DONE);
                mbar_wait_out(DONE, 0);
            }
            __syncwarp();
        } else if (warp == SOFT_THREADS / 32 + 1) {
            for (int n = 0; n < N; ++n) {
                const int b = n & 1;
                const TileRows t = look_up(a, ks, n, lane);
                // buffer b is free when the scores of tile n - 2 are done; by then every thread has passed tile n - 4
                if (n >= 2) mbar_wait(S_DONE + 8 * b, ((n - 2) >> 1) & 1, failed);
                copy_tile(sK + b * q_part, a, ks, t, n, g, Dk, a.k_cache, a.k_new, Dk / 8, q_chunks, lane);
                if (lane < 4) sm.live[n & (RING - 1)][lane] = lane == 0 ? t.live[0] : lane == 1 ? t.live[1] : lane == 2 ? t.live[2] : t.live[3];
                asm volatile("cp.async.wait_all;" ::: "memory");
                fence_async();
                mbar_arrive(K_FULL + 8 * b);
            }
        } else if (warp == SOFT_THREADS / 32 + 2) {
            for (int n = 0; n < N; ++n) {
                const int b = n & 1;
                const TileRows t = look_up(a, ks, n, lane);
                if (n >= 2) mbar_wait(PV_DONE + 8 * b, ((n - 2) >> 1) & 1, failed);
                copy_tile(sV + b * v_tile, a, ks, t, n, g, Dv, a.v_cache, a.v_new, Dv / 8, 2 * ((Dv + 15) / 16), lane);
                asm volatile("cp.async.wait_all;" ::: "memory");
                fence_async();
                mbar_arrive(V_FULL + 8 * b);
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
        // the query rows in three parts; columns up to the padded width and rows past the end are zero
        for (int idx = tid; idx < BM * q_chunks; idx += SOFT_THREADS) {
            const int row = idx / q_chunks, c = idx - row * q_chunks, flat = f0 + row;
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v[e] = 0.f;
            if (flat < n_rows && 8 * c < Dk) {
                const int t = flat / R;
                const float4* src = reinterpret_cast<const float4*>(a.q + ((size_t)t * a.H + g * R + (flat - t * R)) * Dk + 8 * c);
                *reinterpret_cast<float4*>(v) = src[0];
                *reinterpret_cast<float4*>(v + 4) = src[1];
            }
            uint32_t w[3][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) split3(v[2 * e], v[2 * e + 1], w[0][e], w[1][e], w[2][e]);
            uint8_t* dst = smem_raw + (c >> 3) * TILE_BYTES + row * 128 + (((c & 7) ^ (row & 7)) << 4);
#pragma unroll
            for (int s = 0; s < 3; ++s) *reinterpret_cast<uint4*>(dst + s * q_part) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
        }
        fence_async();
        mbar_arrive(Q_FULL);
        const int part = warp >> 2, quarter = warp & 3, row = quarter * 32 + lane, flat = min(f0 + row, n_rows - 1);
        const int t = flat / R, h = g * R + (flat - t * R), i = ks.p0 + t;
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        const float c2 = SHAPED ? LOG2E : a.scale * LOG2E;
        const float dist_a = SHAPED && a.dist_a != nullptr ? a.dist_a[h] : 0.f, dist_b = SHAPED && a.dist_a != nullptr ? a.dist_b[h] : 0.f;
        float m = -INFINITY, l = 0.f, corr_before = 0.f;
        if (a.sink_mode == CC_SINK_LEARNED) { m = __fmul_rn(a.sink[h], LOG2E); l = part == 0 ? ex2(fmaf(a.sink[h], LOG2E, -m)) : 0.f; }
        else if (a.sink_mode == CC_SINK_ZERO) { m = 0.f; l = part == 0 ? 1.f : 0.f; }
        f32x2 O[NO / 2];
#pragma unroll
        for (int c = 0; c < NO / 2; ++c) O[c] = 0ull;
        auto add_result = [&](int n, float corr) {   // O = O corr + the product of tile n
            mbar_wait(PV_DONE + 8 * (n & 1), (n >> 1) & 1, failed);
            fence_after();
            float v[NO];
            if constexpr (NO == 32) tmem_ld32(tmem + lanes + TM_O + part * NO, v);
            else tmem_ld16(tmem + lanes + TM_O + part * NO, v);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < NO; c += 2) O[c / 2] = fma2(O[c / 2], pair(corr, corr), pair(v[c], v[c + 1]));
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(O_READ);
        };
        for (int n = 0; n < N; ++n) {
            const int b = n & 1;
            const int u0 = n * BN, u1 = u0 + BN - 1;
            // whether every row of the tile sees every key of it (only where the whole tile comes from beside the kept rows)
            const int j0 = ks.at(u0), j1 = ks.at(min(u1, ks.n - 1));
            const bool plain = u1 < ks.n && u0 >= ks.kx && j1 <= i_first && (a.window == 0 || i_last - j0 < a.window) &&
                               (a.block == 0 || j0 >= (i_last / a.block) * a.block);
            mbar_wait(S_DONE + 8 * b, (n >> 1) & 1, failed);
            fence_after();
            float s[32];
            tmem_ld32(tmem + lanes + b * BN + part * 32, s);
            tmem_wait_ld();
            const uint32_t live = sm.live[n & (RING - 1)][part];
            if constexpr (SHAPED) {
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    float x = s[c] * a.scale;
                    if (a.softcap > 0.f) x = a.softcap * tanhf(x / a.softcap);
                    if (a.dist_a != nullptr) x -= dist_a * log1pf(dist_b * (float)max(0, i - ks.at(u0 + part * 32 + c)));
                    s[c] = x;
                }
            }
            if (!(plain && live == 0xffffffffu)) {
                const int i_block = a.block > 0 ? (i / a.block) * a.block : 0, u = u0 + part * 32;
#pragma unroll
                for (int c = 0; c < 32; ++c) {
                    const int j = ks.at(u + c);
                    const bool ok = (live >> c & 1u) && j <= i && (a.window == 0 || i - j < a.window || j < a.keep_first) &&
                                    j >= i_block;
                    if (!ok) s[c] = -INFINITY;
                }
            }
            float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
            for (int c = 4; c < 32; ++c) mx[c & 3] = fmaxf(mx[c & 3], s[c]);
            // The maximum itself, in fp32: the exponents below reach from 0 down, so a bound far above it would flush every
            // weight.  The four warps of these rows meet twice per tile, as the maxima of the tile before have to be read:
            // arriving there and waiting here are apart.
            if (n > 0) asm volatile("bar.sync %0, 256;" ::"r"(quarter + 6) : "memory");
            sm.max[part][row] = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * c2;
            asm volatile("bar.sync %0, 128;" ::"r"(quarter + 1) : "memory");
            float m_new = m;
#pragma unroll
            for (int q = 0; q < 4; ++q) m_new = fmaxf(m_new, sm.max[q][row]);
            if (n + 1 < N) asm volatile("bar.arrive %0, 256;" ::"r"(quarter + 6) : "memory");
            const float ms = m_new == -INFINITY ? 0.f : m_new;
            const float corr = m == -INFINITY ? 0.f : ex2(m - ms);
            m = m_new;
            const f32x2 cc = pair(c2, c2), mm = pair(-ms, -ms);
            f32x2 sum[2] = {0ull, 0ull};
            uint32_t p1[16], p2[16], p3[16];
#pragma unroll
            for (int c = 0; c < 32; c += 2) {
                float x, y;
                unpair(fma2(pair(s[c], s[c + 1]), cc, mm), x, y);
                x = ex2(x);
                y = ex2(y);
                sum[(c >> 1) & 1] = add2(sum[(c >> 1) & 1], pair(x, y));
                split3(x, y, p1[c >> 1], p2[c >> 1], p3[c >> 1]);
            }
            const uint32_t at = tmem + lanes + b * BN + part * 32;   // 32 keys = 16 columns a part, over scores that are in registers
            tmem_st16(at, p1);
            tmem_st16(at + 16, p2);
            tmem_st16(tmem + lanes + TM_P3 + b * 64 + part * 16, p3);
            float sum_x, sum_y;
            unpair(add2(sum[0], sum[1]), sum_x, sum_y);
            l = fmaf(l, corr, sum_x + sum_y);
            tmem_wait_st();
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(P_DONE + 8 * b);
            if (n > 0) add_result(n - 1, corr_before);
            corr_before = corr;
        }
        add_result(N - 1, corr_before);
        asm volatile("bar.sync %0, 128;" ::"r"(quarter + 1) : "memory");      // the last maxima of these rows have been read
        sm.max[part][row] = l;
        asm volatile("bar.sync %0, 128;" ::"r"(quarter + 1) : "memory");
        l = (sm.max[0][row] + sm.max[1][row]) + (sm.max[2][row] + sm.max[3][row]);
        if (f0 + row < n_rows) {
            float inv = l > 0.f ? 1.0f / l : 0.f, zero = 0.f * l;      // 0, or NaN once something is not finite
            if (*failed) inv = NAN;
            YT* y = (YT*)a.y + ((size_t)t * a.H + h) * Dv + part * NO;
            const int have = min(NO, Dv - part * NO);
            // rows are multiples of 8 elements wide: 16-byte stores
#pragma unroll
            for (int c = 0; c < NO; c += 8) {
                if (c < have) {
                    __align__(16) YT w[8];
#pragma unroll
                    for (int e = 0; e < 8; e += 2) {
                        float x, x1;
                        unpair(O[(c + e) / 2], x, x1);
                        zero = fmaf(0.f, x, fmaf(0.f, x1, zero));
                        st_out(w, e, x * inv);
                        st_out(w, e + 1, x1 * inv);
                    }
#pragma unroll
                    for (int v = 0; v < (int)sizeof(YT) / 2; ++v) reinterpret_cast<uint4*>(y + c)[v] = reinterpret_cast<const uint4*>(w)[v];
                }
            }
            if (zero != 0.f) atomicOr(&sm.redo[quarter], 1u << lane);
        }
        // the marks of these rows are there, and what row_again writes over is written
        asm volatile("bar.sync %0, 128;" ::"r"(quarter + 1) : "memory");
        if (sm.redo[quarter] != 0 && *failed == 0)
#pragma unroll 1
            for (int r = part; r < 32; r += 4) {
                const int flat = f0 + quarter * 32 + r;
                if (sm.redo[quarter] >> r & 1u) row_again<YT, SHAPED>(a, ks, flat / R, g * R + flat % R, g, lane);
            }
    }
    fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TM_COLS) : "memory");
}

template <typename YT, int NO, bool SHAPED>
int launch_tc(const CcSeqAttn* a, cudaStream_t st) {
    const size_t smem = sizeof(Small) + (size_t)TILE_BYTES * (5 * ((a->Dk + 63) / 64) + 2 * ((a->Dv + 63) / 64));
    auto kern = attn_tc_kernel<YT, NO, SHAPED>;
    static SmemLimit limit;
    const cudaError_t e = limit.allow(kern, smem);
    if (e != cudaSuccess) return fail(CC_SEQ_ERR_CUDA, cudaGetErrorString(e));
    const long long tiles = ((long long)a->T * (a->H / a->G) + BM - 1) / BM;
    launch_under(kern, dim3((unsigned)(tiles * a->G)), dim3(THREADS), smem, st, *a);
    return cuda_check("attn_tc_kernel");
}

template <typename YT>
int dispatch_tc(const CcSeqAttn* a, cudaStream_t st) {
    const bool shaped = a->softcap > 0.f || a->dist_a != nullptr || !(a->scale > 0.f);
    if (a->Dv <= 64) return shaped ? launch_tc<YT, 16, true>(a, st) : launch_tc<YT, 16, false>(a, st);
    return shaped ? launch_tc<YT, 32, true>(a, st) : launch_tc<YT, 32, false>(a, st);
}

}  // namespace

// bf16 rows of whole 16-byte vectors, up to 128 wide (the three query parts, two key and two value tiles fill the shared
// memory), every pointer on a 16-byte boundary.  Any number of tokens: how many positions lie before them is known on the device
// only.  Measured here and on the FMA kernel in us, 2 / 16 / 64 tokens, 32 / 8 heads of 128: behind 0 positions 12.0 / 15.3 / 20.8 and
// 13.5 / 16.6 / 30.3, behind 500 27.8 / 33.6 / 38.4 and 136 / 150 / 174, behind 4000 129 / 131 / 136 and 1028 / 1074 / 1149.  The FMA
// kernel is ahead only where no position lies before a few tokens of a wide group: 16 tokens, 17 / 1 heads of 128 16.6 and
// 15.4, 64 / 8 heads of 64 13.1 and 11.2.
bool attn_tc_serves(const CcSeqAttn* a) {
    const uintptr_t all = (uintptr_t)a->q | (uintptr_t)a->k_new | (uintptr_t)a->v_new | (uintptr_t)a->k_cache | (uintptr_t)a->v_cache | (uintptr_t)a->y;
    return a->cache_dtype == CC_DT_BF16 && a->Dk % 8 == 0 && a->Dv % 8 == 0 && a->Dk <= 128 && a->Dv <= 128 && (all & 15) == 0 &&
           (long long)a->T * (a->H / a->G) < (1ll << 30);
}

int attn_tc(const CcSeqAttn* a, cudaStream_t st) {
    if (a->y_dtype == CC_DT_F32) return dispatch_tc<float>(a, st);
    if (a->y_dtype == CC_DT_BF16) return dispatch_tc<bf16>(a, st);
    return fail(CC_SEQ_ERR_INVALID_ARG, "unknown element type");
}

}  // namespace ccs
