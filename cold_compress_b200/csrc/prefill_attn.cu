// prefill_attn.cu -- causal prompt attention on the 5th-gen tensor cores (tcgen05 + TMEM), with the
// reductions of the GQA-pooled probability map that the prompt compressors and the score-keeping caches
// consume (SnapKV observation-window mean, heavy-hitter column sums, FastGen window bands) produced in
// the same pass, so the [Hq, S, S] map the reference materialises (attention_utils.py:36-54: 4 GiB per
// layer at S = 8192) never exists.
//
// Replaces, for the prefill branch of Attention.forward (model.py:399-427):
//   scaled_dot_product_attention(q, k, v, mask, return_attn=True)      attention_utils.py:36-54
//   attn.view(B, Hkv, G, S, S).mean(2)                                 model.py:413-418
//   attn[:, :, -16:, :].mean(2)  /  attn.sum(2)                        prompt_compression.py:175, 192; cache.py:704
//   band sums of build_masks' windows                                  cache.py:1066-1173
//
// One CTA = one KV head x one block of QB = 128/G query positions, all G query heads of the group
// stacked into the M = 128 rows of the MMA (row = g * QB + i), so a K/V tile is read once per group.
// Two sweeps over the key tiles (BN = 128 keys):
//   sweep 1  S = Q K^T (tcgen05.mma, fp32 in TMEM) -> row max and sum of exp      (softmax statistics)
//   sweep 2  S again -> P = bf16(exp(l - max) / sum), rounded where the reference rounds -> tensor memory
//            -> Y += P V (tcgen05.mma); the same P, added up over the heads of a query, goes into the pooled reductions.
// The reference's rounding points are kept (NAIVE: bf16 after q.k, after *scale, after softmax, after the
// GQA mean; MATH: fp32 logits, one rounding of P for the tensor core).
// K and V are staged by TMA (cp.async.bulk.tensor, 128-byte swizzle) through a ring of tiles; the logits of the next tiles are formed
// under the current tile's softmax.
// A row with a logit that is NaN or +inf is NaN in y, and in the pooled map as far as its block of queries reaches (the reference's map
// carries it on to every later key; those tiles are not visited).  What a query does not see takes no part in its row.
// Per-tile partial column sums go to a scratch buffer and are added in a fixed order by a second small
// kernel: results are bit-reproducible run to run (no floating-point atomics).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdio.h>
#include <stdint.h>

#include <type_traits>

#include "common.cuh"
#include "internal.h"
#include "smem_limit.cuh"

namespace cc {
namespace {

constexpr int BM = 128;                 // MMA rows of a query tile (G * QB, padded)
constexpr int BN = 128;                 // keys of a tile
constexpr int ATOM_BYTES = 128 * 128;   // one 128-byte-swizzled sub-tile: 128 rows x 64 bf16
constexpr int SOFT_WARPS = 16, NTHREADS = 32 * SOFT_WARPS + 128;   // + a warp each for MMAs and loads, two for column sums
constexpr int MAX_WINDOWS = 4;
constexpr int TMEM_COLS = 512;
constexpr uint32_t WAIT_LIMIT = 1u << 22;
constexpr int RED_THREADS = 64, RED_AHEAD = 16;   // the reduction: columns of a CTA, loads under way per column
constexpr float LOG2E = 1.4426950408889634f;

struct PrefillParams {
    __nv_bfloat16* y;
    long long y_stride_s, y_stride_h;   // elements
    float* part_col;                    // [Hkv][n_qtiles][S_pad]
    float* part_obs;                    // [Hkv][n_obs_tiles][S_pad]
    float* part_band;                   // [n_windows][Hkv][n_qtiles][S_pad]
    int S, S_pad, Hkv, G, QB, n_qtiles;
    int obs_start;                      // first query row of the observation window (S = none)
    int first_obs_tile, n_obs_tiles, n_windows;
    int windows[MAX_WINDOWS];
    float scale;
    int stats;
};

// ------------------------------------------------------------------ PTX wrappers
__device__ __forceinline__ void tma_load_3d(uint32_t smem_dst, const CUtensorMap* tm, int c0, int c1, int c2,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        :: "r"(smem_dst), "l"(tm), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ void mbar_init_u32(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx_u32(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_u32(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_u32(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done != 0;
}
// Bounded: a wait that runs out raises `failed`; every later wait of the CTA then gives up at once, the kernel runs to its
// end and stores NaN.
__device__ __forceinline__ void mbar_wait_u32(uint32_t bar, uint32_t parity, volatile int* failed) {
    if (mbar_try_u32(bar, parity)) return;
    for (uint32_t n = 0; !mbar_try_u32(bar, parity); ++n)
        if (n >= WAIT_LIMIT || *failed) { *failed = 1; return; }
}
// What was started is waited for also after another wait has run out: its shared and its tensor memory go to another CTA.
__device__ __forceinline__ void mbar_wait_out(uint32_t bar, uint32_t parity) {
    for (uint32_t n = 0; n < WAIT_LIMIT && !mbar_try_u32(bar, parity); ++n) {}
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// shared-memory matrix descriptor, 128-byte swizzle (layout type 2), descriptor version 1 (sm_100)
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (2ull << 61);
}
// instruction descriptor: bf16 x bf16 -> fp32, A K-major, B K-major or MN-major
__host__ __device__ constexpr uint32_t make_idesc(int M, int N, bool b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn_major ? 1u : 0u) << 16) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}
// One lane of a whole warp.  What issues MMAs is a warp in step: its operands then lie in uniform registers, where the instruction
// wants them.  One thread on its own took 70 to 110 cycles for an MMA that the pipe does in 64.
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(one));
    return one != 0;
}
// A in tensor memory, B in shared memory
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n" :: "r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}
// 32 lanes x 32 consecutive fp32 columns of this warp's TMEM lane quarter -> registers; the caller waits with tmem_wait_ld
__device__ __forceinline__ void tmem_ld_row(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// The warp's 32 lanes x 32 fp32 columns, four rows of eight values per thread; the caller waits with tmem_wait_ld: v[16 h + 4 k + 2 j + e] = lane
// 16 h + 8 j + thread / 4, column 8 k + 2 (thread % 4) + e
__device__ __forceinline__ void tmem_ld_4rows(uint32_t taddr, uint32_t (&v)[32]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t* const r = v + 16 * h;
        asm volatile(
            "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
              "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr + ((uint32_t)(16 * h) << 16)) : "memory");
    }
}
// The loads' values go through the wait, so that nothing reads one before it (an asm takes 30 operands at most).
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&v)[32]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
        : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]),
          "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]) :: "memory");
    asm volatile(""
        : "+r"(v[15]), "+r"(v[16]), "+r"(v[17]), "+r"(v[18]), "+r"(v[19]), "+r"(v[20]), "+r"(v[21]), "+r"(v[22]), "+r"(v[23]), "+r"(v[24]),
          "+r"(v[25]), "+r"(v[26]), "+r"(v[27]), "+r"(v[28]), "+r"(v[29]) :: "memory");
    asm volatile("" : "+r"(v[30]), "+r"(v[31]) :: "memory");
}
// ... and their bf16 pairs into the first 16 columns: x[j][k] = lane 8 j + thread / 4, column 4 k + thread % 4
__device__ __forceinline__ void tmem_st_4rows(uint32_t taddr, const uint32_t (&x)[4][4]) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
        asm volatile(
            "tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n"
            :: "r"(taddr + ((uint32_t)(16 * h) << 16)), "r"(x[2 * h][0]), "r"(x[2 * h + 1][0]), "r"(x[2 * h][1]), "r"(x[2 * h + 1][1]),
               "r"(x[2 * h][2]), "r"(x[2 * h + 1][2]), "r"(x[2 * h][3]), "r"(x[2 * h + 1][3]) : "memory");
}
// one row per thread, N columns
template <int N>
__device__ __forceinline__ void tmem_st_row(uint32_t taddr, const uint32_t (&x)[N]) {
    static_assert(N == 8 || N == 16, "");
    if constexpr (N == 16)
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n"
            :: "r"(taddr), "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]), "r"(x[8]), "r"(x[9]),
               "r"(x[10]), "r"(x[11]), "r"(x[12]), "r"(x[13]), "r"(x[14]), "r"(x[15]) : "memory");
    else
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n"
            :: "r"(taddr), "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(x[4]), "r"(x[5]), "r"(x[6]), "r"(x[7]) : "memory");
}
__device__ __forceinline__ float ex2(float x) {
    float y; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x)); return y;
}
// two fp32 -> packed bf16x2 (round to nearest even), and back
__device__ __forceinline__ uint32_t cvt_bf16x2(float lo, float hi) {
    uint32_t d; asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo)); return d;
}
// pairs of fp32 values: one instruction for two operations, each rounded as the scalar one
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pair(float a, float b) { f32x2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ void unpair(f32x2 r, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) { f32x2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { f32x2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r; }
__device__ __forceinline__ float bf16x2_lo(uint32_t d) { return __uint_as_float(d << 16); }
__device__ __forceinline__ float bf16x2_hi(uint32_t d) { return __uint_as_float(d & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&p);
}

// Packed bf16 operations, each result rounded once to nearest even.
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) { uint32_t d; asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ uint32_t fma_bf16x2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d; asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c)); return d;
}
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) { uint32_t d; asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }

// Two logits as the reference rounds them: bf16(q.k), then bf16(that times the scale).  1 / sqrt(128) is no bf16 number; x times
// it, rounded to fp32 and then to bf16, is fma(x, hi, bf16(x lo)) with its two bf16 parts: equal for every finite bf16 x of at
// least 2^-100 (checked over all of them in tests/test_prefill_rounding.py), and below that both are zero to any exponential.
// Three instructions for a pair where fp32 takes five.  1 / sqrt(64) is a power of two.
constexpr uint32_t SCALE128_HI = 0x3db53db5u, SCALE128_LO = 0x371e371eu, SCALE64 = 0x3e003e00u;
template <int D>
__device__ __forceinline__ uint32_t round_logits(float x, float y) {
    const uint32_t d = cvt_bf16x2(x, y);
    if constexpr (D == 64) return mul_bf16x2(d, SCALE64);
    else return fma_bf16x2(d, SCALE128_HI, mul_bf16x2(d, SCALE128_LO));
}

// N pairs of a row's logits: bf16 with the reference's roundings, or fp32.
template <bool NAIVE, int N = 16>
struct Logits {
    uint32_t w[N];
    template <int D>
    __device__ __forceinline__ void set(int c, float x, float y, f32x2) { w[c] = round_logits<D>(x, y); }
    __device__ __forceinline__ f32x2 get(int c) const { return pair(bf16x2_lo(w[c]), bf16x2_hi(w[c])); }
    __device__ __forceinline__ void hide(int c, bool first, bool second) {
        if (first) w[c] = (w[c] & 0xffff0000u) | 0xff80u;
        if (second) w[c] = (w[c] & 0xffffu) | 0xff800000u;
    }
    __device__ __forceinline__ float max() const {
        uint32_t m[4] = {w[0], w[1], w[2], w[3]};
#pragma unroll
        for (int c = 4; c < N; ++c) m[c & 3] = max_bf16x2(m[c & 3], w[c]);
        m[0] = max_bf16x2(max_bf16x2(m[0], m[1]), max_bf16x2(m[2], m[3]));
        return fmaxf(bf16x2_lo(m[0]), bf16x2_hi(m[0]));
    }
};
template <int N>
struct Logits<false, N> {
    f32x2 w[N];
    template <int D>
    __device__ __forceinline__ void set(int c, float x, float y, f32x2 scale) { w[c] = mul2(pair(x, y), scale); }
    __device__ __forceinline__ f32x2 get(int c) const { return w[c]; }
    __device__ __forceinline__ void hide(int c, bool first, bool second) {
        float x, y;
        unpair(w[c], x, y);
        w[c] = pair(first ? -INFINITY : x, second ? -INFINITY : y);
    }
    __device__ __forceinline__ float max() const {
        float m[2], x, y;
        unpair(w[0], m[0], m[1]);
#pragma unroll
        for (int c = 1; c < N; ++c) {
            unpair(w[c], x, y);
            m[0] = fmaxf(m[0], x);
            m[1] = fmaxf(m[1], y);
        }
        return fmaxf(m[0], m[1]);
    }
};

// ------------------------------------------------------------------ the kernel
struct Small {
    uint64_t bars[30];
    uint32_t tmem;
    int failed;
    float fin[BM][2];       // minus the offset z(maximum) and one over the sum, of every row
    float stat[4][BM][3];   // of a row's key quarters: maximum, offset of the sum, sum
};
// Tiles of K and V in shared memory (the last one is where Q was), and the pooled probabilities of two tiles, [QB][128 keys] bf16.
template <int D, int QQ> __host__ __device__ constexpr int stages() { return D == 64 || QQ <= 8 ? 6 : QQ == 16 ? 5 : 4; }
template <int D, int QQ> constexpr int smem_bytes() {
    return 1024 + stages<D, QQ>() * (D / 64) * ATOM_BYTES + 2 * 4 * QQ * BN * 2 + (int)sizeof(Small);
}

// grid = n_qtiles * Hkv CTAs (longest query tiles first).  Rows: TMEM lane quarter j holds QQ = QB / 4 queries, row = QQ g + i, so
// that all heads of a query lie in one quarter and, read back with tcgen05.ld.16x256b, in one thread (QQ >= 8) or in two that
// are 16 lanes apart (QQ = 4).  Sixteen warps of softmax in two groups that take every second tile: warp w has lane quarter w % 4,
// keys 64 (w / 4 % 2) .. + 63 in two steps of 32, and tiles w / 8, + 2, ...  One warp each issues the MMAs and loads K and V, two
// add up over the queries; nobody meets anybody at a CTA barrier per tile, and while one group waits for the tensor
// memory or a product the other one has the ALUs.
//
// Sweep 1 reads a row per thread.  Its sum is kept relative to a reference that need not be the maximum: the exponentials of a
// step start at once with the reference there is, and only where the step's own maximum turns out to lie more than 2 above
// it are they formed again with that maximum as the reference.  Sweep 2 subtracts the maximum itself.
// Sweep 2 reads four rows x 8 keys per thread: P goes back to tensor memory as the A operand of P V, and a query's heads are
// added up in registers.  The pooled probabilities go to shared memory, where the two warps of the sums over the queries take them.
//
// Bound: issue slots (54 % busy), the exponentials (two per logit at 16 per SM and cycle: 50 %) and the waits between them, at four
// warps of softmax per scheduler; a 128 x 128 tile takes 1430 cycles in sweep 1 and 2000 in sweep 2, of which the MMAs take 515 and
// 1030.  Measured at 7680 tokens x 32 heads of 128 (8 key/value heads) / 4096 / 1531 x 28 (4), in us, reduction included, in bursts: two
// groups of 256 threads that shared a barrier per 64 keys and issued their own MMAs 1397 / 412 / 105, this 814 / 268 / 75 (904 and 70
// over seconds with L2 flushed between calls, where power takes part).
// On the way: MMAs issued by one thread instead of a warp in step 976; mma.sync for the sums over heads and queries 943 (1500
// cycles a tile: it waits for the tensor pipe behind the tcgen05 MMAs); all warps on the same tile 816; a quarter of the
// exponentials as polynomials of degree 6 on the FMA pipe 924; the sums over the heads a tile later, among the exponentials, 899; the next
// tile's logits fetched under the pooling 840; Q in shared memory and two P 839.
template <int D, bool NAIVE, int QQ>
__global__ void __launch_bounds__(NTHREADS, 1)
prefill_attn_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                    const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ PrefillParams p) {
    constexpr int DH = D / 64;                    // 64-column (128-byte) sub-tiles along the head dimension
    constexpr int TILE_BYTES = DH * ATOM_BYTES;   // 128 rows of Q, K or V
    constexpr int QB = 4 * QQ;                    // query positions of a CTA
    constexpr int NS = QQ >= 8 ? QQ / 8 : 1;      // queries of a thread in sweep 2
    constexpr int STAGES = stages<D, QQ>(), POOL_BYTES = QB * BN * 2;
    constexpr int TM_Y = 2 * BN, TM_Q = 3 * BN, TM_P = TM_Q + 64;   // tensor memory: logits 2 x 128 | Y, in sweep 1 logits | Q | P
    extern __shared__ uint8_t smem_raw[];

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int h = blockIdx.x % p.Hkv;
    const int qt = p.n_qtiles - 1 - blockIdx.x / p.Hkv;
    const int i0 = qt * QB;
    const int lim = min(i0 + QB, p.S);                          // keys [0, lim) are visible to this query block
    const int T = (lim + BN - 1) / BN;                          // tiles

    const uint32_t sT = (smem_u32(smem_raw) + 1023u) & ~1023u, sQ = sT + (STAGES - 1) * TILE_BYTES;
    uint8_t* const q_rows = smem_raw + (sQ - smem_u32(smem_raw));
    uint8_t* const pools = q_rows + TILE_BYTES;                 // [2][QB][16 chunks of 8 keys], chunks 4 .. of odd rows first
    Small& sm = *reinterpret_cast<Small*>(pools + 2 * POOL_BYTES);
    volatile int* const failed = &sm.failed;
    const uint32_t bar = smem_u32(sm.bars);
    const uint32_t Q_FULL = bar, Q_READY = bar + 8, Y_DONE = bar + 16;
    auto FULL = [&](int b) { return bar + 24 + 8u * b; };
    auto FREE = [&](int b) { return bar + 72 + 8u * b; };
    auto S_FULL = [&](int b) { return bar + 120 + 8u * b; };
    auto S_READ = [&](int b) { return bar + 144 + 8u * b; };
    auto P_FULL = [&](int b) { return bar + 168 + 8u * b; };
    auto C_FULL = [&](int b) { return bar + 184 + 8u * b; };
    auto C_READ = [&](int b) { return bar + 200 + 8u * b; };
    auto PV_DONE = [&](int b) { return bar + 216 + 8u * b; };
    // Sweep 1 goes round three accumulators (the third where Y comes later), sweep 2 round the first two, after `used` turns each.
    auto used = [&](int b) { return (T - b + 2) / 3; };

    int loaded = 0;                                             // tiles asked for, by the one thread that asks
    auto load = [&](const CUtensorMap* tm, int tile) {
        const int st = loaded % STAGES;
        if (loaded >= STAGES) mbar_wait_u32(FREE(st), (loaded / STAGES - 1) & 1, failed);
        else if (loaded == STAGES - 1) mbar_wait_u32(Q_READY, 0, failed);
        if (*failed) return;
        mbar_expect_tx_u32(FULL(st), TILE_BYTES);
#pragma unroll
        for (int dh = 0; dh < DH; ++dh) tma_load_3d(sT + st * TILE_BYTES + dh * ATOM_BYTES, tm, dh * 64, tile * BN, h, FULL(st));
        ++loaded;
    };
    // Short prompts are a chain of waits: Q and the first tile of K are asked for as soon as their barriers are there, while another warp
    // allocates tensor memory.  One after the other / so, us: 8 heads of 128 without groups or statistics, 17 tokens 6.57 / 6.26, 129 8.37 / 8.0,
    // 384 11.4 / 11.0; 28 / 4 heads with statistics, 64 tokens 11.9 / 11.5.  Further tiles of K asked for here as well: 6.57, 8.2 and 11.6.
    if (warp == SOFT_WARPS + 1 && lane == 0) {
        *failed = 0;
        mbar_init_u32(Q_FULL, 1);
        mbar_init_u32(Q_READY, SOFT_WARPS);
        mbar_init_u32(Y_DONE, 1);
        for (int b = 0; b < STAGES; ++b) { mbar_init_u32(FULL(b), 1); mbar_init_u32(FREE(b), 1); }
        for (int b = 0; b < 3; ++b) { mbar_init_u32(S_FULL(b), 1); mbar_init_u32(S_READ(b), SOFT_WARPS / 2); }
        for (int b = 0; b < 2; ++b) {
            mbar_init_u32(P_FULL(b), SOFT_WARPS / 2);
            mbar_init_u32(C_FULL(b), SOFT_WARPS / 2);
            mbar_init_u32(C_READ(b), 2);
            mbar_init_u32(PV_DONE(b), 1);
        }
        mbar_fence_init();
        fence_proxy_async();
        mbar_expect_tx_u32(Q_FULL, (uint32_t)(4 * DH * p.G * QQ * 128));
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int dh = 0; dh < DH; ++dh) tma_load_3d(sQ + dh * ATOM_BYTES + j * 32 * 128, &tm_q, dh * 64, i0 + j * QQ, h * p.G, Q_FULL);
        load(&tm_k, 0);
    }
    __syncwarp();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(smem_u32(&sm.tmem)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    const int no_head = 32 - p.G * QQ;                          // rows of a quarter that Q does not cover: zero (they only feed unused rows)
    for (int i = tid; i < 4 * no_head * DH * 8; i += NTHREADS) {
        const int r = i >> 3, quarter = r & 3, dh = (r >> 2) % DH, row = p.G * QQ + (r >> 2) / DH;
        reinterpret_cast<uint4*>(q_rows + dh * ATOM_BYTES + (quarter * 32 + row) * 128)[i & 7] = make_uint4(0, 0, 0, 0);
    }
    if (no_head > 0) fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sm.tmem;

    if (warp >= SOFT_WARPS) {
        if (warp == SOFT_WARPS) {
            constexpr uint32_t IDESC_S = make_idesc(BM, BN, false), IDESC_PV = make_idesc(BM, D, true);
            const uint64_t k_desc = smem_desc(sT, 16, 1024), v_desc = smem_desc(sT, ATOM_BYTES, 1024);
            // The tiles come in the order in which they are used: K of sweep 1, then K of tile t + 2 before V of tile t.
            int st = 0;
            uint32_t turn = 0;
            auto next = [&] { if (++st == STAGES) { st = 0; turn ^= 1; } };
            auto lost = [&] { return __any_sync(0xffffffffu, *failed) != 0; };      // the same for all lanes, which elect_one wants together
            auto logits = [&](int b) {                   // S[b] = Q K^T: [128 x 128], Q in tensor memory
                mbar_wait_u32(FULL(st), turn, failed);
                tc_fence_after();
                if (elect_one()) {
                    const uint64_t desc = k_desc + st * (TILE_BYTES >> 4);
#pragma unroll
                    for (int k = 0; k < D / 16; ++k)
                        umma_ts(tmem + b * BN, tmem + TM_Q + 8 * k, desc + ((k >> 2) * ATOM_BYTES + (k & 3) * 32) / 16, IDESC_S, k > 0);
                    umma_commit(S_FULL(b));
                    umma_commit(FREE(st));
                }
                __syncwarp();
                next();
            };
            mbar_wait_u32(Q_READY, 0, failed);
            tc_fence_after();
            uint32_t read = 1;
            for (int n = 0, b = 0; n < T && !lost(); ++n) {
                if (n >= 3) mbar_wait_u32(S_READ(b), read, failed);
                logits(b);
                if (++b == 3) { b = 0; read ^= 1; }
            }
            for (int t = -2; t < T && !lost(); ++t) {
                if (t + 2 < T) {
                    const int b = t & 1, turns = used(b) + ((t + 2) >> 1);            // of this accumulator, so far
                    if (turns > 0) mbar_wait_u32(S_READ(b), (turns - 1) & 1, failed);
                    logits(b);
                }
                if (t < 0) continue;
                mbar_wait_u32(P_FULL(t & 1), (t >> 1) & 1, failed);
                mbar_wait_u32(FULL(st), turn, failed);
                tc_fence_after();
                const int ksteps = min(BN, lim - t * BN + 15) >> 4;       // keys past the last query's take no part
                if (elect_one()) {
                    const uint64_t desc = v_desc + st * (TILE_BYTES >> 4);
#pragma unroll
                    for (int k = 0; k < BN / 16; ++k)
                        if (k < ksteps) umma_ts(tmem + TM_Y, tmem + TM_P + 8 * k, desc + k * 128, IDESC_PV, t > 0 || k > 0);
                    umma_commit(PV_DONE(t & 1));
                    umma_commit(FREE(st));
                }
                __syncwarp();
                next();
            }
            if (elect_one()) umma_commit(Y_DONE);
            __syncwarp();
            mbar_wait_out(Y_DONE, 0);
        } else if (warp == SOFT_WARPS + 1) {
            if (lane == 0) {
                for (int t = loaded; t < T; ++t) load(&tm_k, t);
                for (int t = -2; t < T; ++t) {
                    if (t + 2 < T) load(&tm_k, t + 2);
                    if (t >= 0) load(&tm_v, t);
                }
                mbar_wait_out(Q_FULL, 0);
                for (int m = max(0, loaded - STAGES); m < loaded; ++m) mbar_wait_out(FULL(m % STAGES), (m / STAGES) & 1);
            }
            __syncwarp();
        } else if (p.stats) {
            // Sums over the queries, straight to this block's partials; sums of their own for a band only in tiles that its edge crosses
            // (2047 tokens, two windows, us with sums of their own in every tile / so: 8 heads of 128 without groups 103 / 68, 32 / 8 107 / 90).
            // A warp has 64 keys, a lane 8 of them in every fourth row: chunk c holds keys 32 (c / 4) + 8 k + 2 (c % 4) + e as pair k.
            const int c = 8 * (warp - SOFT_WARPS - 2) + (lane & 7), first = lane >> 3, rows = min(QB, p.S - i0);
            const bool high = lane & 16, odd = lane & 8, obs = qt >= p.first_obs_tile;
            const int key = 32 * (c >> 2) + 8 * ((high ? 2 : 0) + (odd ? 1 : 0)) + 2 * (c & 3);   // of the pair that this lane stores
            float* const col = p.part_col + ((size_t)h * p.n_qtiles + qt) * p.S_pad + key;
            float* const seen = p.part_obs + ((size_t)h * p.n_obs_tiles + (obs ? qt - p.first_obs_tile : 0)) * p.S_pad + key;
            float* const band = p.part_band + ((size_t)h * p.n_qtiles + qt) * p.S_pad + key;
            for (int t = 0; t < T; ++t) {
                const uint8_t* const pool = pools + (t & 1) * POOL_BYTES;
                mbar_wait_u32(C_FULL(t & 1), (t >> 1) & 1, failed);
                __syncwarp();
                auto add = [&](auto banded, int from, int window, float* out) {       // rows from `from` on, banded: of the last `window` keys each
                    f32x2 s[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll 4
                    for (int r = first; r < rows; r += 4) {
                        uint4 u = *reinterpret_cast<const uint4*>(pool + r * (BN * 2) + ((c ^ ((r & 1) << 2)) << 4));
                        if (r < from) continue;
                        if constexpr (decltype(banded)::value) {
                            const int lo = i0 + r - window - (t * BN + 32 * (c >> 2) + 2 * (c & 3));   // pair k is inside past here
                            auto inside = [&](uint32_t w, int k) { return (8 * k > lo ? w & 0xffffu : 0u) | (8 * k + 1 > lo ? w & 0xffff0000u : 0u); };
                            u = make_uint4(inside(u.x, 0), inside(u.y, 1), inside(u.z, 2), inside(u.w, 3));
                        }
                        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                        for (int k = 0; k < 4; ++k) s[k] = add2(s[k], pair(bf16x2_lo(w[k]), bf16x2_hi(w[k])));
                    }
                    // over the four rows at a time: lanes 16 and 8 apart swap pairs
                    f32x2 a[2], b;
#pragma unroll
                    for (int k = 0; k < 2; ++k) a[k] = add2(high ? s[k + 2] : s[k], __shfl_xor_sync(0xffffffffu, high ? s[k] : s[k + 2], 16));
                    b = add2(odd ? a[1] : a[0], __shfl_xor_sync(0xffffffffu, odd ? a[0] : a[1], 8));
                    float2 f;
                    unpair(b, f.x, f.y);
                    if (*failed) f = make_float2(NAN, NAN);
                    *reinterpret_cast<float2*>(out + t * BN) = f;
                    return f;
                };
                const float2 all = add(std::false_type(), 0, 0, col);
                if (obs) add(std::false_type(), p.obs_start - i0, 0, seen);
                for (int w = 0; w < p.n_windows; ++w) {
                    const int window = p.windows[w], from = i0 - t * BN;                 // of the first row, from the tile's first key
                    float* const out = band + (size_t)w * p.Hkv * p.n_qtiles * p.S_pad;
                    if (from - (BN - 1) >= window) continue;                             // no row has a key of the tile inside: never read
                    if (from + rows - 1 < window) *reinterpret_cast<float2*>(out + t * BN) = all;   // every row has every key inside
                    else add(std::true_type(), 0, window, out);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive_u32(C_READ(t & 1));
            }
        }
    } else {
        const int quarter = warp & 3, part = warp >> 2;               // row quarter, of Q and Y a quarter of the columns
        const int half = part & 1, group = part >> 1;                 // half of a tile's keys, of every second tile
        const uint32_t lanes = (uint32_t)(quarter * 32) << 16;
        const int row = quarter * 32 + lane, q0 = i0 + quarter * QQ;
        {   // Q to tensor memory: this row's columns part D / 4 .. (two bf16 a TMEM column)
            mbar_wait_u32(Q_FULL, 0, failed);
            __syncwarp();
            uint32_t w[D / 8];
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
                const int c8 = part * (D / 32) + c;                      // 16-byte chunk of the row
                const uint4 u = *reinterpret_cast<const uint4*>(q_rows + (c8 >> 3) * ATOM_BYTES + row * 128 + (((c8 & 7) ^ (row & 7)) << 4));
                w[4 * c] = u.x; w[4 * c + 1] = u.y; w[4 * c + 2] = u.z; w[4 * c + 3] = u.w;
            }
            tmem_st_row<D / 8>(tmem + lanes + TM_Q + part * (D / 8), w);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_u32(Q_READY);
        }
        const float scale = p.scale;
        const f32x2 log2e2 = pair(LOG2E, LOG2E), scale2 = pair(scale, scale);

        // exp(l - m) = 2^(l log2(e) - z(m)) with z(m) = m log2(e) rounded ONCE: the fma rounds the difference alone, and the rounding
        // of z is a factor common to all terms that the same m scales.  It cancels because every change of reference goes from z to z;
        // a factor formed from m - m' instead left it in the sums (largest weight error at logits near 20 / 100 / 500 / 16384:
        // 2.2e-6 / 6e-6 / 2.8e-5 / 7.6e-4, from z to z 0.9e-6 throughout, as with the difference formed first).
        auto in_log2 = [](float m) { return __fmul_rn(m, LOG2E); };

        // ---- sweep 1: softmax statistics of one row per thread.  The logits of tile n + 1 are fetched and rounded among the
        // exponentials of tile n.
        {
            const int qi = q0 + lane % QQ;
            float m_top = -INFINITY, m_ref = -INFINITY, z_ref = 0.f, s_run = 0.f;
            uint32_t v[32];
            Logits<NAIVE> l;
            // steps: 32 keys at a time, two of a tile
            auto first_key = [&](int i) { return (group + (i & ~1)) * BN + half * 64 + (i & 1) * 32; };
            auto fetch = [&](int i) {
                const int n = group + (i & ~1), b = n % 3;
                if (!(i & 1)) mbar_wait_u32(S_FULL(b), (n / 3) & 1, failed);
                __syncwarp();
                tc_fence_after();
                tmem_ld_row(tmem + lanes + b * BN + half * 64 + (i & 1) * 32, v);
            };
            auto fetched = [&](int i) {
                tmem_wait_ld(v);
                tc_fence_before();
                __syncwarp();
                if ((i & 1) && lane == 0) mbar_arrive_u32(S_READ((group + (i & ~1)) % 3));
            };
            auto cut = [&](int i) {                        // keys past the row's diagonal
                const int kbase = first_key(i);
                if (kbase + 31 > q0) {
                    const int seen = qi - kbase;           // keys 0 .. seen
#pragma unroll
                    for (int c = 0; c < 16; ++c) l.hide(c, 2 * c > seen, 2 * c + 1 > seen);
                }
            };
            auto add_up = [&](const Logits<NAIVE>& x, float z, int from, int to, f32x2 (&a)[2]) {
                const f32x2 off = pair(-z, -z);
#pragma unroll
                for (int c = from; c < to; ++c) {
                    float e, f;
                    unpair(fma2(x.get(c), log2e2, off), e, f);
                    a[c & 1] = add2(a[c & 1], pair(ex2(e), ex2(f)));
                }
            };
            auto total = [&](const f32x2 (&a)[2]) {
                float a0, a1;
                unpair(add2(a[0], a[1]), a0, a1);
                return a0 + a1;
            };
            auto take = [&](const Logits<NAIVE>& x, float top, float sum) {
                m_top = fmaxf(m_top, top);
                if (top > m_ref + 2.f) {       // also for the first finite logit: there is no reference yet
                    const float z = in_log2(top);
                    f32x2 a[2] = {0ull, 0ull};
                    add_up(x, z, 0, 16, a);
                    s_run = s_run * (m_ref == -INFINITY ? 0.f : ex2(z_ref - z)) + total(a);
                    m_ref = top;
                    z_ref = z;
                } else {
                    s_run += sum;
                }
            };
            const int steps = T > group ? (T - group + 1) & ~1 : 0;
            if (steps > 0) {
                fetch(0);
                fetched(0);
#pragma unroll
                for (int c = 0; c < 16; ++c) l.template set<D>(c, __uint_as_float(v[2 * c]), __uint_as_float(v[2 * c + 1]), scale2);
                cut(0);
                for (int i = 1; i < steps; ++i) {
                    fetch(i);
                    const Logits<NAIVE> x = l;
                    const float top = x.max();
                    f32x2 a[2] = {0ull, 0ull};
                    add_up(x, z_ref, 0, 8, a);
                    fetched(i);
#pragma unroll
                    for (int c = 0; c < 16; ++c) l.template set<D>(c, __uint_as_float(v[2 * c]), __uint_as_float(v[2 * c + 1]), scale2);
                    add_up(x, z_ref, 8, 16, a);
                    take(x, top, total(a));
                    cut(i);
                }
                f32x2 a[2] = {0ull, 0ull};
                add_up(l, z_ref, 0, 16, a);
                take(l, l.max(), total(a));
            }
            sm.stat[part][row][0] = m_top;
            sm.stat[part][row][1] = m_ref == -INFINITY ? -INFINITY : z_ref;
            sm.stat[part][row][2] = s_run;
        }
        asm volatile("bar.sync 1, 512;" ::: "memory");
        if (part == 0) {    // the four parts of every row
            float m = sm.stat[0][row][0], tot = 0.f;
#pragma unroll
            for (int q = 1; q < 4; ++q) m = fmaxf(m, sm.stat[q][row][0]);        // finite: key 0 is visible to every query
            const float z = in_log2(m);
#pragma unroll
            for (int q = 0; q < 4; ++q) tot += sm.stat[q][row][2] * ex2(sm.stat[q][row][1] - z);
            sm.fin[row][0] = -z;
            sm.fin[row][1] = 1.0f / tot;
        }
        asm volatile("bar.sync 1, 512;" ::: "memory");

        // ---- sweep 2: probabilities of rows 8 j + lane / 4 of the quarter, keys 8 k + 2 (lane % 4), + 1 of the warp's 32
        const int r8 = lane >> 2, c2 = 2 * (lane & 3);
        f32x2 off[4], inv[4];
        bool no_number = false;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float* const f = sm.fin[quarter * 32 + 8 * j + r8];
            off[j] = pair(f[0], f[0]);
            inv[j] = pair(f[1], f[1]);
            no_number |= f[1] != f[1];
        }
        no_number = __any_sync(0xffffffffu, no_number);            // a row that is NaN is so for the keys that it does not see, too
        const float fG = (float)p.G, invG = 1.0f / (float)p.G;
        const bool g_pow2 = (p.G & (p.G - 1)) == 0, short_heads = p.G * QQ < 32;
        const f32x2 invG2 = pair(invG, invG);
        // where this thread's pooled probabilities go: row = query of the block, chunks of the two steps
        const int pool_row = (quarter * QQ + (QQ == 4 ? r8 & 3 : r8)) * (BN * 2) + half * 128 + ((lane & 3) << 4), pool_swap = (r8 & 1) << 6;
        uint32_t v[32];                                            // v[16 (j / 2) + 4 k + 2 (j % 2) + e]
        uint32_t first[4][4], second[4][4];                       // of a tile's two steps
        auto weigh_all = [&](int kbase, uint32_t (&pk)[4][4]) {
            auto weigh = [&](auto cut) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int seen = q0 + (8 * j + r8) % QQ - kbase - c2;   // key 8 k + e is seen up to here
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const int at_v = 16 * (j >> 1) + 4 * k + 2 * (j & 1);
                        Logits<NAIVE, 1> l;
                        l.template set<D>(0, __uint_as_float(v[at_v]), __uint_as_float(v[at_v + 1]), scale2);
                        if constexpr (decltype(cut)::value) l.hide(0, 8 * k > seen, 8 * k + 1 > seen);
                        float x, y;
                        unpair(fma2(l.get(0), log2e2, off[j]), x, y);
                        unpair(mul2(pair(ex2(x), ex2(y)), inv[j]), x, y);
                        pk[j][k] = cvt_bf16x2(x, y);
                    }
                }
            };
            if (kbase + 31 <= q0) {
                weigh(std::false_type());
            } else if (kbase < q0 + QQ || no_number) {
                weigh(std::true_type());
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int k = 0; k < 4; ++k) pk[j][k] = 0u;         // nobody of the quarter sees these keys
            }
        };
        auto pool = [&](int step, uint32_t (&pk)[4][4]) {
            if (short_heads) {      // rows without a head take no part
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (8 * j + r8 >= p.G * QQ)
#pragma unroll
                        for (int k = 0; k < 4; ++k) pk[j][k] = 0u;
            }
            uint8_t* const at = pools + group * POOL_BYTES + pool_row + ((step << 6) ^ pool_swap);
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                uint32_t w[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if constexpr (QQ == 32) {
                        w[k] = pk[s][k];                                    // one head: the probabilities themselves
                    } else {
                        f32x2 c = pair(bf16x2_lo(pk[s][k]), bf16x2_hi(pk[s][k]));
#pragma unroll
                        for (int j = s + NS; j < 4; j += NS) c = add2(c, pair(bf16x2_lo(pk[j][k]), bf16x2_hi(pk[j][k])));
                        if constexpr (QQ == 4) c = add2(c, __shfl_xor_sync(0xffffffffu, c, 16));
                        float x, y;
                        if (g_pow2) {
                            unpair(mul2(c, invG2), x, y);
                        } else {
                            unpair(c, x, y);
                            x = __fdiv_rn(x, fG);
                            y = __fdiv_rn(y, fG);
                        }
                        w[k] = cvt_bf16x2(x, y);
                    }
                }
                if (QQ >= 8 || r8 < 4) *reinterpret_cast<uint4*>(at + s * 8 * (BN * 2)) = make_uint4(w[0], w[1], w[2], w[3]);
            }
        };
        for (int t = group; t < T; t += 2) {
            const int kbase = t * BN + half * 64;
            const uint32_t at = tmem + lanes + group * BN + half * 64, to = tmem + lanes + TM_P + half * 32;
            mbar_wait_u32(S_FULL(group), (used(group) + (t >> 1)) & 1, failed);
            __syncwarp();
            tc_fence_after();
            tmem_ld_4rows(at, v);
            tmem_wait_ld(v);
            weigh_all(kbase, first);
            tmem_ld_4rows(at + 32, v);                                 // under the pooling
            if (p.stats) {
                if (t >= 2) mbar_wait_u32(C_READ(group), ((t - 2) >> 1) & 1, failed);   // the last contents of this tile's place are summed
                __syncwarp();
                pool(0, first);
            }
            tmem_wait_ld(v);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_u32(S_READ(group));
            weigh_all(kbase + 32, second);
            if (t > 0) mbar_wait_u32(PV_DONE(group ^ 1), ((t - 1) >> 1) & 1, failed);    // the product of the tile before has been through P
            __syncwarp();
            tc_fence_after();
            tmem_st_4rows(to, first);
            tmem_st_4rows(to + 16, second);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_u32(P_FULL(group));
            __syncwarp();
            if (p.stats) {
                pool(1, second);
                __syncwarp();
                if (lane == 0) mbar_arrive_u32(C_FULL(group));
            }
        }

        // ---- epilogue: Y (fp32 in TMEM) -> bf16 -> global; thread = row, columns part D / 4 ..
        mbar_wait_u32(Y_DONE, 0, failed);
        __syncwarp();
        tc_fence_after();
        constexpr int CPT = D / 4;
        const int og = lane / QQ, oqi = q0 + lane % QQ;
        uint32_t y[32];
        tmem_ld_row(tmem + lanes + TM_Y + (CPT == 32 ? part * 32 : (part >> 1) * 32), y);   // D = 64: the enclosing 32 columns
        tmem_wait_ld(y);
        if (og < p.G && oqi < p.S) {
            __nv_bfloat16* yrow = p.y + (long long)(h * p.G + og) * p.y_stride_h + (long long)oqi * p.y_stride_s + part * CPT;
            const bool lost = *failed;
#pragma unroll
            for (int c = 0; c < CPT; c += 8) {
                float e[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) e[u] = lost ? NAN : __uint_as_float((CPT == 16 && (part & 1)) ? y[(16 + c + u) & 31] : y[c + u]);
                *reinterpret_cast<uint4*>(yrow + c) = make_uint4(pack_bf16(e[0], e[1]), pack_bf16(e[2], e[3]),
                                                                  pack_bf16(e[4], e[5]), pack_bf16(e[6], e[7]));
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

// acc + part[qt0] + part[qt0 + 1] + .. + part[qt1 - 1], in this order, RED_AHEAD loads under way at a time.
__device__ __forceinline__ float sum_tiles(const float* __restrict__ part, size_t slab, int qt0, int qt1) {
    float acc = 0.f;
    for (int qt = qt0; qt < qt1; qt += RED_AHEAD) {
        float v[RED_AHEAD];
#pragma unroll
        for (int u = 0; u < RED_AHEAD; ++u) v[u] = qt + u < qt1 ? part[(size_t)(qt + u) * slab] : 0.f;
#pragma unroll
        for (int u = 0; u < RED_AHEAD; ++u) acc += v[u];   // adding the zeros past qt1 changes no bit: the partials are >= 0
    }
    return acc;
}

// Fixed-order sum of the per-tile partials, rounded for its consumers on the way out (three launches of tensor operations behind it: 8 of
// the 81 us that 1531 tokens took): one thread per (head, column).  Bound: latency, a column's sum is a chain of
// as many loads as there are query tiles behind it; so RED_AHEAD of them are under way at once and the CTAs are small
// enough that short prompts reach most of the chip.  Measured at 7680 / 4096 tokens x 8 heads and 1531 x 4 in groups of 7:
// 16.8 / 8.9 / 5.5 us; CTAs of 256 with the loop as the compiler unrolls it 37.9 / 18.7 / 11.9.
// BF16: as the consumers take them, the column sums and the mean of the observed rows in bf16; fp32 sums otherwise.
template <bool BF16>
__global__ void __launch_bounds__(RED_THREADS)
prefill_reduce_kernel(const __grid_constant__ PrefillParams p, void* __restrict__ col_sum, void* __restrict__ obs_sum,
                      float* __restrict__ band_sum, float per_obs_row) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int h = blockIdx.y;
    if (j >= p.S) return;
    const size_t slab = (size_t)p.S_pad, at = (size_t)h * p.S + j;
    const int qt0 = j / p.QB;
    const float col = sum_tiles(p.part_col + (size_t)h * p.n_qtiles * slab + j, slab, qt0, p.n_qtiles);
    if (BF16) ((__nv_bfloat16*)col_sum)[at] = __float2bfloat16_rn(col);
    else ((float*)col_sum)[at] = col;
    if (obs_sum) {
        const int first = max(qt0, p.first_obs_tile) - p.first_obs_tile;
        const float obs = sum_tiles(p.part_obs + (size_t)h * p.n_obs_tiles * slab + j, slab, first, p.n_obs_tiles);
        if (BF16) ((__nv_bfloat16*)obs_sum)[at] = __float2bfloat16_rn(__fmul_rn(obs, per_obs_row));
        else ((float*)obs_sum)[at] = obs;
    }
    for (int w = 0; w < p.n_windows; ++w) {
        const int qt1 = min(p.n_qtiles - 1, (j + p.windows[w] - 1) / p.QB);   // later query tiles are outside the band
        band_sum[((size_t)w * p.Hkv + h) * p.S + j] =
            sum_tiles(p.part_band + ((size_t)w * p.Hkv + h) * p.n_qtiles * slab + j, slab, qt0, qt1 + 1);
    }
}

// ------------------------------------------------------------------ host side
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static const EncodeTiledFn fn = [] {      // looked up once; other threads wait for it
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &found) != cudaSuccess || found != cudaDriverEntryPointSuccess)
            ptr = nullptr;
        return (EncodeTiledFn)ptr;
    }();
    return fn;
}

// bf16 tensor [heads][S][D] with element strides (head, row); box = (64 columns, box_rows, box_heads), 128B swizzle
int make_map(CUtensorMap* tm, const void* base, int D, int S, int heads, long long stride_s, long long stride_h,
             int box_rows, int box_heads) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return set_error(CC_ERR_CUDA, "cc_prefill_attention: cuTensorMapEncodeTiled entry point not available");
    cuuint64_t dims[3] = {(cuuint64_t)D, (cuuint64_t)S, (cuuint64_t)heads};
    cuuint64_t strides[2] = {(cuuint64_t)stride_s * 2, (cuuint64_t)stride_h * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)box_rows, (cuuint32_t)box_heads};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        char msg[160];
        snprintf(msg, sizeof(msg), "cc_prefill_attention: cuTensorMapEncodeTiled failed (CUresult %d)", (int)r);
        return set_error(CC_ERR_CUDA, msg);
    }
    return CC_OK;
}

int query_block(int G) {   // largest power of two <= 128 / G
    int qb = 1;
    while (qb * 2 * G <= BM) qb *= 2;
    return qb;
}

struct Plan {
    int QB, n_qtiles, S_pad, first_obs_tile, n_obs_tiles;
    size_t col_floats, obs_floats, band_floats;
};

Plan make_plan(int S, int Hkv, int G, int obs_len, int n_windows) {
    Plan pl;
    pl.QB = query_block(G);
    pl.n_qtiles = (S + pl.QB - 1) / pl.QB;
    pl.S_pad = (S + BN - 1) / BN * BN;
    const int obs = obs_len > S ? S : obs_len;
    pl.first_obs_tile = obs > 0 ? (S - obs) / pl.QB : pl.n_qtiles;
    pl.n_obs_tiles = pl.n_qtiles - pl.first_obs_tile;
    pl.col_floats = (size_t)Hkv * pl.n_qtiles * pl.S_pad;
    pl.obs_floats = (size_t)Hkv * pl.n_obs_tiles * pl.S_pad;
    pl.band_floats = (size_t)n_windows * pl.col_floats;
    return pl;
}

template <int D, bool NAIVE, int QQ>
int launch(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const PrefillParams& p, int grid,
           cudaStream_t stream) {
    constexpr int smem = smem_bytes<D, QQ>();
    static_assert(smem <= 232448, "");
    static SmemLimit limit;
    cudaError_t e = limit.allow(prefill_attn_kernel<D, NAIVE, QQ>, smem);
    if (e != cudaSuccess) return set_cuda_error(e, "cc_prefill_attention: shared memory attribute");
    prefill_attn_kernel<D, NAIVE, QQ><<<grid, NTHREADS, smem, stream>>>(tq, tk, tv, p);
    e = cudaGetLastError();
    return e == cudaSuccess ? CC_OK : set_cuda_error(e, "cc_prefill_attention launch");
}

template <int D, bool NAIVE>
int launch_group(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const PrefillParams& p, int grid,
                 cudaStream_t stream) {
    switch (p.QB) {
        case 128: return launch<D, NAIVE, 32>(tq, tk, tv, p, grid, stream);
        case 64:  return launch<D, NAIVE, 16>(tq, tk, tv, p, grid, stream);
        case 32:  return launch<D, NAIVE, 8>(tq, tk, tv, p, grid, stream);
        default:  return launch<D, NAIVE, 4>(tq, tk, tv, p, grid, stream);
    }
}

}  // namespace

unsigned long long prefill_attention_workspace_impl(int S, int Hkv, int G, int obs_len, int n_windows) {
    if (S <= 0 || Hkv <= 0 || G <= 0 || G > 8 || n_windows < 0 || n_windows > MAX_WINDOWS) return 0;
    const Plan pl = make_plan(S, Hkv, G, obs_len, n_windows);
    return (uint64_t)(pl.col_floats + pl.obs_floats + pl.band_floats) * sizeof(float) + 256;
}

int prefill_attention_impl(const CcPrefillAttnArgs* a, cudaStream_t stream) {
    if (!a || !a->q || !a->k || !a->v || !a->y) return set_error(CC_ERR_INVALID_ARG, "cc_prefill_attention: null argument");
    const int S = a->seq_len, Hkv = a->n_kv_heads, G = a->q_per_kv, D = a->head_dim;
    if (S <= 0 || Hkv <= 0) return set_error(CC_ERR_INVALID_ARG, "cc_prefill_attention: empty problem");
    if ((D != 64 && D != 128) || G < 1 || G > 8)
        return set_error(CC_ERR_UNSUPPORTED_SHAPE, "cc_prefill_attention: head_dim must be 64 or 128 and q_per_kv <= 8");
    if (a->n_windows < 0 || a->n_windows > MAX_WINDOWS)
        return set_error(CC_ERR_INVALID_ARG, "cc_prefill_attention: at most 4 band windows");
    if (a->attn_mode != CC_ATTN_NAIVE_BF16 && a->attn_mode != CC_ATTN_MATH_FP32)
        return set_error(CC_ERR_INVALID_ARG, "cc_prefill_attention: bad attn_mode");
    if (a->stats_bf16 != 0 && a->stats_bf16 != 1) return set_error(CC_ERR_INVALID_ARG, "cc_prefill_attention: stats_bf16 is 0 or 1");
    const long long strides[] = {a->q_stride_s, a->q_stride_h, a->k_stride_s, a->k_stride_h, a->v_stride_s,
                                 a->v_stride_h, a->y_stride_s, a->y_stride_h};
    for (long long s : strides)
        if (s <= 0 || (s % 8) != 0) return set_error(CC_ERR_INVALID_ARG, "cc_prefill_attention: strides must be positive multiples of 8 elements");
    const uintptr_t ptrs[] = {(uintptr_t)a->q, (uintptr_t)a->k, (uintptr_t)a->v, (uintptr_t)a->y};
    for (uintptr_t q : ptrs)
        if (q % 16) return set_error(CC_ERR_INVALID_ARG, "cc_prefill_attention: tensors must be 16-byte aligned");
    const bool stats = a->col_sum != nullptr;
    if (!stats && (a->obs_sum || a->band_sum || a->n_windows))
        return set_error(CC_ERR_INVALID_ARG, "cc_prefill_attention: obs_sum / band_sum need col_sum");
    if (a->n_windows && !a->band_sum) return set_error(CC_ERR_INVALID_ARG, "cc_prefill_attention: band_sum missing");

    const int obs_len = (stats && a->obs_sum) ? (a->obs_len > S ? S : a->obs_len) : 0;
    const Plan pl = make_plan(S, Hkv, G, obs_len, stats ? a->n_windows : 0);
    PrefillParams p;
    p.y = (__nv_bfloat16*)a->y; p.y_stride_s = a->y_stride_s; p.y_stride_h = a->y_stride_h;
    p.S = S; p.S_pad = pl.S_pad; p.Hkv = Hkv; p.G = G; p.QB = pl.QB; p.n_qtiles = pl.n_qtiles;
    p.obs_start = obs_len > 0 ? S - obs_len : S;
    p.first_obs_tile = pl.first_obs_tile; p.n_obs_tiles = pl.n_obs_tiles;
    p.n_windows = stats ? a->n_windows : 0;
    for (int w = 0; w < MAX_WINDOWS; ++w)      // no rows at all from 0 down, every row from S on
        p.windows[w] = w < p.n_windows ? (a->windows[w] < 0 ? 0 : a->windows[w] > S ? S : a->windows[w]) : 0;
    p.scale = (float)(1.0 / sqrt((double)D));
    p.stats = stats ? 1 : 0;
    p.part_col = p.part_obs = p.part_band = nullptr;
    if (stats) {
        const uint64_t need = prefill_attention_workspace_impl(S, Hkv, G, obs_len, p.n_windows);
        if (!a->workspace || a->workspace_bytes < need)
            return set_error(CC_ERR_INVALID_ARG, "cc_prefill_attention: workspace too small (see cc_prefill_attention_workspace)");
        float* w = (float*)(((uintptr_t)a->workspace + 255) & ~(uintptr_t)255);
        p.part_col = w;
        p.part_obs = w + pl.col_floats;
        p.part_band = p.part_obs + pl.obs_floats;
    }
    CUtensorMap tq, tk, tv;
    int rc;
    if ((rc = make_map(&tq, a->q, D, S, Hkv * G, a->q_stride_s, a->q_stride_h, pl.QB / 4, G)) != CC_OK) return rc;
    if ((rc = make_map(&tk, a->k, D, S, Hkv, a->k_stride_s, a->k_stride_h, BN, 1)) != CC_OK) return rc;
    if ((rc = make_map(&tv, a->v, D, S, Hkv, a->v_stride_s, a->v_stride_h, BN, 1)) != CC_OK) return rc;
    const int grid = pl.n_qtiles * Hkv;
    const bool naive = a->attn_mode == CC_ATTN_NAIVE_BF16;
    if (D == 128) rc = naive ? launch_group<128, true>(tq, tk, tv, p, grid, stream) : launch_group<128, false>(tq, tk, tv, p, grid, stream);
    else          rc = naive ? launch_group<64, true>(tq, tk, tv, p, grid, stream) : launch_group<64, false>(tq, tk, tv, p, grid, stream);
    if (rc != CC_OK) return rc;
    if (stats) {
        dim3 rgrid((S + RED_THREADS - 1) / RED_THREADS, Hkv);
        auto reduce = a->stats_bf16 ? prefill_reduce_kernel<true> : prefill_reduce_kernel<false>;
        reduce<<<rgrid, RED_THREADS, 0, stream>>>(p, a->col_sum, obs_len > 0 ? a->obs_sum : nullptr, a->band_sum,
                                                  obs_len > 0 ? 1.0f / (float)obs_len : 0.f);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return set_cuda_error(e, "cc_prefill_attention reduce launch");
    }
    return CC_OK;
}

}  // namespace cc
