// moe_tc_kernels.cu -- the experts of a prompt portion as two grouped products on the tensor cores (bf16 weights, fp32
// accumulation), sized on the device: act = unit(W_gu x) over the gathered token rows, then y = W_d act.
//
// What it replaces: one library product pair per expert on gathered copies of the rows, launched after the group sizes had
// come to the host; at 2048 tokens and 16 experts of 1536 that was 32 products of ~450 rows with the GPU idle before and
// between them, and the gate and up rows made a round trip through memory in fp32.
//
// A persistent CTA per SM walks 128 x 256 tiles, expert by expert, the row tiles of one weight tile next to one another so
// that the weights are read from HBM once.  Both operands come by TMA: the token rows are gathered by a copy kernel first
// (fetched row by row with cp.async inside the product they held the tensor pipe at 23 %: 237 us where the TMA form takes
// 96 and the copy 10; 2048 tokens, 4 of 16 experts of 1536, width 2048).  A gated tile holds 128 gate columns beside the 128 up columns they
// belong to, so the unit is applied on the way out of tensor memory, four warps emptying one accumulator while the next tile
// fills the other; fp32 results go by way of shared memory, so that rows are stored as whole lines (the unit's bf16 results that way:
// 10 us slower at 400 to 512 tokens).  Bound: the 64 bytes per clock that an SM takes from L2; a 128 x 256 x 64 stage is 48 KB (768 cycles) for
// 512 cycles of MMAs.  The whole mixture with a shared expert of 2048 in a graph, four turns of each side that agree within 1 %: results 16
// bytes of a row at a time and MMAs issued by one thread 251 us, this 241; 4096 tokens 434 / 408; experts of 1000 221 / 208.6; 1024 tokens
// 151 / 147.7, 300 108.4 / 105.2, 64 97.0 / 94.5.  Pairs of CTAs (cta_group::2) on 256 x 256 tiles, which read half of the weights each, beside
// 240, 416, 207 and 146 of this form: 254 at 2048 tokens, 422 at 4096, 215 with experts of 1000 and 158 at 1024.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "../../../include/cc_b200_seq.h"
#include "launch.cuh"
#include "tensor_map.cuh"

namespace ccs {

int fail(int code, const char* msg);
int cuda_check(const char* where);

namespace {

typedef __nv_bfloat16 bf16;

constexpr int BM = 128, BN = 256, BK = 64;      // BK: one 128-byte swizzled row of a tile
constexpr int STAGES = 4, A_BYTES = BM * 128, B_BYTES = BN * 128, STAGE_BYTES = A_BYTES + B_BYTES, OUT_BYTES = 4 * 32 * 128;
constexpr int W_OUT = 4, W_MMA = 4, W_TMA = 5, THREADS = 192;   // warps 0-3 empty tensor memory
constexpr uint32_t WAIT_LIMIT = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done != 0;
}
// Bounded: a wait that runs out raises `failed`; every later wait of the CTA then gives up at once and what it stores is NaN.
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
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {   // 128-byte swizzle, rows of 128 bytes, descriptor version 1
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(one));
    return one != 0;
}
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\ntcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                 ::"r"(d), "l"(a), "l"(b), "r"(IDESC), "r"(acc) : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* tm, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(tm), "r"(bar), "r"(x), "r"(y) : "memory");
}
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
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float sigmoidf_(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float unit_act(float z, int kind) {
    switch (kind) {
        case CC_ACT_GELU_TANH: return 0.5f * z * (1.0f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
        case CC_ACT_SILU: return z * sigmoidf_(z);
        case CC_ACT_TANH: return tanhf(z);
        case CC_ACT_SIGMOID: return sigmoidf_(z);
        case CC_ACT_RELU_SQ: { const float r = fmaxf(z, 0.f); return r * r; }
        default: return z;
    }
}

struct Grouped {
    const int32_t* counts;    // rows per expert
    void* out;                // first: bf16 [rows, F]; second: fp32 [rows, E]
    int n, K, N, w_rows;      // experts, inner size, output columns, weight rows per expert
    int kind;
};

// The tiles in order: expert, column tile, row tile.  A role walks the ids blockIdx.x, + gridDim.x, ...
struct Walk {
    int e, first_row, first_id, rows, row_tiles, col_tiles;
    const int32_t* counts;
    int n;
    __device__ __forceinline__ void start(const int32_t* c, int n_experts, int ct) {
        counts = c; n = n_experts; col_tiles = ct;
        e = -1; first_row = 0; first_id = 0; rows = 0; row_tiles = 0;
    }
    // moves on to the expert of tile `id`; false when there is none
    __device__ __forceinline__ bool seek(int id) {
        while (e < 0 || id >= first_id + row_tiles * col_tiles) {
            if (e >= 0) { first_id += row_tiles * col_tiles; first_row += rows; }
            if (++e >= n) return false;
            rows = counts[e];
            row_tiles = (rows + BM - 1) / BM;
        }
        return true;
    }
    __device__ __forceinline__ int row_tile(int id) const { return (id - first_id) % row_tiles; }
    __device__ __forceinline__ int col_tile(int id) const { return (id - first_id) / row_tiles; }
};

struct Small {
    uint64_t bars[2 * STAGES + 5];     // full, empty, accumulator full[2], empty[2], everything done
    uint32_t tmem;
    int failed;
};

// xs[r] = h[perm[r]] for the rows that the experts have
__global__ void __launch_bounds__(256) moe_rows_kernel(const uint4* __restrict__ h, const int32_t* perm, const int32_t* counts, int n, uint4* __restrict__ xs, int vecs) {
    int rows = 0;
    for (int e = 0; e < n; ++e) rows += counts[e];
    const long long total = (long long)rows * vecs;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int r = (int)(i / vecs);
        xs[i] = h[(size_t)perm[r] * vecs + (i - (long long)r * vecs)];
    }
}

// GATED: 128 gate and 128 up columns per tile, out = unit(gate) up.  UNIT: the first product (bf16 out through the unit),
// otherwise the second (fp32 out).
template <bool UNIT, bool GATED>
__global__ void __launch_bounds__(THREADS, 1) moe_tc_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_a, const Grouped p) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];      // the stages, results on their way out, then Small: no static shared memory in front of them
    uint8_t* const outs = smem_raw + STAGES * STAGE_BYTES;
    Small& sm = *reinterpret_cast<Small*>(outs + OUT_BYTES);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const uint32_t base = smem_u32(smem_raw), bar = smem_u32(sm.bars);
    const uint32_t FULL = bar, EMPTY = bar + 8 * STAGES, ACC_FULL = bar + 16 * STAGES, ACC_EMPTY = ACC_FULL + 16, DONE = ACC_EMPTY + 16;
    volatile int* const failed = &sm.failed;
    if (tid == 0) {
        *failed = 0;
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(FULL + 8 * s, 1);
            mbar_init(EMPTY + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(ACC_FULL + 8 * b, 1);
            mbar_init(ACC_EMPTY + 8 * b, W_OUT);
        }
        mbar_init(DONE, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = sm.tmem;
    pdl_wait_release();

    const int cols = GATED ? BN / 2 : BN;          // output columns of a tile
    const int k_iters = (p.K + BK - 1) / BK;
    Walk w;
    w.start(p.counts, p.n, (p.N + cols - 1) / cols);

    if (warp == W_TMA) {
        if (lane == 0) {
            int it = 0;
            for (int id = blockIdx.x; w.seek(id) && !*failed; id += gridDim.x) {
                const int c0 = w.col_tile(id) * cols, r0 = w.first_row + w.row_tile(id) * BM;
                const int b0 = w.e * p.w_rows + c0, b1 = GATED ? b0 + p.N : b0 + BN / 2;
                for (int k = 0; k < k_iters; ++k, ++it) {
                    const int s = it % STAGES;
                    if (it >= STAGES) mbar_wait(EMPTY + 8 * s, (it / STAGES - 1) & 1, failed);
                    if (*failed) break;
                    const uint32_t sA = base + s * STAGE_BYTES, sB = sA + A_BYTES;
                    mbar_expect(FULL + 8 * s, STAGE_BYTES);
                    tma_load(sB, &tm_w, k * BK, b0, FULL + 8 * s);
                    tma_load(sB + B_BYTES / 2, &tm_w, k * BK, b1, FULL + 8 * s);
                    tma_load(sA, &tm_a, k * BK, r0, FULL + 8 * s);
                }
            }
            for (int m = it < STAGES ? 0 : it - STAGES; m < it; ++m) mbar_wait_out(FULL + 8 * (m % STAGES), (m / STAGES) & 1);
        }
        __syncwarp();
    } else if (warp == W_MMA) {
        int s = 0, n_tile = 0;
        uint32_t turn = 0;
        const uint64_t a_desc = smem_desc(base), b_desc = smem_desc(base + A_BYTES);
        // the flag is the same for all lanes, which elect_one wants together
        for (int id = blockIdx.x; w.seek(id) && !__any_sync(0xffffffffu, *failed); id += gridDim.x, ++n_tile) {
            const int b = n_tile & 1;
            if (n_tile >= 2) mbar_wait(ACC_EMPTY + 8 * b, (n_tile / 2 - 1) & 1, failed);
            for (int k = 0; k < k_iters; ++k) {
                mbar_wait(FULL + 8 * s, turn, failed);
                __syncwarp();
                fence_after();
                if (elect_one()) {
                    const uint64_t at = s * (STAGE_BYTES >> 4);
#pragma unroll
                    for (int kk = 0; kk < BK / 16; ++kk) mma_ss(tmem + b * BN, a_desc + at + 2 * kk, b_desc + at + 2 * kk, k > 0 || kk > 0);
                    mma_commit(EMPTY + 8 * s);
                    if (k == k_iters - 1) mma_commit(ACC_FULL + 8 * b);
                }
                __syncwarp();
                if (++s == STAGES) { s = 0; turn ^= 1; }
            }
        }
        if (elect_one()) mma_commit(DONE);
        __syncwarp();
        mbar_wait_out(DONE, 0);
    } else {
        int n_tile = 0;
        const uint32_t lanes = (uint32_t)(warp * 32) << 16;
        uint8_t* const mine = outs + warp * 32 * 128;           // 32 rows of 128 bytes, 16-byte chunks swizzled by the row
        for (int id = blockIdx.x; w.seek(id); id += gridDim.x, ++n_tile) {
            const int b = n_tile & 1, c0 = w.col_tile(id) * cols, row0 = w.row_tile(id) * BM + warp * 32;
            mbar_wait(ACC_FULL + 8 * b, (n_tile / 2) & 1, failed);
            __syncwarp();
            fence_after();
            const float bad = *failed ? NAN : 0.f;
            const int live_rows = w.rows - row0;
            const size_t at = (size_t)(w.first_row + row0) * p.N + c0;
#pragma unroll 1
            for (int c = 0; c < cols && live_rows > 0; c += 32) {
                float v[32], u[32];
                tmem_ld32(tmem + lanes + b * BN + c, v);
                if (GATED) tmem_ld32(tmem + lanes + b * BN + BN / 2 + c, u);
                tmem_wait_ld();
                if constexpr (UNIT) {
                    if (lane < live_rows) {
#pragma unroll
                        for (int e = 0; e < 32; e += 8) {
                            if (c0 + c + e < p.N) {             // N is a multiple of 8
                                __align__(16) bf16 o[8];
#pragma unroll
                                for (int i = 0; i < 8; ++i) {
                                    float x = unit_act(v[e + i], p.kind);
                                    if (GATED) x *= u[e + i];
                                    o[i] = __float2bfloat16_rn(x + bad);
                                }
                                *reinterpret_cast<uint4*>((bf16*)p.out + at + (size_t)lane * p.N + c + e) = *reinterpret_cast<const uint4*>(o);
                            }
                        }
                    }
                } else {
                    // by way of shared memory, eight lanes to a row: whole 128-byte lines
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        *reinterpret_cast<float4*>(mine + lane * 128 + ((q ^ (lane & 7)) << 4)) =
                            make_float4(v[4 * q] + bad, v[4 * q + 1] + bad, v[4 * q + 2] + bad, v[4 * q + 3] + bad);
                    __syncwarp();
                    const int chunk = lane & 7, col = c + 4 * chunk;
                    if (c0 + col < p.N)
#pragma unroll
                        for (int r = lane >> 3; r < 32; r += 4)
                            if (r < live_rows)
                                *reinterpret_cast<float4*>((float*)p.out + at + (size_t)r * p.N + col) =
                                    *reinterpret_cast<const float4*>(mine + r * 128 + ((chunk ^ (r & 7)) << 4));
                }
                __syncwarp();
            }
            fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(ACC_EMPTY + 8 * b);
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

template <bool UNIT, bool GATED>
int launch_tc(const CUtensorMap& tw, const CUtensorMap& ta, const Grouped& p, int grid, cudaStream_t st) {
    auto kern = moe_tc_kernel<UNIT, GATED>;
    const int smem = STAGES * STAGE_BYTES + OUT_BYTES + (int)sizeof(Small);
    static SmemLimit limit;
    const cudaError_t e = limit.allow(kern, smem);
    if (e != cudaSuccess) return fail(CC_SEQ_ERR_CUDA, cudaGetErrorString(e));
    launch_under(kern, dim3(grid), dim3(THREADS), smem, st, tw, ta, p);
    return cuda_check("moe_tc_kernel");
}

}  // namespace
}  // namespace ccs

using namespace ccs;

extern "C" int cc_seq_moe_grouped(const CcSeqMoeGrouped* a, void* stream) {
    if (!a || !a->wgu || !a->wd || !a->h || !a->perm || !a->counts || !a->xs || !a->act || !a->y || a->n < 1 || a->F < 1 || a->E < 1 || a->M < 1 ||
        a->kind < CC_ACT_NONE || a->kind > CC_ACT_LAST)
        return fail(CC_SEQ_ERR_INVALID_ARG, "moe_grouped: bad argument");
    const uintptr_t all = (uintptr_t)a->wgu | (uintptr_t)a->wd | (uintptr_t)a->h | (uintptr_t)a->xs | (uintptr_t)a->act | (uintptr_t)a->y;
    const long long wide = (long long)a->n * (a->gated ? 2 : 1) * a->F;
    if (a->F % 8 || a->E % 8 || (all & 15) || wide > 0x7fffffffLL - 256 || (long long)a->n * a->E > 0x7fffffffLL - 256)
        return fail(CC_SEQ_ERR_UNSUPPORTED_SHAPE, "moe_grouped: rows of whole 16-byte vectors on 16-byte boundaries expected");
    cudaStream_t st = (cudaStream_t)stream;
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    CUtensorMap tgu, td, tx, ta;
    if (!map_rows(&tgu, a->wgu, wide, a->E) || !map_rows(&td, a->wd, (long long)a->n * a->E, a->F) || !map_rows(&tx, a->xs, a->M, a->E) ||
        !map_rows(&ta, a->act, a->M, a->F))
        return fail(CC_SEQ_ERR_CUDA, "moe_grouped: cuTensorMapEncodeTiled failed or is not available");
    int rc;
    const long long row_tiles = (a->M + BM - 1) / BM + (a->n < a->M ? a->n : a->M);      // at most
    auto grid = [&](int N, int cols) {
        const long long t = row_tiles * ((N + cols - 1) / cols);
        return (int)(t < sms ? t : sms);
    };
    const long long copies = ((long long)a->M * (a->E / 8) + 255) / 256;
    moe_rows_kernel<<<(unsigned)(copies < 16 * sms ? copies : 16 * sms), 256, 0, st>>>((const uint4*)a->h, a->perm, a->counts, a->n, (uint4*)a->xs, a->E / 8);
    if ((rc = cuda_check("moe_rows_kernel"))) return rc;
    const Grouped up = {a->counts, a->act, a->n, a->E, a->F, (a->gated ? 2 : 1) * a->F, a->kind};
    rc = a->gated ? launch_tc<true, true>(tgu, tx, up, grid(a->F, BN / 2), st) : launch_tc<true, false>(tgu, tx, up, grid(a->F, BN), st);
    if (rc) return rc;
    const Grouped down = {a->counts, a->y, a->n, a->F, a->E, a->E, CC_ACT_NONE};
    return launch_tc<false, false>(td, ta, down, grid(a->E, BN), st);
}
