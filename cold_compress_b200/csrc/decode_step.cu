// decode_step.cu -- the fused per-layer decode step for sm_100a.
//
// One launch = eviction decision -> in-place slot overwrite -> masked attention over the live
// cache slots -> GQA pooling -> eviction-score update, for every KV head of one layer.
// Replaces the reference's decode branch of Attention.forward (model.py:389-427):
// KVCache.update_kv (cache.py:314-364), scaled_dot_product_attention
// (attention_utils.py:8-54), the group mean (model.py:413-418) and KVCache.update_state
// (cache.py:690-723), which run there as ~25 ATen ops and materialise 4x K/V copies.
//
// Shape of the launch (HBM-latency bound: 4 MiB of K/V per layer at L=1024):
//   * one thread-block CLUSTER per KV head, C CTAs (<=16) per cluster; the cache rows of the head
//     are cut into chunks of CH rows (16/32/64) dealt round-robin to the CTAs of the cluster, so
//     a head whose live slots are a prefix (hybrid, caches still filling) stays balanced
//     -> Hkv*C CTAs (128 of 148 SMs for Llama-3-8B);
//   * the K and V rows of each chunk are streamed by the TMA engine (cp.async.bulk) into
//     a shared-memory ring, as many chunks in flight as the ring holds from the first instruction;
//   * three DSMEM all-to-all exchanges per step: {arg-min candidate, row max}, {softmax sum},
//     {P.V partials}; the first one carries both the eviction decision and the softmax max, so
//     the evicted slot's old logit is excluded / the new token's logit included without a
//     second pass over K;
//   * what bounds it is the chain of dependent waits, not bytes, so the chain is kept short: rows and policy state are in L2
//     when the launch may read them (asked for before griddepcontrol.wait), all loads of the first phases are requested
//     together, warps reduce with the warp reduction instruction instead of butterflies, every softmax warp owns one query
//     head and sends its own sums, and the P.V phase adds nothing up across lanes.  32 steps in a graph, us a step, before and
//     with all of it: 64 sliding slots 8.2 and 5.4, 1024 heavy-hitter slots 10.9 and 7.8, 512 l2 slots 15.2 and 8.2;
//   * arithmetic order is the bit-reproducible definition in common.cuh (canonical dot tree,
//     det_expf, 2^-40 fixed-point sum), so eviction indices do not depend on C, CH or the
//     thread count.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>

#include "../../include/cc_b200.h"
#include "common.cuh"
#include "internal.h"

namespace cc {

#ifndef CC_DECODE_THREADS
#define CC_DECODE_THREADS 256
#endif
constexpr int kThreads = CC_DECODE_THREADS;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxCluster = 16;
constexpr int kMaxG = 8;
constexpr int kRecWords = 2 + 2 * kMaxG;  // X1 record: key64, lmax[G], candlogit[G]
constexpr uint64_t kNoKey = ~0ull;

struct SmemLayout {
    uint32_t kring, vring, lg, red, yx, rec, sums, x0, maskb, bars, misc, total;
};

struct DecodeParams {
    SmemLayout lay;     // shared-memory carve-up, computed once on the host
    CcCacheState st;
    CcDecodeArgs a;
    int ch_shift;       // log2(rows per chunk)
    int max_local_chunks;  // chunks dealt to rank 0 (the most any CTA gets)
    int n_stages;       // ring depth for K and for V
    int lg_stride;      // floats per query head in the logit/prob array
    float scale;        // (float)(1/sqrt(D))
    int c_shift;        // log2(cluster size)
    unsigned long long* trace;  // diagnostics: [gridDim.x][16] globaltimer stamps (NULL = off)
};

// misc area, indices in 4-byte words
enum : int {
    kMiscNewLg = 0,     // [kMaxG] logits of the new token
    kMiscWarpKey = 8,   // [kWarps] u64
    kMiscWarpMax = 24,  // [kWarps] largest key norm
    kMiscRowMax = 32,   // [kWarps][kMaxG] largest logit of a warp's rows, without the candidate's
    kMiscCandLg = 96,   // [kMaxG] logits of the candidate: a copy, the softmax overwrites the row's own while others still read
    kMiscWords = 104,
};

__host__ __device__ inline uint32_t align_up(uint32_t x, uint32_t a) { return (x + a - 1) / a * a; }

__host__ __device__ inline SmemLayout make_layout(int D, int G, int chunk_rows, int local_rows, int n_stages, int lg_stride) {
    SmemLayout s;
    uint32_t off = 0;
    const uint32_t chunk_bytes = chunk_rows * D * 2;
    s.kring = off; off += align_up(n_stages * chunk_bytes, 128);
    s.vring = off; off += align_up(n_stages * chunk_bytes, 128);
    s.lg = off;    off += align_up(G * lg_stride * 4, 128);
    s.red = off;   off += kWarps * G * D * 4;
    s.yx = off;    off += G * D * 4;
    s.rec = off;   off += kMaxCluster * kRecWords * 4;
    s.sums = off;  off += kMaxCluster * kMaxG * 8;
    s.x0 = off;    off += 128;
    s.maskb = off; off += align_up(local_rows, 128);
    s.bars = off;  off += align_up((2 * n_stages + 4) * 8, 128);  // K ring, V ring, 4 exchange barriers
    s.misc = off;  off += kMiscWords * 4;
    s.total = off;
    return s;
}

// hybrid per-head decision (reference cache.py:896-950)
enum : int { kHybAppend = 0, kHybEvict = 1, kHybDrop = 2 };

__device__ __forceinline__ void stamp(const DecodeParams& p, int k) {
    if (p.trace && threadIdx.x == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        p.trace[(size_t)blockIdx.x * 16 + k] = t;
    }
}

template <int D, int G, int POLICY, bool NAIVE>
__global__ void __launch_bounds__(kThreads, 2)
cc_decode_kernel(const __grid_constant__ DecodeParams p) {
    constexpr int LPR = D / 8;           // lanes per cache row (16-byte slice each)
    constexpr int RPW = 32 / LPR;        // rows per warp iteration
    constexpr int CPL = D / 32;          // P.V phase: value columns per lane
    constexpr int WPG = kWarps / G;      // softmax: warps that share a query head's rows (one head per warp)
    constexpr uint32_t kRowBytes = D * 2;
    constexpr bool hybrid = POLICY == CC_POLICY_HYBRID;

    extern __shared__ __align__(1024) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int li = lane % LPR, sub = lane / LPR;
    const int csh = p.c_shift, C = 1 << csh, rank = (int)cluster_ctarank();
    const bool solo = C == 1;            // the head's rows in one CTA: nothing to exchange
    const int h = blockIdx.x >> csh;
    const CcCacheState& st = p.st;
    const int L = st.max_cache_length, H = st.n_kv_heads;
    const int chs = p.ch_shift, CH = 1 << chs;
    const uint32_t chunk_bytes = CH * kRowBytes;
    const int phases = p.a.phases;
    const bool do_evict = phases & CC_PHASE_EVICT_FILL, do_attend = phases & CC_PHASE_ATTEND,
               do_score = phases & CC_PHASE_SCORE;
    const int NS = p.n_stages, stride = p.lg_stride;
    // shared (cross-head) state is read by every cluster and written by one: order with an epoch barrier
    // heavy hitter with a history window (W > 1): the shared step counter selects the ring column every head writes
    const bool hh_ring = POLICY == CC_POLICY_HEAVY_HITTER && st.history_window > 1;
    const bool needs_epoch = (do_evict && (POLICY == CC_POLICY_RECENT_GLOBAL || POLICY == CC_POLICY_L2)) ||
                             ((hybrid || hh_ring) && (do_evict || do_score));

    // chunk-cyclic ownership: local chunk j <-> global chunk rank + j*C; local row lr = j*CH + r
    const int n_chunks_total = (L + CH - 1) >> chs;
    const int nlc = n_chunks_total > rank ? (n_chunks_total - rank + C - 1) >> csh : 0;
    const int local_rows = nlc << chs;
    auto slot_of = [&](int lr) { return ((((lr >> chs) << csh) + rank) << chs) + (lr & (CH - 1)); };

    const SmemLayout& lay = p.lay;
    uint8_t* kring = smem + lay.kring;
    uint8_t* vring = smem + lay.vring;
    float* lg = reinterpret_cast<float*>(smem + lay.lg);
    float* red = reinterpret_cast<float*>(smem + lay.red);
    float* yx = reinterpret_cast<float*>(smem + lay.yx);
    uint32_t* rec = reinterpret_cast<uint32_t*>(smem + lay.rec);
    unsigned long long* sums = reinterpret_cast<unsigned long long*>(smem + lay.sums);
    float* x0 = reinterpret_cast<float*>(smem + lay.x0);
    uint8_t* maskb = smem + lay.maskb;
    uint64_t* kbar = reinterpret_cast<uint64_t*>(smem + lay.bars);
    uint64_t* vbar = kbar + NS;
    uint64_t* xbar = vbar + NS;  // [0] X0 (L2 max), [1] X1, [2] X2, [3] X3: single-use exchange barriers
    float* misc = reinterpret_cast<float*>(smem + lay.misc);
    uint32_t* miscu = reinterpret_cast<uint32_t*>(misc);

    stamp(p, 0);
    constexpr int NW = 2 + 2 * G;  // words of an X1 record
    if (tid == 0) {
        for (int s = 0; s < 2 * NS + 4; ++s) mbar_init(&kbar[s], 1);
        mbar_fence_init();
        // every exchange delivers a known number of bytes into this CTA: arm the barriers right away
        // (only the exchanges this launch performs: an armed barrier nobody completes is a synccheck finding)
        if (!solo) {
            if (POLICY == CC_POLICY_L2 && do_evict) mbar_expect_tx(&xbar[0], (uint32_t)C * 4);
            mbar_expect_tx(&xbar[1], (uint32_t)C * NW * 4);
            if (do_attend) {
                mbar_expect_tx(&xbar[2], (uint32_t)C * G * WPG * 8);
                mbar_expect_tx(&xbar[3], (uint32_t)G * D * 4);
            }
        }
    }
    // B0: this CTA has started and its exchange barriers exist; peers wait for this before they send
    if (!solo) cluster_arrive_release();
    bool b0_waited = solo;
    // Without the promise that the predecessor leaves this cache alone nothing of it is read before the predecessor has
    // ended; the launch, the barriers and the cluster's start above run under it all the same.
    const bool ahead = p.a.flags & CC_FLAG_OVERLAP_PREDECESSOR;
    const uint16_t* kc = reinterpret_cast<const uint16_t*>(st.k_cache) + (size_t)h * L * D;
    const uint16_t* vc = reinterpret_cast<const uint16_t*>(st.v_cache) + (size_t)h * L * D;
    auto chunk_rows_valid = [&](int j) { return min(CH, L - ((((j << csh) + rank)) << chs)); };
    auto chunk_at = [&](const uint16_t* base, int j) { return base + ((size_t)((j << csh) + rank) << chs) * D; };
    const int pos_row = (st.pos_heads == 1) ? 0 : h;
    const int32_t* posp = st.pos + (size_t)pos_row * L;
    const double* hist = reinterpret_cast<const double*>(st.attn_history_num) + (size_t)h * L;   // heavy hitter with W = 1
    const int32_t* den = st.attn_history_denom + (size_t)h * L;
    const bool hh_sum = POLICY == CC_POLICY_HEAVY_HITTER && !hh_ring;
    const int s0 = slot_of(tid);         // this thread's first row
    const bool in0 = tid < local_rows && s0 < L;
    const uint16_t* qp = reinterpret_cast<const uint16_t*>(p.a.q) + (size_t)h * G * D + li * 8;
    const uint16_t* knp = reinterpret_cast<const uint16_t*>(p.a.k_new) + (size_t)h * D + li * 8;
    const uint16_t* vrow_new = reinterpret_cast<const uint16_t*>(p.a.v_new) + (size_t)h * D;
    if (!ahead) {
        // What will be read is asked for in L2: a hint, which takes no value, so that after the wait the chain below meets
        // L2 and not DRAM.  (Rows of a hybrid head that are live are known from memory only.)
        if constexpr (!hybrid) {
            const int pre = do_attend ? min(NS, nlc) : 0;
            if (tid < 2 * pre) l2_prefetch_bulk(chunk_at(tid & 1 ? vc : kc, tid >> 1), chunk_rows_valid(tid >> 1) * kRowBytes);
        }
        if (in0) {
            l2_prefetch_line(posp + s0);
            l2_prefetch_line(st.mask + (size_t)h * L + s0);
            if (POLICY == CC_POLICY_L2 && do_evict) l2_prefetch_line(reinterpret_cast<const uint16_t*>(st.key_norm) + (size_t)h * L + s0);
            if (hh_sum) {
                l2_prefetch_line(hist + s0);
                l2_prefetch_line(den + s0);
            }
        }
    }
    if (!ahead) pdl_wait();

    // ---- hybrid: per-head decision from scalars (every CTA of the cluster computes the same)
    int hyb_mode = kHybAppend, hyb_bits = 0, hyb_cts = 0, hyb_rw = 0;
    int64_t hyb_counter = 0;
    int live_limit = L;  // slots >= live_limit cannot be live: their chunks are never loaded
    bool last_live = false;
    const bool is_punc = hybrid && (p.a.is_punc_dev ? p.a.is_punc_dev[0] != 0 : p.a.is_punc != 0);
    if constexpr (hybrid) {
        hyb_bits = st.hyb_strategy_bits[h];
        hyb_cts = st.cache_cts[h];
        hyb_rw = (hyb_bits & CC_HYB_WINDOW) ? st.hyb_recent_window[h] : 0;
        if (st.attn_counter) hyb_counter = st.attn_counter[0];
        if (do_evict) {
            if (((hyb_bits & CC_HYB_PUNC) && is_punc) || (hyb_bits & CC_HYB_FULL)) {
                hyb_mode = kHybAppend;
            } else {
                int budget = st.global_tokens;
                if ((hyb_bits & CC_HYB_SPECIAL) && st.num_special) budget += st.num_special[0];
                if ((hyb_bits & CC_HYB_PUNC) && st.num_punc) budget += st.num_punc[0];
                if (hyb_bits & CC_HYB_WINDOW) budget += st.hyb_recent_window[h];
                if (hyb_bits & CC_HYB_HEAVY_HITTER) budget += st.hyb_heavy_budget[h];
                hyb_mode = hyb_cts < budget ? kHybAppend
                         : (hyb_bits & (CC_HYB_HEAVY_HITTER | CC_HYB_WINDOW)) ? kHybEvict : kHybDrop;
            }
        }
        live_limit = min(L, hyb_cts + ((do_evict && hyb_mode == kHybAppend) ? 1 : 0));
        last_live = live_limit == L && st.mask[(size_t)h * L + L - 1] != 0;
    }
    int32_t hh_cts = 0;   // cache_cts before this step (thresholded history compares against 1 / cache_cts)
    if (hh_ring) {
        hyb_counter = st.attn_counter[0];
        hh_cts = st.cache_cts[0];
    }
    const int live_chunks_total = (live_limit + CH - 1) >> chs;
    const int nlc_live = do_attend ? (live_chunks_total > rank ? (live_chunks_total - rank + C - 1) >> csh : 0) : 0;
    const int live_rows = nlc_live << chs;

    // ---- 0. barriers + as many K/V chunks in flight as the ring holds
    // (The keys of a CTA with one short chunk go straight to registers below: they are there when the candidate is, half a
    // microsecond before a bulk copy of the same rows.  32 steps in a graph: 64 sliding slots 185 -> 174 us, 1024 heavy-hitter slots 260 -> 251.)
    constexpr int UR = G >= 7 ? 2 : 4;     // row pairs of a warp per pass (registers: two CTAs per SM, so that the next launch fits beside this one)
    const bool direct = !ahead && nlc_live == 1 && CH <= UR * kWarps * RPW;
    if (tid == 0) {
        fence_proxy_async();
        const int pre = min(NS, nlc_live);
        for (int j = 0; j < pre && !direct; ++j) {
            const uint32_t bytes = chunk_rows_valid(j) * kRowBytes;
            mbar_expect_tx(&kbar[j], bytes);
            tma_load_1d(kring + j * chunk_bytes, chunk_at(kc, j), bytes, &kbar[j]);
        }
        for (int j = 0; j < pre; ++j) {
            const uint32_t bytes = chunk_rows_valid(j) * kRowBytes;
            mbar_expect_tx(&vbar[j], bytes);
            tma_load_1d(vring + j * chunk_bytes, chunk_at(vc, j), bytes, &vbar[j]);
        }
    }
    stamp(p, 1);
    // generation of the cross-cluster "shared reads done" barrier, read by the thread that may
    // later have to wait on it (lane 0 of the last warp) BEFORE this cluster arrives
    int32_t gen = 0;
    if (needs_epoch && tid == kThreads - 32) gen = ld_acquire_gpu(&st.sync_words[1]);

    // Everything the first phases take from global memory is requested here together: one round trip instead of one per phase.
    const int ipos = p.a.input_pos[0];
    uint4 qraw[G], knew8 = make_uint4(0, 0, 0, 0), vnew8 = make_uint4(0, 0, 0, 0);   // the new rows: the last warp stores them
    uint32_t vnew[CPL / 2];                                                          // this lane's columns of the value row
#pragma unroll
    for (int i = 0; i < CPL / 2; ++i) vnew[i] = 0;
    auto load_new = [&] {
        if (do_attend) {
#pragma unroll
            for (int g = 0; g < G; ++g) qraw[g] = *reinterpret_cast<const uint4*>(qp + g * D);
        }
        if (do_evict) {
#pragma unroll
            for (int i = 0; i < CPL / 2; ++i) vnew[i] = reinterpret_cast<const uint32_t*>(vrow_new)[lane * (CPL / 2) + i];
            if (warp == kWarps - 1) {
                knew8 = *reinterpret_cast<const uint4*>(knp);
                vnew8 = *reinterpret_cast<const uint4*>(vrow_new + li * 8);
            }
        }
    };
    int ps0 = 0, den0 = 0;
    double hist0 = 0.0;
    uint8_t mask0 = 0;
    if (in0) {
        mask0 = st.mask[(size_t)h * L + s0];
        if (do_evict) ps0 = posp[s0];
        if (hh_sum) {
            hist0 = hist[s0];
            den0 = den[s0];
        }
    }
    uint4 kdir[UR];      // this lane's parts of the warp's key rows
    if (direct) {
#pragma unroll
        for (int u = 0; u < UR; ++u) {
            const int r = (warp + u * kWarps) * RPW + sub;
            kdir[u] = r < chunk_rows_valid(0) ? *reinterpret_cast<const uint4*>(chunk_at(kc, 0) + (size_t)r * D + li * 8) : make_uint4(0, 0, 0, 0);
        }
    }
    if (!ahead) load_new();
    if (tid < local_rows) maskb[tid] = mask0;
    for (int lr = tid + kThreads; lr < local_rows; lr += kThreads) {
        const int s = slot_of(lr);
        maskb[lr] = (s < L) ? st.mask[(size_t)h * L + s] : 0;
    }

    // The next kernel in the stream may start its own prologue.  Never before this kernel has waited: the one after may read
    // ahead too, on the promise that THIS kernel leaves its cache alone, and must not meet the kernel before this one.
    if (!ahead) pdl_launch_dependents();

    // ---- 1. L2 only: key_norm.max() over every head and slot (cache.py:602) = X0 exchange
    float l2_max = 0.f;
    if constexpr (POLICY == CC_POLICY_L2) {
        if (do_evict) {
            const uint16_t* kn = reinterpret_cast<const uint16_t*>(st.key_norm);
            float m = -CUDART_INF_F;
            for (int hh = warp; hh < H; hh += kWarps)     // a warp per head: its loads are all under way at once
#pragma unroll 4
                for (int lr = lane; lr < local_rows; lr += 32) {
                    const int s = slot_of(lr);
                    if (s < L) m = fmaxf(m, bf16_bits_to_float(kn[(size_t)hh * L + s]));
                }
            m = warp_max_f32(m);
            if (lane == 0) misc[kMiscWarpMax + warp] = m;
            __syncthreads();
            l2_max = misc[kMiscWarpMax];
            for (int w = 1; w < kWarps; ++w) l2_max = fmaxf(l2_max, misc[kMiscWarpMax + w]);
            if (!solo) {
                cluster_wait_acquire();
                b0_waited = true;
                if (tid < C) st_async_u32(map_to_rank(smem_u32(&x0[rank]), tid), __float_as_uint(l2_max), map_to_rank(smem_u32(&xbar[0]), tid));
                mbar_wait(&xbar[0], 0);
                l2_max = x0[0];
                for (int r = 1; r < C; ++r) l2_max = fmaxf(l2_max, x0[r]);
            }
        }
    }

    // ---- 2. local arg-min candidate, key = (order(score) << 32) | slot  (first index wins ties)
    uint64_t ckey = kNoKey;
    if (do_evict) {
        if constexpr (POLICY == CC_POLICY_HEAVY_HITTER) {
#pragma unroll 1
            for (int lr = tid; lr < local_rows; lr += kThreads) {
                const int s = slot_of(lr);
                if (s >= L) continue;
                const bool first = lr == tid;
                const int ps = first ? ps0 : posp[s];
                // cache.py:727-749: mean accumulated attention; globals & recent -> 1.0; unfilled -> 0.0
                float avg;
                if (!hh_ring) {
                    avg = __fdiv_rn(__double2float_rn(first ? hist0 : hist[s]), (float)max(first ? den0 : den[s], 1));
                } else {
                    // sum of the slot's ring (kept as an exact fp64 running sum): bf16 ring -> bf16(fp32 sum),
                    // thresholded (bool) ring -> integer count; / clamp(denom, 1, W)   (cache.py:727-738)
                    const float hs = __double2float_rn(st.attn_history_sum[(size_t)h * L + s]);
                    avg = __fdiv_rn(st.attn_thresholding ? hs : bf16_round(hs), (float)min(max(den[s], 1), st.history_window));
                }
                if (ps < st.global_tokens || ps >= ipos - st.recent_window) avg = 1.0f;
                if (ps == -1) avg = 0.0f;
                const uint64_t k = ((uint64_t)float_order_key(avg) << 32) | (uint32_t)s;
                ckey = k < ckey ? k : ckey;
            }
        } else if constexpr (POLICY == CC_POLICY_L2) {
            const uint16_t* kn = reinterpret_cast<const uint16_t*>(st.key_norm) + (size_t)h * L;
#pragma unroll 1
            for (int lr = tid; lr < local_rows; lr += kThreads) {
                const int s = slot_of(lr);
                if (s >= L) continue;
                const int ps = lr == tid ? ps0 : posp[s];
                // cache.py:597-605 then 366-379: bf16(max - norm); recent -> +inf; first g slots -> +inf; unfilled -> -inf
                float sc = bf16_round(__fsub_rn(l2_max, bf16_bits_to_float(kn[s])));
                if (ps >= ipos - st.recent_window) sc = CUDART_INF_F;
                if (s < st.global_tokens) sc = CUDART_INF_F;
                if (ps == -1) sc = -CUDART_INF_F;
                const uint64_t k = ((uint64_t)float_order_key(sc) << 32) | (uint32_t)s;
                ckey = k < ckey ? k : ckey;
            }
        } else if constexpr (POLICY == CC_POLICY_RECENT_GLOBAL) {
            // cache.py:552-556: oldest position among slots >= g (unfilled = -1 first)
#pragma unroll 1
            for (int lr = tid; lr < local_rows; lr += kThreads) {
                const int s = slot_of(lr);
                if (s >= L || s < st.global_tokens) continue;
                const uint64_t k = ((uint64_t)((uint32_t)(lr == tid ? ps0 : posp[s]) ^ 0x80000000u) << 32) | (uint32_t)s;
                ckey = k < ckey ? k : ckey;
            }
        } else if constexpr (hybrid) {
            if (hyb_mode == kHybEvict) {
                // cache.py:844-894 over the live prefix [0, min(cts, L)): mean ring attention (or position for
                // window-only heads); first g slots, special, punctuation and the recent window are saved
                const int W = st.history_window;
                const double* hsum = st.attn_history_sum + (size_t)h * L;
                for (int lr = tid; lr < local_rows; lr += kThreads) {
                    const int s = slot_of(lr);
                    if (s >= live_limit) continue;      // a head that only appends counts on beyond its last slot
                    const int ps = posp[s];
                    float sc;
                    if (hyb_bits & CC_HYB_HEAVY_HITTER) {
                        const float d = (float)min(den[s], W);
                        sc = __fdiv_rn(bf16_round(__double2float_rn(hsum[s])), d);
                    } else {
                        sc = (float)ps;
                    }
                    bool save = s < st.global_tokens;
                    if ((hyb_bits & CC_HYB_SPECIAL) && st.special_mask) save |= st.special_mask[(size_t)h * L + s] != 0;
                    if ((hyb_bits & CC_HYB_PUNC) && st.punc_mask) save |= st.punc_mask[(size_t)h * L + s] != 0;
                    if ((hyb_bits & CC_HYB_WINDOW) && ps > ipos - hyb_rw) save = true;  // strict >
                    if (save) sc = CUDART_INF_F;
                    // torch.argmin treats NaN (0/0) as the minimum
                    const uint32_t hi = (sc != sc) ? 0u : float_order_key(sc);
                    const uint64_t k = ((uint64_t)hi << 32) | (uint32_t)s;
                    ckey = k < ckey ? k : ckey;
                }
            } else {
                // append at min(L-1, cts); a dropped token is parked in slot L-1 (cache.py:973-979)
                const int idx = hyb_mode == kHybAppend ? min(L - 1, hyb_cts) : L - 1;
                if (tid == 0 && ((idx >> chs) & (C - 1)) == rank) ckey = (uint64_t)(uint32_t)idx;
            }
        } else {  // CC_POLICY_EXTERNAL: the caller chose the slot
            const int64_t idx = p.a.fill_idx[st.pos_heads == 1 ? 0 : h];
            if (tid == 0 && idx >= 0 && idx < L && (((int)idx >> chs) & (C - 1)) == rank) ckey = (uint64_t)(uint32_t)idx;
        }
        ckey = warp_min_u64(ckey);
        if (lane == 0) reinterpret_cast<unsigned long long*>(miscu + kMiscWarpKey)[warp] = ckey;
        if (tid < kMaxG) misc[kMiscCandLg + tid] = -CUDART_INF_F;
        __syncthreads();
        ckey = lane < kWarps ? reinterpret_cast<unsigned long long*>(miscu + kMiscWarpKey)[lane] : kNoKey;
        ckey = warp_min_u64(ckey);
    }
    stamp(p, 2);
    // L2 warm-up hints: from here on this kernel mostly waits on latencies and HBM is idle; ask the
    // memory system to stream the next projections' weights into L2 meanwhile (4 KiB per request,
    // requests dealt round-robin over all CTAs).  Issued after this kernel's own loads.
    for (int i = 0; i < p.a.n_prefetch; ++i) {
        const char* base = reinterpret_cast<const char*>(p.a.prefetch[i].ptr);
        const unsigned long long bytes = p.a.prefetch[i].bytes;
        const unsigned long long n_req = (bytes + 4095) >> 12;
        for (unsigned long long c = (unsigned long long)tid * gridDim.x + blockIdx.x; c < n_req; c += (unsigned long long)kThreads * gridDim.x) {
            const unsigned long long off = c << 12;
            l2_prefetch_bulk(base + off, (uint32_t)min(4096ull, bytes - off));
        }
    }
    // Everything above reads only this layer's cache and policy state, which no kernel in flight
    // writes (CC_FLAG_OVERLAP_PREDECESSOR); q / k_new / v_new come from the projection kernel launched
    // just before this one: wait for it here, with the K/V tiles already on their way.
    if (ahead) {
        pdl_wait();
        pdl_launch_dependents();
        load_new();
    }
    // local row of this CTA's candidate (it owns the slot by construction)
    int cand_local = -1;
    if (ckey != kNoKey) {
        const int s = (int)(uint32_t)(ckey & 0xffffffffu);
        cand_local = (((s >> chs) >> csh) << chs) + (s & (CH - 1));
    }
    // a dropped token is stored in the last slot, whose mask stays as it was: it takes part in attention only if that slot was live
    const bool attend_new = do_evict && !(hybrid && hyb_mode == kHybDrop && !last_live);

    // ---- 3. logits over the K ring (canonical dot tree), new-token logits by the last warp while the rows arrive
    if (do_attend) {
        float q[G][8];
#pragma unroll
        for (int g = 0; g < G; ++g) unpack8(qraw[g], q[g]);
        auto dots = [&](const uint4& row, int* gsel) {
            float kf[8], part[G];
            unpack8(row, kf);
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float acc = 0.f;
#pragma unroll
                for (int i = 0; i < 8; ++i) acc = __fmaf_rn(q[g][i], kf[i], acc);
                part[g] = acc;
            }
            const float dot = group_reduce_multi<LPR, G>(part, li, gsel);
            // naive path rounds q@k^T to bf16, then * scale to bf16 (attention_utils.py:37)
            return NAIVE ? bf16_round(__fmul_rn(bf16_round(dot), p.scale)) : __fmul_rn(dot, p.scale);
        };
        int gsel = group_reduce_head<LPR, G>(li);   // the query head whose sums this lane ends up with
        if (attend_new && warp == kWarps - 1) {
            const float v = dots(knew8, &gsel);
            if (sub == 0 && gsel < G) misc[kMiscNewLg + gsel] = v;  // replicated lanes write the same value
        }
        // rows of chunks that cannot be live
        for (int lr = live_rows + tid; lr < local_rows; lr += kThreads)
#pragma unroll
            for (int g = 0; g < G; ++g) lg[g * stride + lr] = -CUDART_INF_F;
        if (!do_evict) __syncthreads();  // maskb visible
        float m = -CUDART_INF_F;         // of this lane's head over its rows, without the candidate's
        auto row_logits = [&](const uint4& row, int lr) {
            float v = dots(row, &gsel);
            if (!maskb[lr]) v = -CUDART_INF_F;      // rows beyond the cache are masked too
            if (gsel < G) lg[gsel * stride + lr] = v;
            if (lr != cand_local) m = fmaxf(m, v);
            else if (gsel < G) misc[kMiscCandLg + gsel] = v;      // replicated lanes write the same value
        };
        if (direct) {
#pragma unroll
            for (int u = 0; u < UR; ++u) {
                const int r0 = (warp + u * kWarps) * RPW;
                if (r0 < CH) row_logits(kdir[u], r0 + sub);
            }
        }
        // chunks that are all in the ring are walked as one run of rows
        const int per = nlc_live <= NS ? nlc_live : 1;
        for (int j = 0; j < nlc_live && !direct; j += per) {
            const int stage = j % NS, run = per << chs;
            for (int i = 0; i < per; ++i) mbar_wait(&kbar[stage + i], (j / NS) & 1);
            if (j == 0) stamp(p, 3);
            const uint8_t* kbase = kring + stage * chunk_bytes;
            // up to UR row pairs per warp per pass, all fetched before the dependent math (ILP)
#pragma unroll 1
            for (int r0 = warp * RPW; r0 < run; r0 += UR * kWarps * RPW) {
                uint4 kv[UR];
#pragma unroll
                for (int u = 0; u < UR; ++u) {
                    const int r = r0 + u * kWarps * RPW + sub;
                    if (u == 0 || r0 + u * kWarps * RPW < run) kv[u] = *reinterpret_cast<const uint4*>(kbase + r * kRowBytes + li * 16);
                }
#pragma unroll
                for (int u = 0; u < UR; ++u) {
                    const int r = r0 + u * kWarps * RPW + sub, lr = (j << chs) + r;
                    if (u > 0 && r0 + u * kWarps * RPW >= run) break;
                    row_logits(kv[u], lr);
                }
            }
            if (j + NS < nlc_live) {  // ring slot is refilled: everyone must be done with it
                __syncthreads();
                if (tid == 0) {
                    fence_proxy_async();
                    const int jn = j + NS;
                    const uint32_t bytes = chunk_rows_valid(jn) * kRowBytes;
                    mbar_expect_tx(&kbar[stage], bytes);
                    tma_load_1d(kring + stage * chunk_bytes, chunk_at(kc, jn), bytes, &kbar[stage]);
                }
            }
        }
#pragma unroll
        for (int d = 16; d >= LPR; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
        if (sub == 0 && gsel < G) misc[kMiscRowMax + warp * kMaxG + gsel] = m;
    }
    __syncthreads();  // logits and row maxima visible
    stamp(p, 4);
    // ---- 4./5. X1: every CTA learns every candidate, every row maximum without the local candidate, and the candidate's logits
    if (!solo) {
        if (!b0_waited) cluster_wait_acquire();
        for (int idx = tid; idx < C * NW; idx += kThreads) {
            const int dest = idx / NW, w = idx % NW;
            uint32_t word = __float_as_uint(-CUDART_INF_F);
            if (w < 2) {
                word = w == 0 ? (uint32_t)(ckey & 0xffffffffu) : (uint32_t)(ckey >> 32);
            } else if (do_attend) {
                if (w < 2 + G) {
                    float m = misc[kMiscRowMax + w - 2];
#pragma unroll
                    for (int k = 1; k < kWarps; ++k) m = fmaxf(m, misc[kMiscRowMax + k * kMaxG + w - 2]);
                    word = __float_as_uint(m);
                } else if (cand_local >= 0) {
                    word = __float_as_uint(misc[kMiscCandLg + w - 2 - G]);
                }
            }
            st_async_u32(map_to_rank(smem_u32(&rec[rank * kRecWords + w]), dest), word, map_to_rank(smem_u32(&xbar[1]), dest));
        }
        mbar_wait(&xbar[1], 0);
    }
    stamp(p, 5);

    // ---- 6. winner, and the maximum of the query head whose softmax this warp takes (WPG warps share a head's rows)
    uint64_t wkey = ckey;
    if (!solo) {
        wkey = lane < C ? (uint64_t)rec[lane * kRecWords] | ((uint64_t)rec[lane * kRecWords + 1] << 32) : kNoKey;
    }
    const bool lane_has_cand = wkey != kNoKey && lane < C;
    if (!solo) wkey = warp_min_u64(wkey);
    const bool has_slot = do_evict && wkey != kNoKey;  // a slot is overwritten this step
    const int widx = has_slot ? (int)(uint32_t)(wkey & 0xffffffffu) : -1;
    const int owner = has_slot ? (widx >> chs) & (C - 1) : -1;
    const bool i_own = has_slot && owner == rank;
    const int widx_local = has_slot ? (((widx >> chs) >> csh) << chs) + (widx & (CH - 1)) : -1;
    const bool has_new = has_slot && attend_new;  // ... and the new token attends to itself there
    if (needs_epoch && rank == 0 && tid == 0) red_release_gpu_add(&st.sync_words[0], 1);  // shared reads done
    const int wg = warp % G, wpart = warp / G;
    const bool softmax_warp = wpart < WPG;
    float gm = -CUDART_INF_F, nl = -CUDART_INF_F;
    if (do_attend) {
        float m = -CUDART_INF_F;
        // a candidate that is not overwritten keeps its logit; the overwritten one only if the new
        // token does not replace it in attention (hybrid drop: slot L-1 stays as it was)
        const bool cand_stays = lane_has_cand && (lane != owner || !has_new);
        if (solo) {
            if (lane < kWarps) m = misc[kMiscRowMax + lane * kMaxG + wg];
            if (cand_stays) m = fmaxf(m, misc[kMiscCandLg + wg]);
        } else if (lane < C) {
            m = __uint_as_float(rec[lane * kRecWords + 2 + wg]);
            if (cand_stays) m = fmaxf(m, __uint_as_float(rec[lane * kRecWords + 2 + G + wg]));
        }
        nl = has_new ? misc[kMiscNewLg + wg] : -CUDART_INF_F;
        gm = fmaxf(warp_max_f32(m), nl);
    }
    const int patch_row = (i_own && has_new) ? widx_local : -1;  // this row now holds the new token
    stamp(p, 6);

    if (do_attend) {
        // ---- 8. exp and the exact fixed-point softmax denominator = X2: every warp sends its partial sum to every CTA itself;
        // integers, so their order does not matter.
        float* lgw = lg + wg * stride;
        if (softmax_warp) {
            long long part = 0;
            for (int lr = wpart * 32 + lane; lr < live_rows; lr += WPG * 32) {
                const float l = lr == patch_row ? nl : lgw[lr];
                const float e = det_expf(__fsub_rn(l, gm));
                lgw[lr] = e;
                part += __float2ll_rz(__fmul_rn(e, 1099511627776.0f));
            }
            part = (long long)warp_sum_u64((unsigned long long)part);
            unsigned long long* mine = &sums[wg * (kMaxCluster * WPG) + rank * WPG + wpart];
            if (solo) {
                if (lane == 0) *mine = (unsigned long long)part;
            } else if (lane < C) {
                st_async_u64(map_to_rank(smem_u32(mine), lane), (unsigned long long)part, map_to_rank(smem_u32(&xbar[2]), lane));
            }
        }
        stamp(p, 7);
        if (solo) __syncthreads();
        else mbar_wait(&xbar[2], 0);
        stamp(p, 8);
        // ---- 9a. probabilities: every warp adds the partial denominators of its head and goes over its own rows again
        if (softmax_warp) {
            unsigned long long t = 0;
            for (int i = lane; i < C * WPG; i += 32) t += sums[wg * (kMaxCluster * WPG) + i];
            const float sf = __fmul_rn(__ll2float_rn((long long)warp_sum_u64(t)), 9.094947017729282e-13f);  // 2^-40
            for (int lr = wpart * 32 + lane; lr < live_rows; lr += WPG * 32) {
                float pr = __fdiv_rn(lgw[lr], sf);
                if (NAIVE) pr = bf16_round(pr);
                lgw[lr] = pr;
            }
        }
        __syncthreads();
        stamp(p, 9);

        // ---- 10. y = P.V over the V ring, cluster-wide reduction = X3
        // A warp has RPW neighbouring rows out of every kWarps * RPW and all their columns, CPL a lane: nothing to add up across
        // lanes.  Each of the RPW rows has sums of its own, which meet at the end: the order of the additions is part of the result
        // (a bf16 rounding of y), so it stays what it is however rows are dealt to lanes.  (One sum per column for all rows of a
        // warp is no faster: 32 steps in a graph, 64 sliding slots 189.3 and 189.4 us, 1024 heavy-hitter slots 257.0 and 256.9, L2 flushed.)
        float acc[RPW][G][CPL];
#pragma unroll
        for (int x = 0; x < RPW; ++x)
#pragma unroll
            for (int g = 0; g < G; ++g)
#pragma unroll
                for (int i = 0; i < CPL; ++i) acc[x][g][i] = 0.f;
        for (int j = 0; j < nlc_live; ++j) {
            const int stage = j % NS;
            mbar_wait(&vbar[stage], (j / NS) & 1);
            const int r_end = chunk_rows_valid(j);
            const uint8_t* vbase = vring + stage * chunk_bytes + lane * (CPL * 2);
#pragma unroll (G >= 7 ? 1 : 2)        // two at a time would spill with 64 sums in 128 registers
            for (int r = warp * RPW; r < r_end; r += kWarps * RPW) {
                const int lr = (j << chs) + r;
                uint32_t vv[RPW][CPL / 2];
#pragma unroll
                for (int x = 0; x < RPW; ++x) {
                    if constexpr (CPL == 4) {
                        const uint2 u = *reinterpret_cast<const uint2*>(vbase + (r + x) * kRowBytes);
                        vv[x][0] = u.x;
                        vv[x][1] = u.y;
                    } else {
                        vv[x][0] = *reinterpret_cast<const uint32_t*>(vbase + (r + x) * kRowBytes);
                    }
#pragma unroll
                    for (int i = 0; i < CPL / 2; ++i) {
                        if (lr + x == patch_row) vv[x][i] = vnew[i];
                        if (r + x >= r_end) vv[x][i] = 0;      // not loaded: no number
                    }
                }
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    float pr[RPW];
                    if constexpr (RPW == 4) {
                        const float4 t = *reinterpret_cast<const float4*>(lg + g * stride + lr);
                        pr[0] = t.x; pr[1] = t.y; pr[2] = t.z; pr[3] = t.w;
                    } else {
                        const float2 t = *reinterpret_cast<const float2*>(lg + g * stride + lr);
                        pr[0] = t.x; pr[1] = t.y;
                    }
#pragma unroll
                    for (int x = 0; x < RPW; ++x)
#pragma unroll
                        for (int i = 0; i < CPL; ++i)
                            acc[x][g][i] = fmaf(pr[x], __uint_as_float(i & 1 ? vv[x][i / 2] & 0xffff0000u : vv[x][i / 2] << 16), acc[x][g][i]);
                }
            }
            if (j + NS < nlc_live) {  // ring slot is refilled: everyone must be done with it
                __syncthreads();
                if (tid == 0) {
                    fence_proxy_async();
                    const int jn = j + NS;
                    const uint32_t bytes = chunk_rows_valid(jn) * kRowBytes;
                    mbar_expect_tx(&vbar[stage], bytes);
                    tma_load_1d(vring + stage * chunk_bytes, chunk_at(vc, jn), bytes, &vbar[stage]);
                }
            }
        }
        stamp(p, 10);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float* dst = &red[warp * G * D + g * D + lane * CPL];
            float sum[CPL];
#pragma unroll
            for (int i = 0; i < CPL; ++i) {
                if constexpr (RPW == 4) sum[i] = (acc[0][g][i] + acc[2][g][i]) + (acc[1][g][i] + acc[3][g][i]);
                else sum[i] = acc[0][g][i] + acc[1][g][i];
            }
            if constexpr (CPL == 4) *reinterpret_cast<float4*>(dst) = make_float4(sum[0], sum[1], sum[2], sum[3]);
            else *reinterpret_cast<float2*>(dst) = make_float2(sum[0], sum[1]);
        }
        __syncthreads();
        const int SL = (G * D) >> csh;  // outputs reduced by each CTA of the cluster (a multiple of 4)
        for (int o4 = tid; o4 < G * D / 4; o4 += kThreads) {
            const int o = o4 * 4;
            float4 s = *reinterpret_cast<const float4*>(&red[o]);
#pragma unroll
            for (int w = 1; w < kWarps; ++w) {
                const float4 t = *reinterpret_cast<const float4*>(&red[w * G * D + o]);
                s.x += t.x; s.y += t.y; s.z += t.z; s.w += t.w;
            }
            if (solo) {
                __nv_bfloat162 y2[2] = {__floats2bfloat162_rn(s.x, s.y), __floats2bfloat162_rn(s.z, s.w)};
                *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.a.y) + (size_t)h * G * D + o) = *reinterpret_cast<uint2*>(y2);
                continue;
            }
            const int dest = o / SL, off = o - dest * SL;
            st_async_v4f32(map_to_rank(smem_u32(&yx[rank * SL + off]), dest), s, map_to_rank(smem_u32(&xbar[3]), dest));
        }
        stamp(p, 11);
    }

    // ======== off the critical path: global state writes, overlapped with the X3 barrier ========
    // ---- 7. owner CTA: in-place slot overwrite (cache.py:390-401 / 460-490) + policy state
    if (i_own && warp == kWarps - 1) {
        if (lane < LPR) {
            uint16_t* kd = reinterpret_cast<uint16_t*>(st.k_cache) + ((size_t)h * L + widx) * D + lane * 8;
            uint16_t* vd = reinterpret_cast<uint16_t*>(st.v_cache) + ((size_t)h * L + widx) * D + lane * 8;
            *reinterpret_cast<uint4*>(kd) = knew8;     // lane == li
            *reinterpret_cast<uint4*>(vd) = vnew8;
        }
        float knorm = 0.f;
        if constexpr (POLICY == CC_POLICY_L2) {
            // key_norm[idx] = ||k_new||_2 (cache.py:592-593), canonical tree, correctly rounded sqrt
            float kf[8];
            unpack8(knew8, kf);
            float acc = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) acc = __fmaf_rn(kf[i], kf[i], acc);
            knorm = __fsqrt_rn(group_butterfly<LPR>(acc));
        }
        if (lane == 0) {
            const int32_t pos_old = posp[widx];
            if (!hybrid || hyb_mode == kHybAppend) st.mask[(size_t)h * L + widx] = 1;
            if (p.a.fill_idx && POLICY != CC_POLICY_EXTERNAL) p.a.fill_idx[h] = widx;
            if (POLICY == CC_POLICY_HEAVY_HITTER && !do_score) {
                if (hh_ring) st.attn_history_sum[(size_t)h * L + widx] = 0.0;   // the ring row is cleared below
                else reinterpret_cast<double*>(st.attn_history_num)[(size_t)h * L + widx] = 0.0;  // cache.py:753-763
                st.attn_history_denom[(size_t)h * L + widx] = 0;
            }
            if (hybrid && is_punc && st.punc_mask) st.punc_mask[(size_t)h * L + widx] = 1;  // cache.py:1011-1016
            if (needs_epoch) {  // head-constant pos, key_norm, counters are read by every cluster: write after all have read
                const int32_t target = (gen + 1) * H;
                while (ld_acquire_gpu(&st.sync_words[0]) - target < 0) {}
            }
            if constexpr (POLICY == CC_POLICY_L2)
                reinterpret_cast<__nv_bfloat16*>(st.key_norm)[(size_t)h * L + widx] = __float2bfloat16_rn(knorm);
            if (st.pos_heads != 1 || h == 0) st.pos[(size_t)pos_row * L + widx] = ipos;
            if constexpr (hybrid) {
                if (hyb_mode == kHybAppend) st.cache_cts[h] = hyb_cts + 1;
                if (h == 0 && is_punc && st.num_punc) st.num_punc[0] += 1;
            } else if (h == 0) {
                st.cache_cts[0] += (pos_old == -1) ? 1 : 0;  // cache.py:330, 356-360
            }
        }
    }
    if (hh_ring && i_own) {
        // the evicted slot's history restarts (cache.py:753-763): clear its ring row, except the column this very
        // step writes when the score update is fused into the same launch
        const int W = st.history_window;
        const int keep = (do_score && NAIVE) ? (int)(hyb_counter % W) : -1;
        if (st.attn_thresholding) {
            uint8_t* rowp = reinterpret_cast<uint8_t*>(st.attn_history_num) + ((size_t)h * L + widx) * W;
            for (int w = tid; w < W; w += kThreads) if (w != keep) rowp[w] = 0;
        } else {
            uint16_t* rowp = reinterpret_cast<uint16_t*>(st.attn_history_num) + ((size_t)h * L + widx) * W;
            for (int w = tid; w < W; w += kThreads) if (w != keep) rowp[w] = 0;
        }
    }
    if (needs_epoch && h == 0 && rank == 0 && tid == 32) {
        // generation bump (and the shared step counter): only after every cluster has arrived
        const int32_t g0 = ld_acquire_gpu(&st.sync_words[1]);
        const int32_t target = (g0 + 1) * H;
        while (ld_acquire_gpu(&st.sync_words[0]) - target < 0) {}
        if ((hybrid || hh_ring) && do_score && NAIVE) st.attn_counter[0] = hyb_counter + 1;
        st_release_gpu(&st.sync_words[1], g0 + 1);
    }

    // ---- 9b. GQA pooling (model.py:413-418) and the score update (cache.py:716-723)
    {
        const bool hh_score = do_score && NAIVE && POLICY == CC_POLICY_HEAVY_HITTER && !hh_ring;
        const bool hhr_score = do_score && NAIVE && hh_ring;
        const bool ring_score = do_score && NAIVE && hybrid;
        const int W = st.history_window;
        const int wslot = (ring_score || hhr_score) ? (int)(hyb_counter % W) : 0;
        // thresholded history: indicator p >= 1 / cache_cts with cache_cts AFTER this step's insertion (cache.py:330,
        // 708).  While the cache is filling the inserted slot is an unfilled one (score 0.0, first index): + 1.
        const float thr = hhr_score ? __fdiv_rn(1.0f, (float)(hh_cts + ((do_evict && has_slot && hh_cts < L) ? 1 : 0))) : 0.f;
        __nv_bfloat16* probs = reinterpret_cast<__nv_bfloat16*>(p.a.probs);
        if (NAIVE && (hh_score || hhr_score || ring_score || (do_attend && probs))) {
            for (int lr = tid; lr < local_rows; lr += kThreads) {
                const int s = slot_of(lr);
                if (s >= L) continue;
                float pooled = 0.f;
                if (do_attend) {
                    if (lr < live_rows) {
                        float acc = lg[lr];
#pragma unroll
                        for (int g = 1; g < G; ++g) acc = __fadd_rn(acc, lg[g * stride + lr]);
                        pooled = bf16_round(__fdiv_rn(acc, (float)G));  // torch mean: fp32 sum / G, then bf16
                    }
                    if (probs) probs[(size_t)h * L + s] = __float2bfloat16_rn(pooled);
                } else {
                    pooled = __bfloat162float(probs[(size_t)h * L + s]);
                }
                if (hh_score) {
                    const bool first = lr == tid, fresh = has_slot && s == widx;  // evicted slot's history restarts (cache.py:753-763)
                    const double was = first ? hist0 : hist[s];
                    const int seen = first ? den0 : den[s];
                    reinterpret_cast<double*>(st.attn_history_num)[(size_t)h * L + s] = (fresh ? 0.0 : was) + (double)pooled;
                    st.attn_history_denom[(size_t)h * L + s] = (fresh ? 0 : seen) + 1;
                } else if (hhr_score) {
                    // ring[s][counter % W] = pooled (or its indicator), denominators + 1; the evicted slot starts
                    // from a cleared ring (cache.py:716-723, 753-763).  hsum = exact running sum of the ring.
                    double* hs = st.attn_history_sum + (size_t)h * L + s;
                    const bool fresh = has_slot && s == widx;
                    st.attn_history_denom[(size_t)h * L + s] = (fresh ? 0 : den[s]) + 1;
                    if (st.attn_thresholding) {
                        uint8_t* cell = reinterpret_cast<uint8_t*>(st.attn_history_num) + ((size_t)h * L + s) * W + wslot;
                        const float v = pooled >= thr ? 1.f : 0.f;
                        const float old = fresh ? 0.f : (float)(*cell != 0);
                        *hs = ((fresh ? 0.0 : *hs) - (double)old) + (double)v;
                        *cell = (uint8_t)(v != 0.f);
                    } else {
                        __nv_bfloat16* cell = reinterpret_cast<__nv_bfloat16*>(st.attn_history_num) + ((size_t)h * L + s) * W + wslot;
                        const float old = fresh ? 0.f : __bfloat162float(*cell);
                        *hs = ((fresh ? 0.0 : *hs) - (double)old) + (double)pooled;
                        *cell = __float2bfloat16_rn(pooled);
                    }
                } else if (ring_score) {
                    // ring[s][counter % W] = pooled; the evicted slot keeps its ring (the reference's reset is a
                    // silent no-op, cache.py:993-996).  Only live slots can hold non-zero history.
                    st.attn_history_denom[(size_t)h * L + s] = den[s] + 1;
                    if (s < live_limit || pooled != 0.f) {
                        __nv_bfloat16* cell = reinterpret_cast<__nv_bfloat16*>(st.attn_history_num) + ((size_t)h * L + s) * W + wslot;
                        const float old = __bfloat162float(*cell);
                        if (old != pooled) {
                            double* hs = st.attn_history_sum + (size_t)h * L + s;
                            *hs = (*hs - (double)old) + (double)pooled;
                            *cell = __float2bfloat16_rn(pooled);
                        }
                    }
                }
            }
        }
        if (hh_score && h == 0 && rank == 0 && tid == 0) st.attn_counter[0] += 1;
    }

    if (do_attend && !solo) {
        mbar_wait(&xbar[3], 0);
        stamp(p, 12);
        const int SL = (G * D) >> csh;
        __nv_bfloat16* y = reinterpret_cast<__nv_bfloat16*>(p.a.y) + (size_t)h * G * D;
        for (int t = tid; t < SL; t += kThreads) {
            float s = yx[t];
            for (int r = 1; r < C; ++r) s += yx[r * SL + t];
            y[rank * SL + t] = __float2bfloat16_rn(s);
        }
    }
    stamp(p, 13);
}

// --------------------------------------------------------------------------- host side

using KernelFn = void (*)(const DecodeParams);

template <int D, int G>
static KernelFn pick_policy(int policy, bool naive) {
    switch (policy) {
    case CC_POLICY_EXTERNAL: return naive ? (KernelFn)cc_decode_kernel<D, G, CC_POLICY_EXTERNAL, true>   // debug_* full cache
                                          : (KernelFn)cc_decode_kernel<D, G, CC_POLICY_EXTERNAL, false>;
    case CC_POLICY_RECENT_GLOBAL: return naive ? nullptr : (KernelFn)cc_decode_kernel<D, G, CC_POLICY_RECENT_GLOBAL, false>;
    case CC_POLICY_L2: return naive ? nullptr : (KernelFn)cc_decode_kernel<D, G, CC_POLICY_L2, false>;
    case CC_POLICY_HEAVY_HITTER: return naive ? (KernelFn)cc_decode_kernel<D, G, CC_POLICY_HEAVY_HITTER, true> : nullptr;
    case CC_POLICY_HYBRID: return naive ? (KernelFn)cc_decode_kernel<D, G, CC_POLICY_HYBRID, true>
                                        : (KernelFn)cc_decode_kernel<D, G, CC_POLICY_HYBRID, false>;
    default: return nullptr;
    }
}
template <int D>
static KernelFn pick_group(int G, int policy, bool naive) {
    switch (G) {
    case 1: return pick_policy<D, 1>(policy, naive);
    case 2: return pick_policy<D, 2>(policy, naive);
    case 4: return pick_policy<D, 4>(policy, naive);
    case 6: return pick_policy<D, 6>(policy, naive);
    case 7: return pick_policy<D, 7>(policy, naive);
    case 8: return pick_policy<D, 8>(policy, naive);
    default: return nullptr;
    }
}
static KernelFn pick_kernel(int D, int G, int policy, bool naive) {
    if (D == 128) return pick_group<128>(G, policy, naive);
    if (D == 64) return pick_group<64>(G, policy, naive);
    return nullptr;
}

struct LaunchPlan {
    KernelFn fn;
    int cluster, ch_shift, max_local_chunks, n_stages, lg_stride;
    uint32_t smem;
};

static int g_num_sms = 0;
static int g_smem_optin = 0;
static unsigned long long* g_trace = nullptr;  // diagnostics only (cc_debug_set_trace)
void set_trace_buffer(unsigned long long* buf) { g_trace = buf; }

static int g_limits_dev = -1;
static int device_limits() {
    int dev = 0;
    cudaGetDevice(&dev);
    if (g_num_sms && g_limits_dev == dev) return CC_OK;
    g_num_sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return set_error(CC_ERR_NO_DEVICE, "no CUDA device");
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, dev) != cudaSuccess) return set_error(CC_ERR_NO_DEVICE, "cudaGetDeviceProperties failed");
    if (prop.major != 10) return set_error(CC_ERR_NO_DEVICE, "this library is built for sm_100a (Blackwell B200) only");
    g_num_sms = prop.multiProcessorCount;
    g_smem_optin = (int)prop.sharedMemPerBlockOptin;
    g_limits_dev = dev;
    return CC_OK;
}

// Plans are cached per (shape, policy class): the occupancy query is not free.
struct PlanKey { int D, G, naive, H, L, policy, dev; };
struct PlanEntry { PlanKey k; LaunchPlan p; };
static PlanEntry g_plans[128];
static int g_nplans = 0;

static int make_plan(const CcCacheState* st, bool needs_epoch, LaunchPlan* out) {
    const int D = st->head_dim, G = st->q_per_kv, H = st->n_kv_heads, L = st->max_cache_length;
    const bool naive = st->attn_mode == CC_ATTN_NAIVE_BF16;
    int dev = 0;
    cudaGetDevice(&dev);   // plans (occupancy, shared-memory limits) belong to a device
    for (int i = 0; i < g_nplans; ++i) {
        const PlanKey& k = g_plans[i].k;
        if (k.D == D && k.G == G && k.naive == (int)naive && k.H == H && k.L == L && k.policy == st->policy && k.dev == dev) {
            *out = g_plans[i].p;
            return CC_OK;
        }
    }
    int rc = device_limits();
    if (rc) return rc;
    KernelFn fn = pick_kernel(D, G, st->policy, naive);
    if (!fn) return set_error(CC_ERR_UNSUPPORTED_SHAPE, "unsupported head_dim (64/128), q_per_kv (1,2,4,6,7,8) or policy/attention-mode pair");
    cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    // the cap is per function and plans for other shapes share it: raise it once to the device
    // limit instead of to this plan's size (a later, smaller plan must not lower it)
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, g_smem_optin) != cudaSuccess) {
        cudaGetLastError();
        return set_error(CC_ERR_CUDA, "cannot raise the dynamic shared memory limit");
    }
    int c_max = kMaxCluster;
    if (const char* e = getenv("CC_B200_MAX_CLUSTER")) c_max = atoi(e) > 0 ? atoi(e) : c_max;  // experiments only
    // 16 CTAs per head from 1024 slots, or from 257 if they take at most half of the SMs; else up to 8: an exchange among 16 costs more
    // than the shorter rows give.  32 steps in a graph, 16 / 8 / 4 CTAs, us a step: 8 heads of group 4, 256 slots 7.0 / 6.5 / 6.9, 512
    // slots 7.4 / 7.0 / 8.3, 1024 slots of heavy hitters 8.5 / 8.7 / 11.4; 4 heads of group 7, 256 slots 7.0 / 7.2 / 7.8, 512 slots
    // 7.5 / 7.9 / 9.5.  Up to 128 slots 4 and 8 are alike; one CTA without exchanges loses to both from 64 slots on (6.7 / 6.3).
    if (L < 1024 && (L <= 256 || H * kMaxCluster > g_num_sms / 2) && c_max > 8) c_max = 8;
    for (int C = c_max; C >= 1; C >>= 1) {
        // chunk size: the largest of 64/32/16 rows that still gives every CTA of the cluster a chunk
        int chs = 6;
        while (chs > 4 && ((L + (1 << chs) - 1) >> chs) < C) --chs;
        const int n_chunks = (L + (1 << chs) - 1) >> chs;
        if (C > 1 && (H * C > g_num_sms || C > n_chunks)) continue;
        const int mlc = (n_chunks + C - 1) / C;
        const int stride = ((mlc << chs) + 31) / 32 * 32;
        for (int ns = mlc < 4 ? mlc : 4; ns >= 1; --ns) {
            const SmemLayout lay = make_layout(D, G, 1 << chs, mlc << chs, ns, stride);
            if ((int)lay.total > g_smem_optin) continue;
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(H * C);
            cfg.blockDim = dim3(kThreads);
            cfg.dynamicSmemBytes = lay.total;
            cudaLaunchAttribute attr;
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = C; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
            cfg.attrs = &attr; cfg.numAttrs = 1;
            int max_clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&max_clusters, fn, &cfg) != cudaSuccess) { cudaGetLastError(); continue; }
            // every cluster of the layer must be co-resident: the epoch barrier needs it for correctness,
            // and a second wave of clusters would double the step time in any case
            if (getenv("CC_B200_DEBUG_PLAN"))
                fprintf(stderr, "[cc plan] D=%d G=%d policy=%d L=%d: C=%d stages=%d smem=%u max_active_clusters=%d\n", D, G,
                        st->policy, L, C, ns, lay.total, max_clusters);
            // (the epoch barrier spins on the other heads' clusters: without co-residency it would never complete,
            // whatever the cluster size)
            if (max_clusters < H && (C > 1 || needs_epoch)) continue;
            LaunchPlan p = {fn, C, chs, mlc, ns, stride, lay.total};
            if (g_nplans < 128) g_plans[g_nplans++] = {{D, G, (int)naive, H, L, st->policy, dev}, p};
            *out = p;
            return CC_OK;
        }
    }
    return set_error(CC_ERR_UNSUPPORTED_SHAPE, "no cluster size / shared-memory plan fits this cache shape");
}

static int validate(const CcCacheState* st, const CcDecodeArgs* a) {
    if (!st || !a) return set_error(CC_ERR_INVALID_ARG, "null state or args");
    if (st->n_kv_heads < 1 || st->q_per_kv < 1 || st->max_cache_length < 1) return set_error(CC_ERR_INVALID_ARG, "bad shape");
    if (st->policy < CC_POLICY_EXTERNAL || st->policy > CC_POLICY_HYBRID) return set_error(CC_ERR_INVALID_ARG, "bad policy");
    if (!st->k_cache || !st->v_cache || !st->pos || !st->mask || !st->cache_cts) return set_error(CC_ERR_INVALID_ARG, "null cache buffer");
    if (st->pos_heads != 1 && st->pos_heads != st->n_kv_heads) return set_error(CC_ERR_INVALID_ARG, "pos_heads must be 1 or n_kv_heads");
    const int phases = a->phases;
    if (phases < 1 || phases > CC_PHASE_ALL) return set_error(CC_ERR_INVALID_ARG, "bad phases mask");
    if (!a->input_pos) return set_error(CC_ERR_INVALID_ARG, "null input_pos");
    if ((phases & CC_PHASE_EVICT_FILL) && (!a->k_new || !a->v_new)) return set_error(CC_ERR_INVALID_ARG, "evict/fill needs k_new and v_new");
    if ((phases & CC_PHASE_ATTEND) && (!a->q || !a->y)) return set_error(CC_ERR_INVALID_ARG, "attend needs q and y");
    if (st->policy == CC_POLICY_EXTERNAL && (phases & CC_PHASE_EVICT_FILL) && !a->fill_idx)
        return set_error(CC_ERR_INVALID_ARG, "external policy needs fill_idx");
    const bool naive = st->attn_mode == CC_ATTN_NAIVE_BF16;
    if (naive && (phases & CC_PHASE_SCORE) && !(phases & CC_PHASE_ATTEND) && !a->probs)
        return set_error(CC_ERR_INVALID_ARG, "score-only phase needs probs");
    if (st->policy == CC_POLICY_HEAVY_HITTER) {
        if (st->history_window < 1) return set_error(CC_ERR_INVALID_ARG, "history_window must be >= 1");
        if (!st->attn_history_num || !st->attn_history_denom || !st->attn_counter) return set_error(CC_ERR_INVALID_ARG, "null heavy_hitter state");
        if (st->history_window > 1 && !st->attn_history_sum)
            return set_error(CC_ERR_INVALID_ARG, "heavy_hitter with a history window needs the running ring sums (attn_history_sum)");
        if (st->attn_thresholding && st->history_window == 1)
            return set_error(CC_ERR_INVALID_ARG, "attn_thresholding needs history_window_size > 1 (the reference cannot add into a bool history)");
        if (!naive) return set_error(CC_ERR_INVALID_ARG, "heavy_hitter needs the naive (probability-returning) attention mode");
    }
    if (st->policy == CC_POLICY_HYBRID) {
        if (st->cts_heads != st->n_kv_heads) return set_error(CC_ERR_INVALID_ARG, "hybrid needs per-head cache_cts");
        if (st->pos_heads != st->n_kv_heads) return set_error(CC_ERR_INVALID_ARG, "hybrid needs per-head pos");
        if (!st->hyb_strategy_bits || !st->hyb_recent_window || !st->hyb_heavy_budget) return set_error(CC_ERR_INVALID_ARG, "null hybrid strategy tables");
        if (naive && (st->history_window < 2 || !st->attn_history_num || !st->attn_history_denom || !st->attn_counter || !st->attn_history_sum))
            return set_error(CC_ERR_INVALID_ARG, "hybrid with heavy hitters needs the ring history, its denominators, counter and running sums");
        if (!st->sync_words) return set_error(CC_ERR_INVALID_ARG, "hybrid needs sync_words");
    }
    if (st->policy == CC_POLICY_L2 && !st->key_norm) return set_error(CC_ERR_INVALID_ARG, "null key_norm");
    if (a->n_prefetch < 0 || a->n_prefetch > 3) return set_error(CC_ERR_INVALID_ARG, "n_prefetch must be 0..3");
    for (int i = 0; i < a->n_prefetch; ++i)
        if (!a->prefetch[i].ptr || ((uintptr_t)a->prefetch[i].ptr & 15) || (a->prefetch[i].bytes & 15))
            return set_error(CC_ERR_INVALID_ARG, "prefetch ranges must be non-null and 16-byte aligned/sized");
    if ((st->policy == CC_POLICY_RECENT_GLOBAL || st->policy == CC_POLICY_L2) && !st->sync_words)
        return set_error(CC_ERR_INVALID_ARG, "this policy needs sync_words");
    if (st->policy == CC_POLICY_RECENT_GLOBAL && st->global_tokens >= st->max_cache_length)
        return set_error(CC_ERR_INVALID_ARG, "global_tokens must be < max_cache_length");
    return CC_OK;
}

static bool plan_needs_epoch(const CcCacheState* st) {
    return st->policy == CC_POLICY_RECENT_GLOBAL || st->policy == CC_POLICY_L2 || st->policy == CC_POLICY_HYBRID ||
           (st->policy == CC_POLICY_HEAVY_HITTER && st->history_window > 1);
}

int decode_step_impl(const CcCacheState* st, const CcDecodeArgs* a, cudaStream_t stream) {
    int rc = validate(st, a);
    if (rc) return rc;
    if (a->flags & CC_FLAG_VIA_TOKEN_KERNEL) return decode_step_via_token_impl(st, a, stream);
    LaunchPlan plan;
    rc = make_plan(st, plan_needs_epoch(st), &plan);
    if (rc) return rc;
    DecodeParams p;
    p.st = *st;
    p.a = *a;
    p.ch_shift = plan.ch_shift;
    p.max_local_chunks = plan.max_local_chunks;
    p.n_stages = plan.n_stages;
    p.lg_stride = plan.lg_stride;
    p.scale = (float)(1.0 / sqrt((double)st->head_dim));
    p.lay = make_layout(st->head_dim, st->q_per_kv, 1 << plan.ch_shift, plan.max_local_chunks << plan.ch_shift,
                        plan.n_stages, plan.lg_stride);
    p.c_shift = 0;
    while ((1 << p.c_shift) < plan.cluster) ++p.c_shift;
    p.trace = g_trace;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(st->n_kv_heads * plan.cluster);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = plan.cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, plan.fn, p);
    if (e != cudaSuccess) return set_cuda_error(e, "cc_decode_step launch");
    return CC_OK;
}

int decode_cluster_size_impl(const CcCacheState* st) {
    if (!st) return set_error(CC_ERR_INVALID_ARG, "null state");
    LaunchPlan plan;
    int rc = make_plan(st, plan_needs_epoch(st), &plan);
    return rc ? rc : plan.cluster;
}

}  // namespace cc
