// Dequant-GEMM for prefill-sized steps: a pair of CTAs takes 256 weight rows x 256 activation rows per work item, the
// converted weights in tensor memory (the arithmetic of gemm_ta.cu).
//
// Each CTA converts its 128 weight rows once for all 256 activation rows and holds half of the activations; the leading
// CTA issues the products of both (cta_group::2: M = 256, N = 128, each CTA's tensor core reading half of the columns from
// the other's shared memory).  With one CTA per item (two units of 128 rows x 128 activation rows) conversion, products and
// folds were all near their limits side by side: of 7,000 clocks per k tile the conversion warps worked 5,960, the fold
// 5,100, and the products, 4,224, took 5,770, because the issuing warp waits for its slots among theirs.  A pair halves the
// conversion and the operand reads: gate | up of the 8B model at 2,048 rows 757 -> 667 us, down 516 -> 402 us.
//
// Tensor memory: two sums in turn at columns 0 and 128 (128 activation rows, a group; hi and lo parts in one, lo first), the
// minima's sums at 256, A stages at 384 and 448: 128 inputs of Q4_K's one plane, 64 inputs of the others' two.  A stage
// meets both groups, so a group's fold hides under the other group's products: once per 128 inputs of the K-quants, once per
// k tile of Q8_0.  (An addition in tensor memory cuts at the sum's last bit, see gemm_ta.cu.  With one sum per k tile, whose
// second half's lo parts met a large sum already, the K-quants were 1.5 times as far from the exact results as the kernel of
// gemm_tc.cu: 1.1e-6 of a row's results against 7.2e-7 for Q4_K, 6.7e-7 against 4.6e-7 for Q6_K; now 3.7e-7 and 3.2e-7.
// Q8_0's one sum per tile, 8.4e-7, replaced one over all inputs.)  The F32 sums of a CTA (128 x 256) live in the registers
// of sixteen warps.
// What bounds it now: the folds, 5,300 of 6,500 clocks per k tile when they read eight columns at a time (694 and 434 us); they
// read sixteen, as many as the registers hold (32: 712 us).  A thread's arrival at the other CTA's barrier must not be
// `.release.cluster`: its wait for all earlier accesses doubled the fold (1,060 us).  Fewer product columns for a group of
// few rows gained nothing at 777 and 1,047 rows: its conversion and folds remain.  An item of one row group (65 to 128 rows) pays
// for the pair's barriers without sharing a conversion: gate | up 59.5 and 63.6 us at 65 and 128 rows against 57.9 and 61.4 of
// one CTA per item.  Whole steps gained all the same (8 layers of the 8B model, 65 / 80 / 100 / 128 tokens: 1.70 / 1.64 / 1.79 / 1.76
// -> 1.59 / 1.60 / 1.64 / 1.69 ms), so the pair serves every size.
// Roles of the 28 warps: 0..15 fold and store (one row and 32 columns of each group per thread), 16..23 convert (two row
// tiles, half of a stage), 24 / 26 copy weights / activations, 25 issues MMAs in the leading CTA and tells it in the other
// what has landed there.  Every wait is bounded.
#include <cuda_fp16.h>

#include <algorithm>

#include "blocks.cuh"
#include "gemv.cuh"
#include "tmem.cuh"

namespace ribn {

namespace {

constexpr int kCols = 128;                                    // activation rows of a group
constexpr int kMineCols = kCols / 2;                          // of them in one CTA's shared memory
constexpr int kChunkBytes = kMineCols * 2 * 128 * 2;          // 128 inputs of their hi and lo parts: 32 KB
constexpr int kSumBytes = kMineCols * 16 * 2, kScaleBytes = kCols * 4, kTailBytes = kSumBytes + kScaleBytes;   // their group sums, all rows' scales
constexpr int kMainBytes = 4 * kChunkBytes, kBlockBytes = kMainBytes + 2 * kSumBytes + kScaleBytes;
constexpr int kFoldWarps = 16, kConvertWarp0 = 16, kConvertWarps = 8, kWeightWarp = 24, kMmaWarp = 25, kBlockWarp = 26;
constexpr int kThreads = 28 * 32;
constexpr int kMine = 32;                                     // columns of a group per fold thread
// Register shares: the launch gives each thread 72 (64,512 in all); fold 512 x 88, conversion 256 x 56, the rest 128 x 40.
constexpr int kFoldRegs = 88, kConvertRegs = 56, kOtherRegs = 40;
constexpr uint32_t kSpinLimit = 1u << 22;
constexpr int kWStages = 4, kBSlots = 4, kScaleSlots = 4;
constexpr int kSmemMost = 232448;
constexpr int kBarBytes = 336;

// ---- the pair: rank 0 leads (issues the products of both), barriers that both sides arrive on are rank 0's ----
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() { asm volatile("barrier.cluster.arrive;\n\tbarrier.cluster.wait;" ::: "memory"); }
// An arrival at rank 0's barrier, in the default form, which like mbar_wait synchronises threads of one CTA only; the pair's
// barriers rely on no more.  No thread reads what a thread of the other CTA wrote: what passes between them is tensor memory
// (behind tcgen05.wait and tcgen05.fence on both sides of the barrier) and shared memory that the tensor core reads through the
// asynchronous proxy (bulk copies that have landed, and the minima operand behind fence.proxy.async).  A fold thread reads its
// rows' scales, which threads of its own CTA stored before they arrived here.
__device__ __forceinline__ void arrive_leader(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .b32 r;\n\t"
        "mapa.shared::cluster.u32 r, %0, 0;\n\t"
        "mbarrier.arrive.shared::cluster.b64 _, [r];\n\t}" ::"r"(bar) : "memory");
}
// to the barrier at this place in both CTAs
__device__ __forceinline__ void commit_both(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void commit_own(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// M = 256: 128 rows from each CTA, N / 2 columns from each
constexpr uint32_t kIdescPair = (1u << 4) | ((uint32_t)(kCols >> 3) << 17) | ((uint32_t)(2 * kUnitRows >> 4) << 24);
__device__ __forceinline__ void pair_mma_ts(bool leader, uint32_t d_tmem, uint32_t a_tmem, uint32_t b_desc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 b;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %7, 0;\n\t"
        "mov.b64 b, {%2, %6};\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], b, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_desc), "r"(kIdescPair), "r"(accumulate), "r"(0u), "r"(kDescHigh), "r"((uint32_t)leader) : "memory");
}
__device__ __forceinline__ void pair_mma_ss(uint32_t d_tmem, uint32_t a_desc, uint32_t b_desc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
        "setp.ne.b32 p, %4, %4;\n\t"
        "mov.b64 a, {%1, %5};\n\t"
        "mov.b64 b, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, {%4, %4, %4, %4, %4, %4, %4, %4}, p;\n\t}"
        ::"r"(d_tmem), "r"(a_desc), "r"(b_desc), "r"(kIdescPair), "r"(0u), "r"(kDescHigh) : "memory");
}

__device__ __forceinline__ float4 lds128f(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}

// acc += sx (f x) over four columns, or sx (f x - g z)
__device__ __forceinline__ void fold_pair(float* acc, float sx0, float sx1, float2 v) {
    const float2 r = __ffma2_rn(make_float2(sx0, sx1), v, make_float2(acc[0], acc[1]));
    acc[0] = r.x; acc[1] = r.y;
}
__device__ __forceinline__ void fold4(float* acc, const float* x, float f, uint32_t sx_at) {
    const float4 s = lds128f(sx_at);
    const float2 ff = make_float2(f, f);
    fold_pair(acc, s.x, s.y, __fmul2_rn(make_float2(x[0], x[1]), ff));
    fold_pair(acc + 2, s.z, s.w, __fmul2_rn(make_float2(x[2], x[3]), ff));
}
__device__ __forceinline__ void fold4(float* acc, const float* x, const float* z, float f, float g, uint32_t sx_at) {
    const float4 s = lds128f(sx_at);
    const float2 ff = make_float2(f, f), gg = make_float2(-g, -g);
    fold_pair(acc, s.x, s.y, __ffma2_rn(make_float2(z[0], z[1]), gg, __fmul2_rn(make_float2(x[0], x[1]), ff)));
    fold_pair(acc + 2, s.z, s.w, __ffma2_rn(make_float2(z[2], z[3]), gg, __fmul2_rn(make_float2(x[2], x[3]), ff)));
}

// A stages whose products one sum holds: 128 inputs of the K-quants, a whole k tile of Q8_0.
template <int TYPE>
__device__ __forceinline__ int stages_per_sum(int type) { return type == kQ4_K ? 1 : TYPE == kKQuants || type == kQ6_K ? 2 : 4; }

template <int TYPE>
__global__ void __launch_bounds__(kThreads, 1) gemm_pf_kernel(const StepGemm a, const StepSplit split, const int w_bytes, const int nw) {
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int worker = (int)blockIdx.x >> 1;
    const uint32_t spin_limit = a.spin_limit ? a.spin_limit : kSpinLimit;
    const uint32_t b_ring = smem_u32(smem), tails = b_ring + kBSlots * kChunkBytes, a2_buf = tails + 4 * kTailBytes, scales = a2_buf + 2 * kA2Bytes,
                   inv_at = scales + kScaleSlots * kUnitRows * 4, tmem_slot = inv_at + 2 * kCols * 4, bars = tmem_slot + 16, w_ring = (bars + kBarBytes + 127) & ~127u;
    // b / t: a ring slot of activations, the tail of (k tile parity, group); _peer (of rank 0): the other CTA's has landed.
    // a: A stages, d: sums, m: the minima's sums; a_full, d_free and m_free are rank 0's
    const uint32_t w_full = bars, w_empty = bars + 32, b_full = bars + 64, b_peer = bars + 96, b_empty = bars + 128, t_full = bars + 160, t_peer = bars + 192,
                   t_empty = bars + 224, a_full = bars + 256, a_free = bars + 272, d_full = bars + 288, d_free = bars + 304, m_free = bars + 320, drained = bars + 328;
    const int k_tiles = split.k_tiles, groups = split.groups, item_groups = split.unit_items, runs = split.runs(worker);

    if (threadIdx.x == 0) {
        for (int i = 0; i < nw; ++i) { mbar_init(w_full + 8 * i, 1); mbar_init(w_empty + 8 * i, kConvertWarps); }
        for (int i = 0; i < 4; ++i) {
            mbar_init(b_full + 8 * i, 1); mbar_init(b_peer + 8 * i, 1); mbar_init(b_empty + 8 * i, 1);
            mbar_init(t_full + 8 * i, 1); mbar_init(t_peer + 8 * i, 1); mbar_init(t_empty + 8 * i, kFoldWarps);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(a_full + 8 * i, 2 * kConvertWarps); mbar_init(a_free + 8 * i, 1);
            mbar_init(d_full + 8 * i, 1); mbar_init(d_free + 8 * i, 2 * kFoldWarps);
        }
        mbar_init(m_free, 2 * kFoldWarps);
        mbar_init(drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // the other CTA's barriers and tensor memory are there
    tc_fence_after();
    const uint32_t tmem = lds32(tmem_slot);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (warp >= kWeightWarp) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
        bool alive = true;
        if (warp == kWeightWarp && lane == 0) {
            // ---------------- weights: this CTA's half of the unit; they depend on no other kernel ----------------
            int ws = 0, filled = 0;
            uint32_t parity = 1;
            for (int r = 0; r < runs && alive; ++r) {
                const StepRun run = split.run(worker, r);
                const UnitAt at = unit_at(a, run.item / item_groups, 2 * kUnitTiles);
                const GemvSegment& seg = a.seg[at.seg];
                const uint32_t bytes = kUnitTiles * (uint32_t)packed_tile_bytes(type_of<TYPE>(seg));
                for (int kb = run.begin; kb < run.end && alive; ++kb) {
                    if (filled == nw) alive = mbar_wait(w_empty + 8 * ws, parity, a.error_flag, 101, spin_limit);
                    else ++filled;
                    if (!alive) break;
                    mbar_expect_tx(w_full + 8 * ws, bytes);
                    tiles_g2s(w_ring + ws * w_bytes, seg.map, kb, at.rt0 + kUnitTiles * (int)rank, w_full + 8 * ws);
                    if (++ws == nw) { ws = 0; parity ^= 1u; }
                }
            }
            if (!alive) for (int i = 0; i < 2 * nw; ++i) mbar_wait(w_full + 8 * (i % nw), (uint32_t)(i / nw), nullptr, 0, spin_limit);
        } else if (warp == kBlockWarp && lane == 0) {
            // ---------------- activations, 64 rows of each group: per k tile the tails, then two chunks of each group ----------------
            asm volatile("griddepcontrol.wait;" ::: "memory");
            uint32_t n = 0, pos = 0, t_used = 0;   // k tiles and ring slots so far; bit i: tail i has been used an odd number of times
            for (int r = 0; r < runs && alive; ++r) {
                const StepRun run = split.run(worker, r);
                const int group0 = run.item % item_groups * 2, both = min(2, groups - group0);
                for (int kb = run.begin; kb < run.end && alive; ++kb, ++n) {
                    const unsigned char* from = a.blocks + ((size_t)group0 * k_tiles + kb) * kBlockBytes;
                    const size_t next = (size_t)k_tiles * kBlockBytes;
                    for (int u = 0; u < both && alive; ++u) {
                        const uint32_t i = 2 * (n & 1u) + u;
                        alive = mbar_wait(t_empty + 8 * i, ((t_used >> i) & 1u) ^ 1u, a.error_flag, 102, spin_limit);
                        t_used ^= 1u << i;
                        if (!alive) break;
                        mbar_expect_tx(t_full + 8 * i, kTailBytes);
                        bulk_g2s(tails + i * kTailBytes, from + u * next + kMainBytes + rank * kSumBytes, kSumBytes, t_full + 8 * i);
                        bulk_g2s(tails + i * kTailBytes + kSumBytes, from + u * next + kMainBytes + 2 * kSumBytes, kScaleBytes, t_full + 8 * i);
                    }
                    for (int j = 0; j < 2; ++j) {
                        for (int u = 0; u < both && alive; ++u, ++pos) {
                            const uint32_t slot = pos % kBSlots;
                            if (pos >= kBSlots) alive = mbar_wait(b_empty + 8 * slot, (pos / kBSlots - 1u) & 1u, a.error_flag, 103, spin_limit);
                            if (!alive) break;
                            mbar_expect_tx(b_full + 8 * slot, kChunkBytes);
                            bulk_g2s(b_ring + slot * kChunkBytes, from + u * next + (2 * rank + j) * kChunkBytes, kChunkBytes, b_full + 8 * slot);
                        }
                    }
                }
            }
            // the leader's tensor core still arrives here for the last slots: not after this block has ended
            for (uint32_t i = pos > kBSlots ? pos - kBSlots : 0u; i < pos && alive; ++i) alive = mbar_wait(b_empty + 8 * (i % kBSlots), (i / kBSlots) & 1u, a.error_flag, 115, spin_limit);
            if (!alive) {
                for (int i = 0; i < 8; ++i) { mbar_wait(b_full + 8 * (i & 3), (uint32_t)(i >> 2), nullptr, 0, spin_limit); mbar_wait(t_full + 8 * (i & 3), (uint32_t)(i >> 2), nullptr, 0, spin_limit); }
            }
        } else if (warp == kMmaWarp && rank != 0) {
            // ---------------- tell the leader what has landed here ----------------
            if (lane == 0) {
                uint32_t n = 0, pos = 0, t_used = 0;
                for (int r = 0; r < runs && alive; ++r) {
                    const StepRun run = split.run(worker, r);
                    const int both = min(2, groups - run.item % item_groups * 2);
                    for (int kb = run.begin; kb < run.end && alive; ++kb, ++n) {
                        for (int u = 0; u < both && alive; ++u) {
                            const uint32_t i = 2 * (n & 1u) + u;
                            alive = mbar_wait(t_full + 8 * i, (t_used >> i) & 1u, a.error_flag, 113, spin_limit);
                            t_used ^= 1u << i;
                            if (alive) arrive_leader(t_peer + 8 * i);
                        }
                        for (int i = 0; i < 2 * both && alive; ++i, ++pos) {
                            alive = mbar_wait(b_full + 8 * (pos % kBSlots), (pos / kBSlots) & 1u, a.error_flag, 114, spin_limit);
                            if (alive) arrive_leader(b_peer + 8 * (pos % kBSlots));
                        }
                    }
                }
            }
        } else if (warp == kMmaWarp) {
            // ---------------- products of both CTAs (the warp as a whole, one elected lane in it): stage by stage, group by group ----------------
            const bool leader = elect_one();
            constexpr uint32_t kBLbo = kMineCols * 16, kStep = 2 * kBLbo >> 4, kLo = kChunkBytes / 2 >> 4;
            const uint32_t b_desc0 = umma_desc(b_ring, kBLbo), sum_desc0 = umma_desc(tails, kBLbo), a2_desc0 = umma_desc(a2_buf, kA2Lbo);
            uint32_t n = 0, pos = 0, uses = 0, sums = 0;   // k tiles, ring slots, A stages and sums so far
            uint32_t taken = 0, t_used = 0;                // bit i: sums i (2: the minima's), tail i, used an odd number of times
            auto take = [&](uint32_t i) {
                if (alive) alive = mbar_wait(i == 2 ? m_free : d_free + 8 * i, ((taken >> i) & 1u) ^ 1u, a.error_flag, 105, spin_limit);
                taken ^= 1u << i;
            };
            for (int r = 0; r < runs; ++r) {
                const StepRun run = split.run(worker, r);
                // broadcast, so that the loop below stays on uniform registers
                const int type = TYPE >= 0 ? TYPE : __shfl_sync(0xffffffffu, a.seg[unit_at(a, run.item / item_groups, 2 * kUnitTiles).seg].type, 0);
                const int both = __shfl_sync(0xffffffffu, min(2, groups - run.item % item_groups * 2), 0);
                const bool q4k = type == kQ4_K;
                const int stages = q4k ? 2 : 4, per_sum = stages_per_sum<TYPE>(type), stop = __shfl_sync(0xffffffffu, (int)n + run.end - run.begin, 0);
                for (; (int)n < stop; ++n) {
#pragma unroll 1
                    for (int h = 0; h < stages; ++h, ++uses) {
                        const bool opens = (h & (per_sum - 1)) == 0, closes = (h & (per_sum - 1)) == per_sum - 1;   // a sum
                        const bool first = q4k || (h & 1) == 0, last = q4k || (h & 1) == 1;                        // stage of a chunk
                        const uint32_t st = uses & 1u, a_at = tmem + 384 + 64 * st;
                        if (alive) alive = mbar_wait(a_full + 8 * st, (uses >> 1) & 1u, a.error_flag, 106, spin_limit);
#pragma unroll 1
                        for (int u = 0; u < both; ++u) {
                            const uint32_t db = (sums + u) & 1u, d_main = tmem + 128 * db, slot = (pos + u) % kBSlots;
                            if (opens) take(db);
                            if (first) {
                                if (alive) alive = mbar_wait(b_full + 8 * slot, ((pos + u) / kBSlots) & 1u, a.error_flag, 104, spin_limit);
                                if (alive) alive = mbar_wait(b_peer + 8 * slot, ((pos + u) / kBSlots) & 1u, a.error_flag, 104, spin_limit);
                            }
                            tc_fence_after();
                            const uint32_t b_desc = b_desc0 + slot * (kChunkBytes >> 4) + (q4k ? 0u : (h & 1) * 4 * kStep);
                            if (q4k) {
#pragma unroll
                                for (int i = 0; i < 8; ++i) pair_mma_ts(leader, d_main, a_at + 8 * i, b_desc + kLo + i * kStep, (uint32_t)(i != 0));
#pragma unroll
                                for (int i = 0; i < 8; ++i) pair_mma_ts(leader, d_main, a_at + 8 * i, b_desc + i * kStep, 1u);
                                if (h == u) {
                                    // minima x group sums: the first group's with its first sum, the second's with its last, so that
                                    // the other's have been folded by the time the stage's products are through
                                    const uint32_t i = 2 * (n & 1u) + u;
                                    if (alive) alive = mbar_wait(t_full + 8 * i, (t_used >> i) & 1u, a.error_flag, 107, spin_limit);
                                    if (alive) alive = mbar_wait(t_peer + 8 * i, (t_used >> i) & 1u, a.error_flag, 107, spin_limit);
                                    take(2);
                                    tc_fence_after();
                                    if (leader) pair_mma_ss(tmem + 256, a2_desc0 + (n & 1u) * (kA2Bytes >> 4), sum_desc0 + i * (kTailBytes >> 4));
                                }
                            } else {
                                // position i of the stage holds step 2 (i & 1) + (i >> 1) of its 64 inputs; p2 x lo left out as in gemm_ta.cu
#pragma unroll
                                for (int i = 0; i < 4; ++i) pair_mma_ts(leader, d_main, a_at + 8 * i, b_desc + kLo + (2 * (i & 1) + (i >> 1)) * kStep, (uint32_t)(!opens || i != 0));
#pragma unroll
                                for (int i = 0; i < 4; ++i) pair_mma_ts(leader, d_main, a_at + 32 + 8 * i, b_desc + (2 * (i & 1) + (i >> 1)) * kStep, 1u);
#pragma unroll
                                for (int i = 0; i < 4; ++i) pair_mma_ts(leader, d_main, a_at + 8 * i, b_desc + (2 * (i & 1) + (i >> 1)) * kStep, 1u);
                            }
                            if (leader) {
                                if (last) commit_both(b_empty + 8 * slot);
                                if (closes) commit_both(d_full + 8 * db);
                            }
                        }
                        if (leader) commit_both(a_free + 8 * st);
                        if (closes) sums += both;
                        if (last) pos += both;
                    }
                    t_used ^= (both == 2 ? 3u : 1u) << (2 * (n & 1u));   // waited for or not
                }
            }
            if (!alive) {
                // products in flight read both CTAs' memory, which the other gives up behind the barrier below: a commit follows them all.
                // (Those behind the expired wait are issued too: a predicate against it took the fold's registers, with which a
                // prompt of 300 tokens, 4 layers of the 8B model, was 2.08 ms and not 1.81.)
                if (leader) commit_own(drained);
                mbar_wait(drained, 0, nullptr, 0, kSpinLimit);
            }
        }
    } else if (warp >= kConvertWarp0) {
        // ---------------- conversion of this CTA's 128 rows ----------------
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kConvertRegs));
        const int quadrant = warp & 3, part = (warp - kConvertWarp0) >> 2;
        bool alive = true;
        uint32_t uses = 0, n = 0, ws = 0, parity = 0;
        for (int r = 0; r < runs; ++r) {
            const StepRun run = split.run(worker, r);
            const int type = type_of<TYPE>(a.seg[unit_at(a, run.item / item_groups, 2 * kUnitTiles).seg]);
            const int stages = type == kQ4_K ? 2 : 4;
            const uint32_t row_bytes = 2 * quadrant * packed_tile_bytes(type);
            for (int kb = run.begin; kb < run.end; ++kb, ++n) {
                if (alive) alive = mbar_wait(w_full + 8 * ws, parity, a.error_flag, 109, spin_limit);
                const uint32_t tile = w_ring + ws * w_bytes + row_bytes, sc = scales + (n % kScaleSlots) * (kUnitRows * 4);
#pragma unroll 1
                for (int h = 0; h < stages; ++h, ++uses) {
                    const uint32_t st = uses & 1u, a_at = tmem + 384 + 64 * st + ((uint32_t)(32 * quadrant) << 16);
                    if (uses >= 2 && alive) alive = mbar_wait(a_free + 8 * st, ((uses >> 1) - 1u) & 1u, a.error_flag, 110, spin_limit);
                    tc_fence_after();
                    if (type == kQ4_K) {
                        convert_q4k(tile, 2 * h + part, a_at + 32 * part, sc, a2_buf + (n & 1u) * kA2Bytes, 32 * quadrant, lane);
                        if (h == 0) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the minima operand
                    } else if (TYPE == kKQuants || type == kQ6_K) {
                        convert_q6k(tile, h >> 1, part + 2 * (h & 1), a_at + 16 * part, 32, sc, 32 * quadrant, lane);
                    } else {
                        convert_q8_0(tile, h >> 1, part + 2 * (h & 1), a_at + 16 * part, 32, sc, 32 * quadrant, lane);
                    }
                    tmem_wait_st();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        arrive_leader(a_full + 8 * st);
                        if (h == stages - 1) mbar_arrive(w_empty + 8 * ws);
                    }
                }
                if (++ws == (uint32_t)nw) { ws = 0; parity ^= 1u; }
            }
        }
        // likewise the arrivals that give the last stages back
        for (uint32_t i = uses > 2u ? uses - 2u : 0u; i < uses && alive; ++i) alive = mbar_wait(a_free + 8 * (i & 1u), (i >> 1) & 1u, a.error_flag, 116, spin_limit);
    } else {
        // ---------------- fold and store: one row and 32 columns of each group ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kFoldRegs));
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int quadrant = warp & 3, col0 = kMine * (warp >> 2), row = quadrant * 32 + lane;
        bool alive = true;
        int inv_group = -1;
        uint32_t n = 0, sums = 0, used = 0;   // k tiles, sums so far; bits 0, 1: sums i, bits 2 .. 5: tail i - 2, used an odd number of times
        float* inv = reinterpret_cast<float*>(smem + (inv_at - b_ring));
        for (int r = 0; r < runs; ++r) {
            const StepRun run = split.run(worker, r);
            const int group0 = run.item % item_groups * 2, both = min(2, groups - group0);
            const UnitAt at = unit_at(a, run.item / item_groups, 2 * kUnitTiles);
            const GemvSegment& seg = a.seg[at.seg];
            const int type = type_of<TYPE>(seg), per_tile = (type == kQ4_K ? 2 : 4) / stages_per_sum<TYPE>(type);
            const bool q4k = type == kQ4_K;
            float acc[2][kMine];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
#pragma unroll
                for (int i = 0; i < kMine; ++i) acc[u][i] = 0.0f;
            }
            for (int kb = run.begin; kb < run.end; ++kb, ++n) {
                const uint32_t p = n & 1u;
#pragma unroll 1
                for (int i = 0; i < per_tile; ++i) {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        if (u == 1 && both == 1) continue;
                        const uint32_t db = (sums + u) & 1u, tail = 2 * p + u, sx_at = tails + tail * kTailBytes + kSumBytes + col0 * 4;
                        if (i == 0) {
                            if (alive) alive = mbar_wait(t_full + 8 * tail, (used >> (2 + tail)) & 1u, a.error_flag, 111, spin_limit);
                            used ^= 4u << tail;
                        }
                        if (alive) alive = mbar_wait(d_full + 8 * db, (used >> db) & 1u, a.error_flag, 112, spin_limit);
                        used ^= 1u << db;
                        tc_fence_after();
                        const float2 d = __half22float2(as_half2(lds32(scales + (n % kScaleSlots) * (kUnitRows * 4) + row * 4)));
                        const uint32_t t_at = tmem + ((uint32_t)(quadrant * 32) << 16) + col0, main_at = t_at + 128 * db;
                        if (q4k && i == u) {   // the minima came with these products
#pragma unroll
                            for (int c = 0; c < kMine; c += 8) {
                                float x[8], z[8];
                                tmem_ld8(main_at + c, x);
                                tmem_ld8(t_at + 256 + c, z);
                                tmem_wait_ld();
                                tmem_tie(x);
                                tmem_tie(z);
                                if (c == kMine - 8) { tc_fence_before(); __syncwarp(); if (lane == 0) { arrive_leader(d_free + 8 * db); arrive_leader(m_free); } }
                                fold4(&acc[u][c], x, z, d.x, d.y, sx_at + c * 4);
                                fold4(&acc[u][c + 4], x + 4, z + 4, d.x, d.y, sx_at + c * 4 + 16);
                            }
                        } else {
#pragma unroll
                            for (int c = 0; c < kMine; c += 16) {
                                float x[8], y[8];
                                tmem_ld8(main_at + c, x);
                                tmem_ld8(main_at + c + 8, y);
                                tmem_wait_ld();
                                tmem_tie(x);
                                tmem_tie(y);
                                if (c == kMine - 16) { tc_fence_before(); __syncwarp(); if (lane == 0) arrive_leader(d_free + 8 * db); }
                                fold4(&acc[u][c], x, d.x, sx_at + c * 4);
                                fold4(&acc[u][c + 4], x + 4, d.x, sx_at + c * 4 + 16);
                                fold4(&acc[u][c + 8], y, d.x, sx_at + c * 4 + 32);
                                fold4(&acc[u][c + 12], y + 4, d.x, sx_at + c * 4 + 48);
                            }
                        }
                        if (i == per_tile - 1) {
                            __syncwarp();
                            if (lane == 0) mbar_arrive(t_empty + 8 * tail);
                        }
                    }
                    sums += both;
                }
            }
            if (a.partial == nullptr && group0 != inv_group) {
                inv_group = group0;
                asm volatile("bar.sync 1, 512;" ::: "memory");   // the previous groups' factors have been read
                for (int m = warp; m < 2 * kCols; m += kFoldWarps) {
                    const int member = group0 * kCols + m;
                    float sum = 0.0f;
                    if (a.ss != nullptr && member < a.members) for (int i = lane; i < k_tiles; i += 32) sum += a.ss[(size_t)member * k_tiles + i];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                    if (lane == 0) inv[m] = a.ss != nullptr ? 1.0f / sqrtf(sum / (float)a.k + a.eps) : 1.0f;
                }
                asm volatile("bar.sync 1, 512;" ::: "memory");
            }
            const int n_index = (at.rt0 + kUnitTiles * (int)rank) * kTileRows + row;
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                if ((u == 1 && both == 1) || n_index >= seg.n) continue;
                const int group = group0 + u, live = min(kMine, a.members - group * kCols - col0);
                if (a.partial != nullptr) {
                    const StepSums to = step_sums(a, split, worker, run.part, group, col0, at.seg, n_index);
#pragma unroll
                    for (int i = 0; i < kMine; ++i) {
                        if (i < live) to.at[i * to.stride] = acc[u][i];
                    }
                } else {
                    float* y = seg.y + (size_t)(group * kCols + col0) * seg.n + n_index;
#pragma unroll
                    for (int i = 0; i < kMine; ++i) {
                        if (i >= live) continue;
                        const float v = acc[u][i] * inv[u * kCols + col0 + i];
                        y[(size_t)i * seg.n] = a.epilogue == kResidual ? y[(size_t)i * seg.n] + v : v;
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // nothing of the other CTA reaches here any more
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

template <int TYPE>
cudaError_t launch_typed(cudaStream_t stream, const StepGemm& a, int w_bytes, bool programmatic) {
    static bool configured[kMaxDevices] = {false};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    if (!configured[dev]) {
        e = cudaFuncSetAttribute(gemm_pf_kernel<TYPE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMost);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    w_bytes = (w_bytes + 127) & ~127;
    const int fixed = kBSlots * kChunkBytes + 4 * kTailBytes + 2 * kA2Bytes + kScaleSlots * kUnitRows * 4 + 2 * kCols * 4 + 16 + kBarBytes + 127;
    const int nw = std::min(kWStages, (kSmemMost - fixed) / w_bytes);
    if (nw < 2) return cudaErrorInvalidValue;
    const StepSplit split = step_split(a, a.partial == nullptr);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * split.workers));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)(fixed + nw * w_bytes);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, gemm_pf_kernel<TYPE>, a, split, w_bytes, nw);
}

}  // namespace

cudaError_t launch_gemm_pf(cudaStream_t stream, const StepGemm& a, int w_bytes, bool programmatic) {
    switch (common_type(a)) {
        case kQ6_K: return launch_typed<kQ6_K>(stream, a, w_bytes, programmatic);
        case kQ8_0: return launch_typed<kQ8_0>(stream, a, w_bytes, programmatic);
        case kQ4_K:   // compiled for Q4_K alone, the fold's registers spill (o_proj 105 -> 111 us at 2,048 rows)
        case kKQuants: return launch_typed<kKQuants>(stream, a, w_bytes, programmatic);
        default: return launch_typed<kAnyType>(stream, a, w_bytes, programmatic);
    }
}

}  // namespace ribn
