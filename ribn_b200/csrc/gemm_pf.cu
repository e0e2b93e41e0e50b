// Dequant-GEMM for prefill-sized steps: 256 weight rows x 128 activation rows per work item, the
// converted weights in tensor memory (the arithmetic of gemm_ta.cu).
//
// What bounds it.  An activation is four bytes (a binary16 hi + lo pair) per input, so a 128-row unit that multiplies T
// activation rows pulls T KB per 256 inputs out of L2 for T x 16 clocks of products: 64 bytes per clock and SM, twice what
// L2 delivers to all SMs together.  TWO units per CTA share every activation chunk that arrives (170 KB against 4,096
// clocks of products per k tile), and the chunk meets the packed weights' conversion once per 128 activation rows.
//
// Tensor memory: sums of unit u at columns 128 u (one accumulator for hi and lo parts, lo first), minima sums at 256
// (shared by the units in turn), A stages at 384 + 64 u: 128 inputs of Q4_K's one plane, 64 inputs of the others' two.  The
// units alternate stage by stage, so a unit's conversion hides under the other unit's products, and so does the fold of
// its sums: once per 128 inputs of the K-quants, once per k tile of Q8_0.  (An addition in tensor memory cuts at the sum's
// last bit, see gemm_ta.cu.  With one sum per k tile, whose second half's lo parts met a large sum already, the K-quants were
// 1.5 times as far from the exact results as the kernel of gemm_tc.cu: 1.1e-6 of a row's results against 7.2e-7 for Q4_K,
// 6.7e-7 against 4.6e-7 for Q6_K; now 3.7e-7 and 3.2e-7.  The additional reads of tensor memory beside the products take
// time: gate | up of the 8B model 689 -> 746 us at 2,048 rows, down 450 -> 516 us.  A third set of sums in turn for Q6_K took
// 490 us for down by itself, and a chunk as long as before; reads of 16 columns at a time, or sums handed back before the
// reads, changed nothing; both halves' A operand resident, with the minima folded first in the products' columns, took
// 917 us for gate | up.  Q8_0's one sum per tile, 8.4e-7, replaced one over all inputs.)  The F32 sums of a work item
// (2 x 128 x 128) live in the registers of sixteen warps.
// Roles of the 28 warps: 0..15 fold and store (one row of each unit and 32 columns per thread), 16..23 convert (two row
// tiles, half of a stage), 24 / 26 copy weights / activations, 25 issues MMAs.  Every wait is bounded.
#include <cuda_fp16.h>

#include <algorithm>

#include "blocks.cuh"
#include "gemv.cuh"
#include "tmem.cuh"

namespace ribn {

namespace {

constexpr int kCols = 128;                                    // activation rows per item
constexpr int kChunkBytes = kCols * 2 * 128 * 2;              // 128 inputs of hi and lo parts: 64 KB
constexpr int kSumBytes = kCols * 16 * 2, kTailBytes = kSumBytes + kCols * 4;   // group sums, then the tile scales
constexpr int kBlockBytes = 2 * kChunkBytes + kTailBytes;
constexpr int kFoldWarps = 16, kConvertWarp0 = 16, kConvertWarps = 8, kWeightWarp = 24, kMmaWarp = 25, kBlockWarp = 26;
constexpr int kThreads = 28 * 32;
constexpr int kMine = 32;                                     // columns per fold thread
// Register shares: the launch gives each thread 72 (64,512 in all); fold 512 x 88, conversion 256 x 56, the rest 128 x 40.
constexpr int kFoldRegs = 88, kConvertRegs = 56, kOtherRegs = 40;
constexpr uint32_t kSpinLimit = 1u << 22;
constexpr int kWStages = 4;
constexpr int kSmemMost = 232448;
constexpr int kBarBytes = 208;

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
    const uint32_t spin_limit = a.spin_limit ? a.spin_limit : kSpinLimit;
    const uint32_t b_ring = smem_u32(smem), tails = b_ring + 2 * kChunkBytes, a2_buf = tails + 2 * kTailBytes, scales = a2_buf + 2 * kA2Bytes,
                   inv_at = scales + 4 * kUnitRows * 4, tmem_slot = inv_at + kCols * 4, bars = tmem_slot + 16, w_ring = (bars + kBarBytes + 127) & ~127u;
    const uint32_t w_full = bars, w_empty = bars + 32, b_full = bars + 64, b_empty = bars + 80, a_full = bars + 96, a_free = bars + 112,
                   d_full = bars + 128, d_free = bars + 152, t_full = bars + 176, t_empty = bars + 192;
    const int k_tiles = split.k_tiles, groups = split.groups, runs = split.runs((int)blockIdx.x);   // item = pair of units * groups + group

    if (threadIdx.x == 0) {
        for (int i = 0; i < nw; ++i) { mbar_init(w_full + 8 * i, 1); mbar_init(w_empty + 8 * i, kConvertWarps); }
        for (int i = 0; i < 2; ++i) {
            mbar_init(b_full + 8 * i, 1); mbar_init(b_empty + 8 * i, 1);
            mbar_init(a_full + 8 * i, kConvertWarps); mbar_init(a_free + 8 * i, 1);
            mbar_init(t_full + 8 * i, 1); mbar_init(t_empty + 8 * i, kFoldWarps);
        }
        for (int i = 0; i < 3; ++i) { mbar_init(d_full + 8 * i, 1); mbar_init(d_free + 8 * i, kFoldWarps); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMmaWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = lds32(tmem_slot);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (warp >= kWeightWarp) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
        bool alive = true;
        if (warp == kWeightWarp && lane == 0) {
            // ---------------- weights: the two units of a pair in turn; they depend on no other kernel ----------------
            int ws = 0, filled = 0;
            uint32_t parity = 1;
            for (int r = 0; r < runs && alive; ++r) {
                const StepRun run = split.run((int)blockIdx.x, r);
                const UnitAt at = unit_at(a, run.item / groups, 2 * kUnitTiles);
                const GemvSegment& seg = a.seg[at.seg];
                const uint32_t bytes = kUnitTiles * (uint32_t)packed_tile_bytes(type_of<TYPE>(seg));
                for (int kb = run.begin; kb < run.end && alive; ++kb) {
                    for (int u = 0; u < 2 && alive; ++u) {
                        if (filled == nw) alive = mbar_wait(w_empty + 8 * ws, parity, a.error_flag, 101, spin_limit);
                        else ++filled;
                        if (!alive) break;
                        mbar_expect_tx(w_full + 8 * ws, bytes);
                        tiles_g2s(w_ring + ws * w_bytes, seg.map, kb, at.rt0 + kUnitTiles * u, w_full + 8 * ws);
                        if (++ws == nw) { ws = 0; parity ^= 1u; }
                    }
                }
            }
            if (!alive) for (int i = 0; i < 2 * nw; ++i) mbar_wait(w_full + 8 * (i % nw), (uint32_t)(i / nw), nullptr, 0, spin_limit);
        } else if (warp == kBlockWarp && lane == 0) {
            // ---------------- activations: per k tile the sums and scales, then two chunks ----------------
            asm volatile("griddepcontrol.wait;" ::: "memory");
            uint32_t n = 0;   // k tiles so far
            for (int r = 0; r < runs && alive; ++r) {
                const StepRun run = split.run((int)blockIdx.x, r);
                const unsigned char* from = a.blocks + ((size_t)(run.item % groups) * k_tiles + run.begin) * kBlockBytes;
                for (int kb = run.begin; kb < run.end && alive; ++kb, ++n, from += kBlockBytes) {
                    const uint32_t p = n & 1u;
                    if (n >= 2) alive = mbar_wait(t_empty + 8 * p, ((n >> 1) - 1u) & 1u, a.error_flag, 102, spin_limit);
                    if (!alive) break;
                    mbar_expect_tx(t_full + 8 * p, kTailBytes);
                    bulk_g2s(tails + p * kTailBytes, from + 2 * kChunkBytes, kTailBytes, t_full + 8 * p);
                    for (int j = 0; j < 2; ++j) {
                        if (n >= 1) alive = mbar_wait(b_empty + 8 * j, (n - 1u) & 1u, a.error_flag, 103, spin_limit);
                        if (!alive) break;
                        mbar_expect_tx(b_full + 8 * j, kChunkBytes);
                        bulk_g2s(b_ring + j * kChunkBytes, from + j * kChunkBytes, kChunkBytes, b_full + 8 * j);
                    }
                }
            }
            if (!alive) {
                for (int i = 0; i < 4; ++i) { mbar_wait(b_full + 8 * (i & 1), (uint32_t)(i >> 1), nullptr, 0, spin_limit); mbar_wait(t_full + 8 * (i & 1), (uint32_t)(i >> 1), nullptr, 0, spin_limit); }
            }
        } else if (warp == kMmaWarp) {
            // ---------------- MMA issue (the warp as a whole, one elected lane in it): stage by stage, unit 0 then unit 1 ----------------
            const bool leader = elect_one();
            constexpr uint32_t kBLbo = 2 * kCols * 16, kStep = 2 * kBLbo >> 4, kLo = kCols * 16 >> 4;
            constexpr uint32_t idesc = umma_idesc(kCols);
            const uint32_t b_desc0 = umma_desc(b_ring, kBLbo), sum_desc0 = umma_desc(tails, kCols * 16), a2_desc0 = umma_desc(a2_buf, kA2Lbo);
            uint32_t n = 0, uses = 0;   // k tiles, A stages per unit
            uint32_t taken = 0;         // bit i: sums i (a unit's, or 2: the minima's) have been taken an odd number of times
            auto take = [&](uint32_t i) {
                if (alive) alive = mbar_wait(d_free + 8 * i, ((taken >> i) & 1u) ^ 1u, a.error_flag, 105, spin_limit);
                taken ^= 1u << i;
            };
            for (int r = 0; r < runs; ++r) {
                const StepRun run = split.run((int)blockIdx.x, r);
                // broadcast, so that the loop below stays on uniform registers
                const int type = TYPE >= 0 ? TYPE : __shfl_sync(0xffffffffu, a.seg[unit_at(a, run.item / groups, 2 * kUnitTiles).seg].type, 0);
                const bool q4k = type == kQ4_K;
                const int stages = q4k ? 2 : 4, per_sum = stages_per_sum<TYPE>(type), stop = __shfl_sync(0xffffffffu, (int)n + run.end - run.begin, 0);
                for (; (int)n < stop; ++n) {
#pragma unroll 1
                    for (int h = 0; h < stages; ++h, ++uses) {
                        const int chunk = q4k ? h : h >> 1;
                        const bool opens = (h & (per_sum - 1)) == 0, closes = (h & (per_sum - 1)) == per_sum - 1;   // a sum
                        if (q4k || !(h & 1)) { if (alive) alive = mbar_wait(b_full + 8 * chunk, n & 1u, a.error_flag, 104, spin_limit); }
                        const uint32_t b_desc = b_desc0 + chunk * (kChunkBytes >> 4) + (q4k ? 0u : (h & 1) * 4 * kStep);
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const uint32_t d_main = tmem + 128 * u, a_at = tmem + 384 + 64 * u;
                            if (opens) take(u);
                            if (alive) alive = mbar_wait(a_full + 8 * u, uses & 1u, a.error_flag, 106, spin_limit);
                            tc_fence_after();
                            if (q4k) {
#pragma unroll
                                for (int i = 0; i < 8; ++i) umma_ts_if(leader, d_main, a_at + 8 * i, b_desc + kLo + i * kStep, idesc, (uint32_t)(i != 0));
#pragma unroll
                                for (int i = 0; i < 8; ++i) umma_ts_if(leader, d_main, a_at + 8 * i, b_desc + i * kStep, idesc, 1u);
                                if (h == u) {
                                    // minima x group sums: unit 0's with its first stage, unit 1's with its last, so that the
                                    // other unit's have been folded by the time the stage's products are through
                                    if (u == 0 && alive) alive = mbar_wait(t_full + 8 * (n & 1u), (n >> 1) & 1u, a.error_flag, 107, spin_limit);
                                    take(2);
                                    tc_fence_after();
                                    if (leader) umma_ss(tmem + 256, a2_desc0 + u * (kA2Bytes >> 4), sum_desc0 + (n & 1u) * (kTailBytes >> 4), idesc, 0u);
                                }
                            } else {
                                // position i of the stage holds step 2 (i & 1) + (i >> 1) of its 64 inputs; p2 x lo left out as in gemm_ta.cu
#pragma unroll
                                for (int i = 0; i < 4; ++i) umma_ts_if(leader, d_main, a_at + 8 * i, b_desc + kLo + (2 * (i & 1) + (i >> 1)) * kStep, idesc, (uint32_t)(!opens || i != 0));
#pragma unroll
                                for (int i = 0; i < 4; ++i) umma_ts_if(leader, d_main, a_at + 32 + 8 * i, b_desc + (2 * (i & 1) + (i >> 1)) * kStep, idesc, 1u);
#pragma unroll
                                for (int i = 0; i < 4; ++i) umma_ts_if(leader, d_main, a_at + 8 * i, b_desc + (2 * (i & 1) + (i >> 1)) * kStep, idesc, 1u);
                            }
                            if (leader) {
                                umma_commit(a_free + 8 * u);
                                if (closes) umma_commit(d_full + 8 * u);
                            }
                        }
                        if (leader && (q4k || (h & 1))) umma_commit(b_empty + 8 * chunk);
                    }
                }
            }
        }
    } else if (warp >= kConvertWarp0) {
        // ---------------- conversion ----------------
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kConvertRegs));
        const int quadrant = warp & 3, part = (warp - kConvertWarp0) >> 2;
        bool alive = true;
        uint32_t uses = 0, n = 0, ws0 = 0, wp0 = 0;   // ws0 / wp0: ring place and phase of the k tile's first unit
        for (int r = 0; r < runs; ++r) {
            const StepRun run = split.run((int)blockIdx.x, r);
            const int type = type_of<TYPE>(a.seg[unit_at(a, run.item / groups, 2 * kUnitTiles).seg]);
            const int stages = type == kQ4_K ? 2 : 4;
            const uint32_t row_bytes = 2 * quadrant * packed_tile_bytes(type);
            for (int kb = run.begin; kb < run.end; ++kb, ++n) {
                const uint32_t wrap = ws0 + 1 == (uint32_t)nw, ws1 = wrap ? 0u : ws0 + 1, wp1 = wp0 ^ wrap;
#pragma unroll 1
                for (int h = 0; h < stages; ++h, ++uses) {
#pragma unroll 1
                    for (int u = 0; u < 2; ++u) {
                        const uint32_t ws = u ? ws1 : ws0;
                        if (h == 0 && alive) alive = mbar_wait(w_full + 8 * ws, u ? wp1 : wp0, a.error_flag, 109, spin_limit);
                        if (uses >= 1 && alive) alive = mbar_wait(a_free + 8 * u, (uses - 1u) & 1u, a.error_flag, 110, spin_limit);
                        tc_fence_after();
                        const uint32_t tile = w_ring + ws * w_bytes + row_bytes, a_at = tmem + 384 + 64 * u + ((uint32_t)(32 * quadrant) << 16);
                        const uint32_t sc = scales + (2 * (n & 1u) + u) * (kUnitRows * 4);
                        if (type == kQ4_K) {
                            convert_q4k(tile, 2 * h + part, a_at + 32 * part, sc, a2_buf + u * kA2Bytes, 32 * quadrant, lane);
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
                            mbar_arrive(a_full + 8 * u);
                            if (h == stages - 1) mbar_arrive(w_empty + 8 * ws);
                        }
                    }
                }
                wp0 = wp1 ^ (ws1 + 1 == (uint32_t)nw);
                ws0 = ws1 + 1 == (uint32_t)nw ? 0u : ws1 + 1;
            }
        }
    } else {
        // ---------------- fold and store ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kFoldRegs));
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int quadrant = warp & 3, col0 = kMine * (warp >> 2), row = quadrant * 32 + lane;
        bool alive = true;
        int inv_group = -1;
        uint32_t n = 0, folds = 0;   // k tiles, sums per unit
        float* inv = reinterpret_cast<float*>(smem + (inv_at - b_ring));
        for (int r = 0; r < runs; ++r) {
            const StepRun run = split.run((int)blockIdx.x, r);
            const int group = run.item % groups;
            const UnitAt at = unit_at(a, run.item / groups, 2 * kUnitTiles);
            const GemvSegment& seg = a.seg[at.seg];
            const int type = type_of<TYPE>(seg), sums = (type == kQ4_K ? 2 : 4) / stages_per_sum<TYPE>(type);
            const bool q4k = type == kQ4_K;
            float acc[2][kMine];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
#pragma unroll
                for (int i = 0; i < kMine; ++i) acc[u][i] = 0.0f;
            }
            for (int kb = run.begin; kb < run.end; ++kb, ++n) {
                const uint32_t p = n & 1u, sx_at = tails + p * kTailBytes + kSumBytes + col0 * 4;
                if (alive) alive = mbar_wait(t_full + 8 * p, (n >> 1) & 1u, a.error_flag, 111, spin_limit);
#pragma unroll 1
                for (int i = 0; i < sums; ++i, ++folds) {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
                        if (alive) alive = mbar_wait(d_full + 8 * u, folds & 1u, a.error_flag, 112, spin_limit);
                        tc_fence_after();
                        const float2 d = __half22float2(as_half2(lds32(scales + (2 * p + u) * (kUnitRows * 4) + row * 4)));
                        const uint32_t t_at = tmem + ((uint32_t)(quadrant * 32) << 16) + col0;
                        if (q4k && i == u) {   // the minima came with these products
#pragma unroll
                            for (int c = 0; c < kMine; c += 4) {
                                float x[4], z[4];
                                tmem_ld4(t_at + 128 * u + c, x);
                                tmem_ld4(t_at + 256 + c, z);
                                tmem_wait_ld();
                                tmem_tie(x);
                                tmem_tie(z);
                                if (c == kMine - 4) { tc_fence_before(); __syncwarp(); if (lane == 0) { mbar_arrive(d_free + 8 * u); mbar_arrive(d_free + 16); } }
                                fold4(&acc[u][c], x, z, d.x, d.y, sx_at + c * 4);
                            }
                        } else {
#pragma unroll
                            for (int c = 0; c < kMine; c += 8) {
                                float x[8];
                                tmem_ld8(t_at + 128 * u + c, x);
                                tmem_wait_ld();
                                tmem_tie(x);
                                if (c == kMine - 8) { tc_fence_before(); __syncwarp(); if (lane == 0) mbar_arrive(d_free + 8 * u); }
                                fold4(&acc[u][c], x, d.x, sx_at + c * 4);
                                fold4(&acc[u][c + 4], x + 4, d.x, sx_at + c * 4 + 16);
                            }
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(t_empty + 8 * p);
            }
            if (a.partial == nullptr && group != inv_group) {
                inv_group = group;
                asm volatile("bar.sync 1, 512;" ::: "memory");   // the previous group's factors have been read
                for (int m = warp; m < kCols; m += kFoldWarps) {
                    const int member = group * kCols + m;
                    float sum = 0.0f;
                    if (a.ss != nullptr && member < a.members) for (int i = lane; i < k_tiles; i += 32) sum += a.ss[(size_t)member * k_tiles + i];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                    if (lane == 0) inv[m] = a.ss != nullptr ? 1.0f / sqrtf(sum / (float)a.k + a.eps) : 1.0f;
                }
                asm volatile("bar.sync 1, 512;" ::: "memory");
            }
            const int live = min(kMine, a.members - group * kCols - col0);
            const StepSums to = step_sums(a, split, (int)blockIdx.x, run.part, group, col0, at.seg, at.rt0 * kTileRows + row);
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int n_index = (at.rt0 + kUnitTiles * u) * kTileRows + row;
                if (n_index >= seg.n) continue;
                if (a.partial != nullptr) {
#pragma unroll
                    for (int i = 0; i < kMine; ++i) {
                        if (i < live) to.at[i * to.stride + kUnitRows * u] = acc[u][i];
                    }
                } else {
                    float* y = seg.y + (size_t)(group * kCols + col0) * seg.n + n_index;
#pragma unroll
                    for (int i = 0; i < kMine; ++i) {
                        if (i >= live) continue;
                        const float v = acc[u][i] * inv[col0 + i];
                        y[(size_t)i * seg.n] = a.epilogue == kResidual ? y[(size_t)i * seg.n] + v : v;
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
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
    const int fixed = 2 * kChunkBytes + 2 * kTailBytes + 2 * kA2Bytes + 4 * kUnitRows * 4 + kCols * 4 + 16 + kBarBytes + 127;
    const int nw = std::min(kWStages, (kSmemMost - fixed) / w_bytes);
    if (nw < 2) return cudaErrorInvalidValue;
    const StepSplit split = step_split(a, a.partial == nullptr);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)split.workers);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)(fixed + nw * w_bytes);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 1 : 0;
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
