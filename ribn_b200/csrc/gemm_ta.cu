// Dequant-GEMM with the converted weights in TENSOR MEMORY (tcgen05, A operand in TMEM).
//
//   y[m][n] = sum_k deq(W[n][k]) x[m][k]
//
// The tensor core multiplies the blocks' exact integers, as binary16, by the activations' binary16 hi + lo pairs:
// sc q (at most 945) for Q4_K, sc (q - 32) (up to 4096 in magnitude, as p1 = its value rounded to binary16 and the exact
// rest p2) for Q6_K; d q (d scaled by a power of two per row and 256 inputs, again in two parts) for Q8_0.  Per 256 inputs the F32 sums leave tensor memory and are folded into F32 registers with the row's
// super-block scale d and the activations' power-of-two tile scale, round-to-nearest, in order; the Q4_K minima are one
// more K = 16 MMA per 256 inputs against the activations' group sums.
//
// What bounds a small batch is everything but the products: a 128-row, 256-input tile of Q4_K is 18 KB of HBM traffic
// (about 820 clocks of one SM's share) and 32,768 weights to convert.  The MMA-fragment kernel (gemm_frag.cu) re-reads
// the activations' fragments from shared memory for every row-tile pair and was measured at about 1,300 clocks a tile
// from eight rows on; staging a converted A operand through shared memory costs 64 KB written and read back per tile.
// Here a conversion warp keeps the packed tile's own fragment order (lane = row g / g + 8, input pairs 4 t + ..): that
// is exactly the register layout of `tcgen05.st.16x128b`, so converted pairs go straight to tensor memory, and shared
// memory carries the packed bytes and the activations only.
//
// Roles of the 20 warps: 0..7 fold and store (one output row per thread, every other eight of the rows of activations),
// 8..15 convert (tensor-memory lane quadrant = warp & 3, so two row tiles each; half of the tile's inputs), 16 / 18 copy
// weights / activations, 17 issues MMAs.  A hand-off to or from the tensor core costs the MMA-issuing thread some 0.2 us
// (measured: with the products and the conversion left out, a k tile with three `tcgen05.commit`s still took 1,900 clocks), so
// a k tile has ONE commit (two for Q6_K, whose A operand fills two stages), which frees its A stage and starts its fold; one
// arrival per fold warp frees the sums and the activations' slot.
// Tensor memory: main sums of k tile parity p at columns 64 p, at 128 + 64 p the minima sums of Q4_K or the sums of
// Q6_K's second half, A stages at 256 + 128 s (256 inputs of Q4_K's one plane, 128 inputs of the others' two).
// An addition in tensor memory cuts at the sum's last bit, so its error grows with the number of steps that a sum is already
// large in.  With one sum per tile and p1 before p2, Q6_K was 1.5 times as far from the exact results as the kernel of
// gemm_tc.cu (6.7e-7 against 4.6e-7 of a row's results at 48 and more columns); with a sum per half and the small parts
// first it is at 2.0e-7, for 0.7 % of a step of 64 rows.  Q8_0's one sum per tile (5.2e-7, 7.1e-7 at 48 and more columns)
// replaced one over all inputs there (2.7e-6 to 2.9e-5); a sum per half (2.0e-7) would cost 4 % of a step of 32 rows of
// the 0.6B model.  Slots (unit, k tile) are dealt to the CTAs evenly when another kernel finishes the sums, in
// whole items otherwise (StepSplit).  Every wait is bounded.
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "blocks.cuh"
#include "gemv.cuh"
#include "tmem.cuh"

namespace ribn {

namespace {

constexpr int kEpilogueWarps = 8, kConvertWarp0 = 8, kConvertWarps = 8, kWeightWarp = 16, kMmaWarp = 17, kBlockWarp = 18;
constexpr int kThreads = 20 * 32;
// Register shares: the launch gives each thread 96 (61,440 in all); conversion 256 x 96, fold 256 x 112, the rest 128 x 64.
constexpr int kEpilogueRegs = 112, kOtherRegs = 64;
constexpr uint32_t kSpinLimit = 1u << 22;
constexpr size_t kSmemBudget = 224 * 1024;

// Columns of a launch's operand: MP rows of activations, in one group.
template <int MP>
struct Cols {
    static constexpr bool kJoined = MP <= 32;               // hi and lo parts side by side in one MMA, or one after the other
    static constexpr int kSumCols = (MP + 15) / 16 * 16;
    static constexpr int kMain = 1024 * MP, kSums = 32 * kSumCols;
    static constexpr int kBlock = kMain + kSums + 4 * MP;
};

struct TaRings { int w_stages, b_stages, w_bytes; };

template <int MP, int TYPE>
__global__ void __launch_bounds__(kThreads, 1) gemm_ta_kernel(const StepGemm a, const StepSplit split, const TaRings rings) {
    using C = Cols<MP>;
    constexpr int kBBytes = (C::kBlock + 127) & ~127;
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t spin_limit = a.spin_limit ? a.spin_limit : kSpinLimit;
    const int nw = rings.w_stages, nb = rings.b_stages, k_tiles = split.k_tiles;
    const uint32_t w_ring = smem_u32(smem), b_ring = w_ring + nw * rings.w_bytes, a2_buf = b_ring + nb * kBBytes,
                   scales_ring = a2_buf + 2 * kA2Bytes, inv_at = scales_ring + 4 * kUnitRows * 4, tmem_slot = inv_at + MP * 4, bars = tmem_slot + 16;
    // done: the k tile's products are complete (ring of nb); half: those of a Q6_K tile's first A stage; folded: the k tile's
    // sums and activations are free (ring of nb).  Each waiting role sees every phase of a barrier, or none it has not passed.
    const uint32_t w_full = bars, w_empty = bars + 64, b_full = bars + 128, folded = bars + 192, done = bars + 256, a_full = bars + 320, half_done = bars + 336;
    const int s0 = split.begin((int)blockIdx.x), s1 = split.begin((int)blockIdx.x + 1);

    if (threadIdx.x == 0) {
        for (int i = 0; i < nw; ++i) { mbar_init(w_full + 8 * i, 1); mbar_init(w_empty + 8 * i, kConvertWarps); }
        for (int i = 0; i < nb; ++i) { mbar_init(b_full + 8 * i, 1); mbar_init(folded + 8 * i, kEpilogueWarps); mbar_init(done + 8 * i, 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(a_full + 8 * i, kConvertWarps); mbar_init(half_done + 8 * i, 1); }
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
            // ---------------- weights: they depend on no other kernel ----------------
            int ws = 0, filled = 0;
            uint32_t parity = 1;
            for (int s = s0; s < s1 && alive;) {
                const int unit = s / k_tiles, end = min(s1, (unit + 1) * k_tiles);
                const UnitAt at = unit_at(a, unit, kUnitTiles);
                const GemvSegment& seg = a.seg[at.seg];
                const uint32_t bytes = kUnitTiles * (uint32_t)packed_tile_bytes(type_of<TYPE>(seg));
                for (int kb = s - unit * k_tiles; s < end; ++s, ++kb) {
                    if (filled == nw) alive = mbar_wait(w_empty + 8 * ws, parity, a.error_flag, 91, spin_limit);
                    else ++filled;
                    if (!alive) break;
                    mbar_expect_tx(w_full + 8 * ws, bytes);
                    tiles_g2s(w_ring + ws * rings.w_bytes, seg.map, kb, at.rt0, w_full + 8 * ws);
                    if (++ws == nw) { ws = 0; parity ^= 1u; }
                }
            }
            if (!alive) for (int i = 0; i < 2 * nw; ++i) mbar_wait(w_full + 8 * (i % nw), (uint32_t)(i / nw), nullptr, 0, spin_limit);
        } else if (warp == kBlockWarp && lane == 0) {
            // ---------------- activations, from the previous kernel ----------------
            asm volatile("griddepcontrol.wait;" ::: "memory");
            int bs = 0, filled = 0;
            uint32_t parity = 1;
            for (int s = s0; s < s1 && alive;) {
                const int unit = s / k_tiles, end = min(s1, (unit + 1) * k_tiles);
                const unsigned char* from = a.blocks + (size_t)(s - unit * k_tiles) * C::kBlock;
                for (; s < end; ++s, from += C::kBlock) {
                    if (filled == nb) alive = mbar_wait(folded + 8 * bs, parity, a.error_flag, 92, spin_limit);
                    else ++filled;
                    if (!alive) break;
                    mbar_expect_tx(b_full + 8 * bs, C::kBlock);
                    bulk_g2s(b_ring + bs * kBBytes, from, C::kBlock, b_full + 8 * bs);
                    if (++bs == nb) { bs = 0; parity ^= 1u; }
                }
            }
            if (!alive) for (int i = 0; i < 2 * nb; ++i) mbar_wait(b_full + 8 * (i % nb), (uint32_t)(i / nb), nullptr, 0, spin_limit);
        } else if (warp == kMmaWarp) {
            // ---------------- MMA issue (the warp as a whole, one elected lane in it) ----------------
            const bool leader = elect_one();
            constexpr uint32_t kBLbo = 2 * MP * 16;
            constexpr uint32_t kStep = 2 * kBLbo >> 4, kLo = MP * 16 >> 4;   // descriptor units: a k16 step, the lo columns
            constexpr uint32_t idesc_both = umma_idesc(2 * MP), idesc_one = umma_idesc(MP), idesc_sum = umma_idesc(C::kSumCols);
            const uint32_t b_desc0 = umma_desc(b_ring, kBLbo), sum_desc0 = umma_desc(b_ring + C::kMain, C::kSumCols * 16),
                           a2_desc0 = umma_desc(a2_buf, kA2Lbo);
            int bs = 0, fold_slot = 0;
            uint32_t b_parity = 0, fold_parity = 0, a_count = 0, kt = 0, q6_count = 0;
            for (int s = s0; s < s1;) {
                const int unit = s / k_tiles, end = min(s1, (unit + 1) * k_tiles);
                const int type = type_of<TYPE>(a.seg[unit_at(a, unit, kUnitTiles).seg]);
                const bool q4k = type == kQ4_K, q6k = TYPE == kKQuants ? !q4k : type == kQ6_K;
                for (; s < end; ++s, ++kt) {
                    const uint32_t p = kt & 1u, d_main = tmem + 64 * p, d_min = tmem + 128 + 64 * p;
                    if (kt >= 2) {   // the fold of k tile kt - 2 has left these sums
                        if (alive) alive = mbar_wait(folded + 8 * fold_slot, fold_parity, a.error_flag, 93, spin_limit);
                        if (++fold_slot == nb) { fold_slot = 0; fold_parity ^= 1u; }
                    }
                    if (alive) alive = mbar_wait(b_full + 8 * bs, b_parity, a.error_flag, 94, spin_limit);
                    const uint32_t b_desc = b_desc0 + (uint32_t)(bs * (kBBytes >> 4));
                    const uint32_t st = a_count & 1u, a_at = tmem + 256 + 128 * st;
                    if (alive) alive = mbar_wait(a_full + 8 * st, (a_count >> 1) & 1u, a.error_flag, 95, spin_limit);
                    tc_fence_after();
                    if (q4k) {
                        if (leader) {
                            umma_ss(d_min, a2_desc0 + st * (kA2Bytes >> 4), sum_desc0 + bs * (kBBytes >> 4), idesc_sum, 0u);
                            if (C::kJoined) {
#pragma unroll
                                for (int i = 0; i < 16; ++i) umma_ts(d_main, a_at + 8 * i, b_desc + i * kStep, idesc_both, i != 0);
                            } else {   // lo parts first: the sums they join are still small
#pragma unroll
                                for (int i = 0; i < 16; ++i) umma_ts(d_main, a_at + 8 * i, b_desc + kLo + i * kStep, idesc_one, i != 0);
#pragma unroll
                                for (int i = 0; i < 16; ++i) umma_ts(d_main, a_at + 8 * i, b_desc + i * kStep, idesc_one, 1u);
                            }
                            umma_commit(done + 8 * bs);
                        }
                        ++a_count;
                    } else {
#pragma unroll 1
                        for (int half = 0; half < 2; ++half, ++a_count) {
                            const uint32_t hs = a_count & 1u, h_at = tmem + 256 + 128 * hs;
                            if (half == 1) {
                                if (alive) alive = mbar_wait(a_full + 8 * hs, (a_count >> 1) & 1u, a.error_flag, 95, spin_limit);
                                tc_fence_after();
                            }
                            const uint32_t b_half = b_desc + 8 * half * kStep, d_half = half == 1 && q6k ? d_min : d_main;
                            // position i of the stage holds step 4 (i >> 2) + 2 (i & 1) + ((i >> 1) & 1) of the half.  The
                            // small parts first.  p2 x lo is left out where it costs an MMA: at most 2^-22 of a product, and
                            // only p of more than eleven bits have a p2, so that it is 3e-8 of a row's result
                            if (leader) {
#pragma unroll
                                for (int pass = C::kJoined ? 1 : 0; pass < 3; ++pass) {   // (p1 x lo apart,) p2, p1
#pragma unroll
                                    for (int i = 0; i < 8; ++i) {
                                        const uint32_t b = b_half + (4 * (i >> 2) + 2 * (i & 1) + ((i >> 1) & 1)) * kStep;
                                        const uint32_t acc = i != 0 || pass != (C::kJoined ? 1 : 0) || (half == 1 && !q6k);
                                        if (pass == 0) umma_ts(d_half, h_at + 8 * i, b + kLo, idesc_one, acc);
                                        else umma_ts(d_half, h_at + (pass == 1 ? 64 : 0) + 8 * i, b, C::kJoined ? idesc_both : idesc_one, acc);
                                    }
                                }
                                umma_commit(half == 0 ? half_done + 8 * (q6_count & 1u) : done + 8 * bs);
                            }
                        }
                        ++q6_count;
                    }
                    if (++bs == nb) { bs = 0; b_parity ^= 1u; }
                }
            }
        }
    } else if (warp >= kConvertWarp0) {
        // ---------------- conversion ----------------
        const int quadrant = warp & 3, part = (warp - kConvertWarp0) >> 2;
        bool alive = true;
        int ws = 0, done_slot = 0;
        uint32_t parity = 0, done_parity = 0, a_count = 0, kt = 0, q6_count = 0, half_count = 0;
        uint32_t by_half = 0;   // bit st: the stage's last products were a Q6_K tile's first half
        // wait for the products that last read stage st; the `done` phases come in k tile order
        auto stage_free = [&](uint32_t st) {
            if (a_count < 2) return;
            if ((by_half >> st) & 1u) {
                if (alive) alive = mbar_wait(half_done + 8 * (half_count & 1u), (half_count >> 1) & 1u, a.error_flag, 97, spin_limit);
                ++half_count;
            } else {
                if (alive) alive = mbar_wait(done + 8 * done_slot, done_parity, a.error_flag, 97, spin_limit);
                if (++done_slot == nb) { done_slot = 0; done_parity ^= 1u; }
            }
        };
        for (int s = s0; s < s1;) {
            const int unit = s / k_tiles, end = min(s1, (unit + 1) * k_tiles);
            const int type = type_of<TYPE>(a.seg[unit_at(a, unit, kUnitTiles).seg]);
            for (; s < end; ++s, ++kt) {
                if (alive) alive = mbar_wait(w_full + 8 * ws, parity, a.error_flag, 96, spin_limit);
                const uint32_t tile = w_ring + ws * rings.w_bytes + 2 * quadrant * packed_tile_bytes(type);
                const uint32_t scales = scales_ring + (kt & 3u) * (kUnitRows * 4);
                const int halves = type == kQ4_K ? 1 : 2;
                for (int half = 0; half < halves; ++half, ++a_count) {
                    const uint32_t st = a_count & 1u, a_at = tmem + 256 + 128 * st + ((uint32_t)(32 * quadrant) << 16);
                    stage_free(st);
                    by_half = (by_half & ~(1u << st)) | ((uint32_t)(halves == 2 && half == 0) << st);
                    tc_fence_after();
                    if (type == kQ4_K) {
#pragma unroll 1
                        for (int c = 2 * part; c < 2 * part + 2; ++c) convert_q4k(tile, c, a_at + 32 * c, scales, a2_buf + st * kA2Bytes, 32 * quadrant, lane);
                    } else {
#pragma unroll 1
                        for (int hi = 0; hi < 2; ++hi) {
                            if (TYPE == kKQuants || type == kQ6_K) convert_q6k(tile, half, part + 2 * hi, a_at + 16 * (part + 2 * hi), 64, scales, 32 * quadrant, lane);
                            else convert_q8_0(tile, half, part + 2 * hi, a_at + 16 * (part + 2 * hi), 64, scales, 32 * quadrant, lane);
                        }
                    }
                    tmem_wait_st();
                    tc_fence_before();
                    if (part == 0) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the minima operand
                    __syncwarp();
                    if (lane == 0) mbar_arrive(a_full + 8 * st);
                }
                if (lane == 0) mbar_arrive(w_empty + 8 * ws);
                if (++ws == nw) { ws = 0; parity ^= 1u; }
            }
        }
    } else {
        // ---------------- fold and store: one output row and every other eight columns per thread ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kEpilogueRegs));
        asm volatile("griddepcontrol.wait;" ::: "memory");
        constexpr int kChunks = (MP + 15) / 16;   // eights of columns per thread: 16 j + 8 (warp >> 2)
        const int quadrant = warp & 3, mine = 8 * (warp >> 2), row = quadrant * 32 + lane;
        bool alive = true;
        int bs = 0;
        bool factors = a.partial != nullptr;   // the rows' RMSNorm factors are in place, or another kernel applies them
        uint32_t b_parity = 0, kt = 0;
        float* inv = reinterpret_cast<float*>(smem + (inv_at - w_ring));
        for (int s = s0; s < s1;) {
            const int unit = s / k_tiles;
            const UnitAt at = unit_at(a, unit, kUnitTiles);
            const GemvSegment& seg = a.seg[at.seg];
            const int type = type_of<TYPE>(seg);
            const bool q4k = type == kQ4_K, q6k = TYPE == kKQuants ? !q4k : type == kQ6_K;
            const int end = min(s1, (unit + 1) * k_tiles);
            float acc[kChunks][8];
#pragma unroll
            for (int j = 0; j < kChunks; ++j) {
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[j][i] = 0.0f;
            }
            for (; s < end; ++s, ++kt) {
                const uint32_t p = kt & 1u;
                if (alive) alive = mbar_wait(b_full + 8 * bs, b_parity, a.error_flag, 99, spin_limit);   // for the scales' bytes
                if (alive) alive = mbar_wait(done + 8 * bs, b_parity, a.error_flag, 98, spin_limit);
                tc_fence_after();
                const uint32_t t_main = tmem + 64 * p + ((uint32_t)(quadrant * 32) << 16) + mine, t_min = t_main + 128;
                const float2 dd = __half22float2(as_half2(lds32(scales_ring + (kt & 3u) * (kUnitRows * 4) + row * 4)));
                const float d = dd.x, dmin = dd.y;
                const uint32_t sx_at = b_ring + bs * kBBytes + C::kMain + C::kSums + mine * 4;
                constexpr int kBatch = 2;   // eights of columns in flight together
#pragma unroll
                for (int j0 = 0; j0 < kChunks; j0 += kBatch) {
                    float x[kBatch][8], y[kBatch][8], z[kBatch][8], w[kBatch][8];
#pragma unroll
                    for (int b = 0; b < kBatch; ++b) {
                        const int j = j0 + b;
                        if (16 * j + mine < MP) {
                            tmem_ld8(t_main + 16 * j, x[b]);
                            if (C::kJoined) tmem_ld8(t_main + MP + 16 * j, y[b]);
                            if (q4k || q6k) tmem_ld8(t_min + 16 * j, z[b]);       // minima sums, or the second half's
                            if (C::kJoined && q6k) tmem_ld8(t_min + MP + 16 * j, w[b]);
                        }
                    }
                    tmem_wait_ld();
#pragma unroll
                    for (int b = 0; b < kBatch; ++b) {
                        const int j = j0 + b;
                        if (j >= kChunks || 16 * j + mine >= MP) continue;
                        tmem_tie(x[b]);
                        if (C::kJoined) tmem_tie(y[b]);
                        if (q4k || q6k) tmem_tie(z[b]);
                        if (C::kJoined && q6k) tmem_tie(w[b]);
#pragma unroll
                        for (int i = 0; i < 8; i += 4) {
                            float sx[4];
                            asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(sx[0]), "=f"(sx[1]), "=f"(sx[2]), "=f"(sx[3])
                                         : "r"(sx_at + (16 * j + i) * 4));
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                float v = q6k ? x[b][i + q] + z[b][i + q] : x[b][i + q];
                                if (C::kJoined) v += q6k ? y[b][i + q] + w[b][i + q] : y[b][i + q];
                                v *= d;
                                if (q4k) v = fmaf(-dmin, z[b][i + q], v);
                                acc[j][i + q] = fmaf(sx[q], v, acc[j][i + q]);
                            }
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(folded + 8 * bs);
                if (++bs == nb) { bs = 0; b_parity ^= 1u; }
            }
            if (!factors) {
                factors = true;
                for (int m = warp; m < MP; m += kEpilogueWarps) {
                    float sum = 0.0f;
                    if (a.ss != nullptr && m < a.members) for (int i = lane; i < k_tiles; i += 32) sum += a.ss[(size_t)m * k_tiles + i];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                    if (lane == 0) inv[m] = a.ss != nullptr ? 1.0f / sqrtf(sum / (float)a.k + a.eps) : 1.0f;
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
            }
            const int n_index = at.rt0 * kTileRows + row;
            if (n_index < seg.n) {
                StepSums to{};
                if (a.partial != nullptr) to = step_sums(a, split, (int)blockIdx.x, split.whole ? 0 : (int)blockIdx.x - split.first_worker(unit), 0, mine, at.seg, n_index);
#pragma unroll
                for (int j = 0; j < kChunks; ++j) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int m = 16 * j + mine + i;
                        if (m >= MP || m >= a.members) continue;
                        if (a.partial != nullptr) {
                            to.at[(16 * j + i) * to.stride] = acc[j][i];
                        } else {
                            float* y = seg.y + (size_t)m * seg.n + n_index;
                            *y = a.epilogue == kResidual ? *y + acc[j][i] * inv[m] : acc[j][i] * inv[m];
                        }
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

template <int MP, int TYPE>
cudaError_t launch_variant(cudaStream_t stream, const StepGemm& a, int w_bytes, bool programmatic) {
    static bool configured[kMaxDevices] = {false};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    if (!configured[dev]) {
        e = cudaFuncSetAttribute(gemm_ta_kernel<MP, TYPE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    TaRings rings{};
    rings.w_bytes = (w_bytes + 127) & ~127;
    const size_t b_bytes = (size_t)((Cols<MP>::kBlock + 127) & ~127), fixed = 2 * kA2Bytes + 4 * kUnitRows * 4 + MP * 4 + 16 + 352;
    rings.b_stages = MP <= 32 ? 3 : 2;
    rings.w_stages = (int)std::min<size_t>(8, (kSmemBudget - fixed - rings.b_stages * b_bytes) / rings.w_bytes);
    if (rings.w_stages < 2) return cudaErrorInvalidValue;
    const StepSplit split = step_split(a, a.partial == nullptr);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)split.workers);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = fixed + rings.b_stages * b_bytes + (size_t)rings.w_stages * rings.w_bytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, gemm_ta_kernel<MP, TYPE>, a, split, rings);
}

template <int TYPE>
cudaError_t launch_typed(cudaStream_t stream, const StepGemm& a, int w_bytes, bool programmatic) {
    switch (step_shape(a.members, kColumnForm).ng) {
        case 3: return launch_variant<24, TYPE>(stream, a, w_bytes, programmatic);
        case 4: return launch_variant<32, TYPE>(stream, a, w_bytes, programmatic);
        case 6: return launch_variant<48, TYPE>(stream, a, w_bytes, programmatic);
        default: return launch_variant<64, TYPE>(stream, a, w_bytes, programmatic);
    }
}

}  // namespace

cudaError_t launch_gemm_ta(cudaStream_t stream, const StepGemm& a, int w_bytes, bool programmatic) {
    if (a.members > kColumnMaxMembers) return cudaErrorInvalidValue;
    switch (common_type(a)) {
        case kQ4_K: return launch_typed<kQ4_K>(stream, a, w_bytes, programmatic);
        case kQ6_K: return launch_typed<kQ6_K>(stream, a, w_bytes, programmatic);
        case kQ8_0: return launch_typed<kQ8_0>(stream, a, w_bytes, programmatic);
        case kKQuants: return launch_typed<kKQuants>(stream, a, w_bytes, programmatic);
        default: return launch_typed<kAnyType>(stream, a, w_bytes, programmatic);
    }
}

}  // namespace ribn
