// Attention of a prefill chunk on the tcgen05 tensor cores: consecutive tokens of one sequence against the paged cache.
//
// A CTA serves one kv head and two tiles of 128 query rows (row = token x query head of the group), each with its own
// softmax warps, so that one tile's products run while the other's probabilities are formed.  Per 128 keys and tile:
//   S = Q K^T   A = Q as binary16 hi + lo in shared memory (converted once), B = the K rows as they lie in the cache: two
//               products per element, lo first, F32 sums in tensor memory;
//   P           a thread owns a row: online softmax in base 2, P as binary16 hi + lo written over S in tensor memory (32 keys
//               of S become 16 columns of hi and 16 of lo);
//   O += P V    A = P from tensor memory, B = the V rows (the same core matrices, read with the other major order).
// Q, the probabilities and the sums keep the precision of the span kernels (attention.cu).  A row's reference maximum only
// moves when a tile's maximum passes it by 2^8 in the exponent, which binary16 pairs and F32 sums hold with the same
// relative precision; then the row's sums are rescaled where they lie.  Key tiles begin at multiples of 128, and a row's
// bits depend on its own keys and on its chunk's tokens and prefix (which choose among the kernel's forms), never
// on the other rows of a step.
//
// What bounds it: the products, 2 x (1,024 + 1,024) clocks per 128 keys and CTA, which take about 5,200: those of Q K^T read
// both operands from shared memory, 128 bytes per clock, beside the copies.  A tile's softmax takes 2,400 clocks beside
// the other's products.  8B model, 2,048 tokens without prefix: 90 us a layer as first built (108 with the windows below, cold),
// against 372 us of the mma.sync kernel that attention.cu keeps for other head widths (0.6B model, 777 tokens: 33 against 64 us,
// and no spans for the last 9); behind 14,336 tokens 943 against 5,338 us.  All 128 scores of a row in registers: 93 us against
// 90; the next 32 scores requested under the present ones' arithmetic: 91 us.
// Roles of the 12 warps: 0..3 / 4..7 softmax and output of tile 0 / 1, 8 issues the products, 9..11 copy K / V tiles (keys
// past the chunk's last one are zero, so that a zero probability meets no NaN).  Every wait is bounded.
#include <cuda_fp16.h>
#include <math.h>

#include <algorithm>

#include "kernels.cuh"
#include "step_operand.cuh"
#include "tmem.cuh"

namespace ribn {

namespace {

constexpr int kHd = 128, kRows = 128, kKeys = 128;
constexpr int kPieceBytes = 128 * 16;                 // one 8-dimension column of 128 rows or keys
constexpr int kTileBytes = kHd / 8 * kPieceBytes;     // 128 x 128 binary16: 32 KB
constexpr int kSlots = 3;                             // K / V tiles in shared memory: K0 V0 K1 V1 ..
constexpr int kSoftmaxWarps = 8, kMmaWarp = 8, kLoadWarp0 = 9, kLoadWarps = 3, kThreads = 12 * 32;
constexpr size_t kSmem = 4 * kTileBytes + kSlots * kTileBytes + 128 + kRows * 8;
constexpr uint32_t kSpinLimit = 1u << 22;
constexpr float kLog2e = 1.4426950408889634f;
constexpr size_t kWideBlock = 1028 * 128 + 32 * 128;  // one k tile of 128 rows in the wide operand form
constexpr int kWindow = 4;                            // key tiles whose products one sum in tensor memory holds
constexpr float kSlack = 8.0f;                        // the reference maximum may lag by 2^8
// Register shares: 384 x 168 at launch (64,512); softmax 256 x 208, the others 128 x 88.
constexpr int kSoftmaxRegs = 208, kOtherRegs = 88;

// B = V: rows are keys (the products' K), 16 bytes of a row are eight of its dimensions (N): N-major core matrices
constexpr uint32_t kIdescQk = umma_idesc(kKeys), kIdescPv = umma_idesc(kHd) | (1u << 16);
constexpr uint32_t kDescHighPv = ((uint32_t)kPieceBytes >> 4) | (1u << 14);
__device__ __forceinline__ void umma_pv(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_desc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 b, {%2, %6};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_desc), "r"(kIdescPv), "r"(accumulate), "r"(0u), "r"(kDescHighPv) : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
        "%29,%30,%31}, [%32];"
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]), "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]),
          "=f"(v[12]), "=f"(v[13]), "=f"(v[14]), "=f"(v[15]), "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]), "=f"(v[22]),
          "=f"(v[23]), "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]), "=f"(v[29]), "=f"(v[30]), "=f"(v[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_tie32(float (&v)[32]) {   // the values of a load, after its wait
#pragma unroll
    for (int i = 0; i < 32; i += 8) {
        asm volatile("" : "+f"(v[i]), "+f"(v[i + 1]), "+f"(v[i + 2]), "+f"(v[i + 3]), "+f"(v[i + 4]), "+f"(v[i + 5]), "+f"(v[i + 6]), "+f"(v[i + 7]) :: "memory");
    }
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
                 "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ float exp2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// x0, x1 = hi + lo as binary16 pairs
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(x0, x1);
    const float2 back = __half22float2(h), rest = __fadd2_rn(make_float2(x0, x1), make_float2(-back.x, -back.y));
    hi = as_bits(h);
    lo = as_bits(__floats2half2_rn(rest.x, rest.y));
}
// keys past the row's last one
__device__ __forceinline__ void mask_keys(float (&s)[32], int see) {
#pragma unroll
    for (int i = 0; i < 32; ++i) s[i] = i <= see ? s[i] : -INFINITY;
}
__device__ __forceinline__ void sts128(uint32_t addr, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// The wide operand form of a warp's 32 result rows (32 / heads tokens from `token0` on), which lie in `stage` as 512 bytes each,
// 16-byte pieces in the order of their number ^ (row % 8): the values and bits of write_step_operand (step_operand.cuh), eight
// tokens of a pair of heads (one k tile) at a time.  Rows past the last token keep what they held: only their own columns of the
// products see them, and nothing stores those.  A lane holds eight neighbouring inputs of each; its halves go back to where the
// 16 rows lay, so that the stores are the eight tokens' 16-byte pieces side by side.
// In place of F32 results and a launch that reads them: 2,048 tokens of the 8B model (4 layers) 7.15 -> 7.10 ms, 777 of the 0.6B
// model 4.96 -> 4.87 ms.
__device__ __forceinline__ void write_wide_operand(const StepOperand& out, uint32_t stage, int k_tiles, int kt0, int heads, int token0, int token_end, int lane) {
#pragma unroll 1
    for (int it = 0; it < 2; ++it) {   // 2 heads: eight and eight tokens; 4 heads: one pair and the other
        const int first = heads == 2 ? 8 * it : 0, pair = heads == 2 ? 0 : it;
        const auto row_of = [&](int r) { return (first + (r >> 1)) * heads + 2 * pair + (r & 1); };   // r: 2 x token + head
        const int kt = kt0 + pair;
        float v[8][8];
#pragma unroll
        for (int tk = 0; tk < 8; ++tk) {
            const int r = row_of(2 * tk + (lane >> 4)), c = (lane & 15) * 2;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4 x = lds128(stage + r * 512 + (((c + h) ^ (r & 7)) << 4));
                v[tk][4 * h] = __uint_as_float(x.x); v[tk][4 * h + 1] = __uint_as_float(x.y);
                v[tk][4 * h + 2] = __uint_as_float(x.z); v[tk][4 * h + 3] = __uint_as_float(x.w);
            }
        }
        __syncwarp();   // all read; the halves take the same 16 rows
        const uint32_t row_at = stage + row_of(lane >> 1) * 512 + (lane & 1) * 8;
        const int swap = (lane >> 1) & 7;
#pragma unroll
        for (int tk = 0; tk < 8; ++tk) {
            float top = 0.0f;
#pragma unroll
            for (int u = 0; u < 8; ++u) top = fmaxf(top, fabsf(v[tk][u]));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const int biased = (int)(__float_as_uint(top) >> 23), e = biased == 255 ? 10 : max(-126, min(126, 136 - biased));
            const float scale = power2(e);
            uint32_t word[2][4];   // [inputs 0..3, 4..7][hi of 0, 2; lo of 0, 2; hi of 1, 3; lo of 1, 3]
            float part[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float* x = &v[tk][4 * h];
                const __half2 h02 = __floats2half2_rn(x[0] * scale, x[2] * scale), h13 = __floats2half2_rn(x[1] * scale, x[3] * scale);
                const float2 b02 = __half22float2(h02), b13 = __half22float2(h13);
                const __half2 l02 = __floats2half2_rn(x[0] * scale - b02.x, x[2] * scale - b02.y), l13 = __floats2half2_rn(x[1] * scale - b13.x, x[3] * scale - b13.y);
                const float2 r02 = __half22float2(l02), r13 = __half22float2(l13);
                part[h] = (((b02.x + r02.x) + (b13.x + r13.x)) + (b02.y + r02.y)) + (b13.y + r13.y);
                word[h][0] = as_bits(h02); word[h][1] = as_bits(l02); word[h][2] = as_bits(h13); word[h][3] = as_bits(l13);
            }
            float sum = part[0] + part[1];
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
#pragma unroll
            for (int p = 0; p < 4; ++p) {   // the piece of (8-input block, hi or lo, token): number 8 p + token of its row
                asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(row_at + (((8 * p + tk) ^ swap) << 4)), "r"(word[0][p]), "r"(word[1][p]) : "memory");
            }
            const int member = token0 + first + tk, col = member & 127;
            if (member < token_end) {
                unsigned char* sums = out.blocks + ((size_t)(member >> 7) * k_tiles + kt) * kWideBlock + 1024 * 128;
                if ((lane & 3) == 0) {
                    const __half hi = __float2half_rn(sum), lo = __float2half_rn(sum - __half2float(hi));
                    __half* to = reinterpret_cast<__half*>(sums + ((col >> 6) * 128 + (col & 63)) * 16) + (lane >> 2);
                    to[0] = hi;
                    to[8 * 64] = lo;
                }
                if (lane == 0) reinterpret_cast<float*>(sums + 32 * 128)[col] = power2(-e);
            }
        }
        __syncwarp();
        const int member = token0 + first + (lane & 7), col = member & 127;
        unsigned char* block = out.blocks + ((size_t)(member >> 7) * k_tiles + kt) * kWideBlock;
#pragma unroll
        for (int n = 0; n < 16; ++n) {
            const uint4 x = lds128(stage + row_of(n) * 512 + ((lane ^ (n & 7)) << 4));
            const int kb = 2 * n + (lane >> 4), half = (lane >> 3) & 1;
            if (member < token_end) *reinterpret_cast<uint4*>(block + (size_t)((((col >> 6) * 2 + (kb >> 4)) * 2 + half) * 1024 + (kb & 15) * 64 + (col & 63)) * 16) = x;
        }
    }
}

// kPairs: two query tiles per CTA.  kWindows: the same for more keys than a window, whose sum in tensor memory is added to the
// rows' sums in the softmax warps' registers at each window's end.  An addition in tensor memory cuts at the sum's last bit:
// with one sum over all keys a result was 3.4e-5 from the exact one at 8,838 keys and 6.4e-5 at 16,384 (the mma.sync kernel:
// 2.6e-5 and 5.0e-5), with windows of 512 keys 1.8e-6 at either.  2,048 tokens of the 8B model (4 layers): 102 to 107 us a layer
// without, 108 with windows (of 1,024 keys: 108), a step of 6.94 and 6.97 ms; behind 14,336 tokens 11.6 and 11.6 ms.  In short
// chunks its longer code cost 2 % of a step: they take kPairs.
// kShared (SPLIT): one query tile per CTA, whose even key tiles are the first four softmax warps' and odd ones the others'; their
// two results meet at the end.  For launches that would leave half of the SMs without a pair of tiles.  (1.6e-5 at 8,262 keys:
// half as many additions per sum.)
enum Form : int { kPairs, kWindows, kShared };
template <int FORM>
__global__ void __launch_bounds__(kThreads, 1) attention_tc_kernel(const PrefillAttention a, const int tile_tokens) {
    constexpr bool SPLIT = FORM == kShared, WINDOWS = FORM == kWindows;
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t q_at = smem_u32(smem), ring = q_at + 4 * kTileBytes, bars = ring + kSlots * kTileBytes;
    const uint32_t q_full = bars, s_full = bars + 16, p_full = bars + 32, o_full = bars + 48, kv_full = bars + 64, kv_empty = bars + 88, tmem_slot = bars + 112, drained = bars + 120;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(q_full + 8 * i, kSoftmaxWarps / 2); mbar_init(s_full + 8 * i, 1); mbar_init(p_full + 8 * i, kSoftmaxWarps / 2); mbar_init(o_full + 8 * i, 1);
        }
        for (int i = 0; i < kSlots; ++i) { mbar_init(kv_full + 8 * i, kLoadWarps); mbar_init(kv_empty + 8 * i, 1); }
        mbar_init(drained, 1);
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
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // the tiles with the most keys first
    const int q_per_kv = a.q_heads / a.kv_heads, places = (int)gridDim.x / a.kv_heads;
    const int place = places - 1 - (int)blockIdx.x / a.kv_heads, kvh = (int)blockIdx.x % a.kv_heads;
    const int pos0 = a.token_pos[a.first];
    int local[2], tokens[2], n[2];   // a tile's first token inside the chunk, its tokens, its key tiles
    for (int t = 0; t < 2; ++t) {
        local[t] = (SPLIT ? place : 2 * place + t) * tile_tokens;
        tokens[t] = max(0, min(tile_tokens, a.count - local[t]));
        n[t] = tokens[t] > 0 ? (pos0 + local[t] + tokens[t] - 1) / kKeys + 1 : 0;
        if (SPLIT) n[t] = (n[t] + 1 - t) / 2;
    }
    const int n_tiles = max(n[0], n[1]), all_tiles = SPLIT ? n[0] + n[1] : n_tiles, total_copies = 2 * all_tiles;
    bool alive = true;

    if (warp >= kMmaWarp) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
        if (warp == kMmaWarp) {
            // ---------------- products (the warp as a whole, one elected lane in it) ----------------
            const bool leader = elect_one();
            const uint32_t q_desc = umma_desc(q_at, kPieceBytes), k_desc = umma_desc(ring, kPieceBytes), v_desc = umma_desc(ring, 128);
            auto slot_wait = [&](int idx) {
                if (alive) alive = mbar_wait(kv_full + 8 * (idx % kSlots), (uint32_t)(idx / kSlots) & 1u, a.error_flag, 121, kSpinLimit);
            };
            // S of query tile t against the K tile that is copy `idx`
            auto scores = [&](int t, int idx) {
                slot_wait(idx);
                tc_fence_after();
                const uint32_t b = k_desc + (idx % kSlots) * (kTileBytes >> 4), hi = q_desc + (SPLIT ? 0 : 2 * t) * (kTileBytes >> 4), lo = hi + (kTileBytes >> 4);
                if (leader && alive) {
#pragma unroll
                    for (int i = 0; i < kHd / 16; ++i) umma_ss(tmem + 128 * t, lo + i * (2 * kPieceBytes >> 4), b + i * (2 * kPieceBytes >> 4), kIdescQk, (uint32_t)(i != 0));
#pragma unroll
                    for (int i = 0; i < kHd / 16; ++i) umma_ss(tmem + 128 * t, hi + i * (2 * kPieceBytes >> 4), b + i * (2 * kPieceBytes >> 4), kIdescQk, 1u);
                }
                if (leader) umma_commit(s_full + 8 * t);
            };
            // O of tile t += P of its j-th key tile times the V tile that is copy `idx`
            auto values = [&](int t, int j, int idx) {
                if (alive) alive = mbar_wait(p_full + 8 * t, (uint32_t)j & 1u, a.error_flag, 123, kSpinLimit);
                slot_wait(idx);
                tc_fence_after();
                if (leader && alive) {
                    const uint32_t goes_on = WINDOWS ? j % kWindow != 0 : j != 0, p_at = tmem + 128 * t, o_at = tmem + 256 + 128 * t, b = v_desc + (idx % kSlots) * (kTileBytes >> 4);
#pragma unroll
                    for (int i = 0; i < kKeys / 16; ++i) umma_pv(o_at, p_at + 32 * (i >> 1) + 8 * (i & 1) + 16, b + i * (256 >> 4), goes_on | (uint32_t)(i != 0));
#pragma unroll
                    for (int i = 0; i < kKeys / 16; ++i) umma_pv(o_at, p_at + 32 * (i >> 1) + 8 * (i & 1), b + i * (256 >> 4), 1u);
                }
                if (leader && j + 1 == n[t]) umma_commit(o_full + 8 * t);
            };
            // (the last copies' slots are not asked for again: an arrival there could come after the block's end)
            auto release = [&](int idx) { if (leader && idx + kSlots < total_copies) umma_commit(kv_empty + 8 * (idx % kSlots)); };
            if (SPLIT) {
                int idx = 0;   // copies in the order of their use, each used once
                if (alive) alive = mbar_wait(q_full, 0, a.error_flag, 122, kSpinLimit);
                for (int t = 0; t < 2; ++t) if (n[t] > 0) { scores(t, idx); release(idx++); }
                for (int j = 0; j < n_tiles; ++j) {
#pragma unroll 1
                    for (int t = 0; t < 2; ++t) {
                        if (j < n[t]) { values(t, j, idx); release(idx++); }
                        if (j + 1 < n[t]) { scores(t, idx); release(idx++); }
                    }
                }
            } else {
                for (int t = 0; t < 2; ++t) {
                    if (n[t] == 0) continue;
                    if (alive) alive = mbar_wait(q_full + 8 * t, 0, a.error_flag, 122, kSpinLimit);
                    scores(t, 0);
                }
                release(0);
                for (int j = 0; j < n_tiles; ++j) {
#pragma unroll 1
                    for (int t = 0; t < 2; ++t) {
                        if (j < n[t]) values(t, j, 2 * j + 1);
                        if (t == 1) release(2 * j + 1);
                        if (j + 1 < n[t]) scores(t, 2 * j + 2);   // over the probabilities that the products above have read
                        if (t == 1 && j + 1 < n_tiles) release(2 * j + 2);
                    }
                }
            }
            if (!alive) {
                // let what was issued come to its end before the block, and its tensor memory, can: a commit follows all products before it
                if (leader) umma_commit(drained);
                mbar_wait(drained, 0, nullptr, 0, kSpinLimit);
            }
        } else {
            // ---------------- K / V tiles: lane = (key of a group of eight, 16-byte piece of four) ----------------
            const int lw = warp - kLoadWarp0, sub = lane >> 2, last = pos0 + local[0] + tokens[0] + (SPLIT ? 0 : tokens[1]) - 1;
            const int32_t* table = a.page_tables + (long long)(a.token_seq != nullptr ? a.token_seq[a.first] : 0) * a.pages_per_sequence;
            const long long stride = (long long)a.kv_heads * kHd;
            constexpr int kGroups = (kKeys / 8 + kLoadWarps - 1) / kLoadWarps;
            // Copy `idx`: K0 V0 K1 V1 .., or (SPLIT) K0 K1, then V j, K j + 2 in turn: 2 (j + 1) and 2 (j + 1) + 1, what does not exist left out
            const int total = total_copies;
            auto what = [&](int idx, bool& v) -> int {   // its key tile
                if (!SPLIT) { v = idx & 1; return idx >> 1; }
                if (idx < 2 || all_tiles == 1) { v = all_tiles == 1 ? idx == 1 : false; return all_tiles == 1 ? 0 : idx; }
                const int place = idx - 2;   // V0 K2 V1 K3 .. V(n-3) K(n-1) V(n-2) V(n-1)
                if (place < 2 * (all_tiles - 2)) { v = (place & 1) == 0; return (place >> 1) + (v ? 0 : 2); }
                v = true;
                return place - (all_tiles - 2);
            };
            long long rows[kGroups];   // cache rows of this lane's keys of the next copy
            auto look_up = [&](int idx) {
                bool v;
                const int j = what(idx, v);
#pragma unroll
                for (int i = 0; i < kGroups; ++i) {
                    const int key = j * kKeys + (lw + i * kLoadWarps) * 8 + sub;
                    rows[i] = lw + i * kLoadWarps < kKeys / 8 && key <= last ? (long long)table[key / kPageTokens] * kPageTokens + key % kPageTokens : -1;
                }
            };
            auto copy = [&](int idx) {
                bool v;
                what(idx, v);
                const __half* from = (v ? a.cache_v : a.cache_k) + (long long)kvh * kHd + (lane & 3) * 8;
                const uint32_t to = ring + (idx % kSlots) * kTileBytes + (lane & 3) * kPieceBytes + (lw * 8 + sub) * 16;
#pragma unroll
                for (int i = 0; i < kGroups; ++i) {
                    if (lw + i * kLoadWarps >= kKeys / 8) break;
                    const __half* src = from + (rows[i] < 0 ? 0 : rows[i] * stride);
                    const uint32_t bytes = rows[i] < 0 ? 0u : 16u;   // nothing read, zeros written
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + i * (kLoadWarps * 128) + p * (4 * kPieceBytes)), "l"(src + p * 32), "r"(bytes) : "memory");
                    }
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (idx + 1 < total) look_up(idx + 1);   // under the copies
            };
            auto landed = [&](int idx) {
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(kv_full + 8 * (idx % kSlots));
            };
            look_up(0);   // `total` is even, at least 2
            copy(0);
            copy(1);
            if (total > 2) copy(2); else asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 2;" ::: "memory");
            landed(0);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            landed(1);
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            if (total > 2) landed(2);
            for (int idx = 3; idx < total; ++idx) {
                if (alive) alive = mbar_wait(kv_empty + 8 * (idx % kSlots), (uint32_t)(idx / kSlots - 1) & 1u, a.error_flag, 124, kSpinLimit);
                copy(idx);
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                landed(idx);
            }
        }
    } else {
        // ---------------- softmax: one row per thread ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kSoftmaxRegs));
        const int t = warp >> 2, quadrant = warp & 3, row0 = quadrant * 32, row = row0 + lane;
        const uint32_t q_tile = q_at + 2 * t * kTileBytes;
        const int live_rows = tokens[t] * q_per_kv;
        int live = live_rows;   // rows that these warps store
        if (n[t] > 0) {
            if (!SPLIT || t == 0) {
                // the warp's 32 query rows as hi + lo: lane = (row of eight, 8-dimension piece of four)
                const int sub = lane & 7, pc = lane >> 3;
                float4 x[4][4][2];   // everything in flight together
#pragma unroll
                for (int rg = 0; rg < 4; ++rg) {
                    const int r = row0 + rg * 8 + sub;
                    const bool have = r < live_rows;
                    const float* from = a.q + ((long long)(a.first + local[t] + (have ? r / q_per_kv : 0)) * a.q_heads + kvh * q_per_kv + (have ? r % q_per_kv : 0)) * kHd + pc * 8;
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) x[rg][p][h] = have ? *reinterpret_cast<const float4*>(from + p * 32 + 4 * h) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    }
                }
#pragma unroll
                for (int rg = 0; rg < 4; ++rg) {
#pragma unroll
                    for (int p = 0; p < 4; ++p) {
                        const float4 x0 = x[rg][p][0], x1 = x[rg][p][1];
                        uint4 hi, lo;
                        split2(x0.x, x0.y, hi.x, lo.x); split2(x0.z, x0.w, hi.y, lo.y);
                        split2(x1.x, x1.y, hi.z, lo.z); split2(x1.z, x1.w, hi.w, lo.w);
                        const uint32_t to = q_tile + (p * 4 + pc) * kPieceBytes + (row0 + rg * 8 + sub) * 16;
                        sts128(to, hi);
                        sts128(to + kTileBytes, lo);
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(q_full + 8 * t);
            }
            const float c = kLog2e / sqrtf((float)kHd);
            const int limit = row < live_rows ? pos0 + local[t] + row / q_per_kv : -1;   // the row's last key
            const int warp_limit = row0 + 31 < live_rows ? pos0 + local[t] + row0 / q_per_kv : -1;   // keys that every row of the warp sees
            const uint32_t lanes = (uint32_t)row0 << 16, s_at = tmem + lanes + 128 * t, o_at = s_at + 256;
            float m = -INFINITY;
            float2 l = make_float2(0.0f, 0.0f);
            float sum[WINDOWS ? kHd : 1], since = 1.0f;   // earlier windows' results; the factor that has come to them since the last one's end
#pragma unroll
            for (int i = 0; i < (WINDOWS ? kHd : 1); ++i) sum[i] = 0.0f;
            for (int j = 0; j < n[t]; ++j) {
                if (alive) alive = mbar_wait(s_full + 8 * t, (uint32_t)j & 1u, a.error_flag, 125, kSpinLimit);
                tc_fence_after();
                const int key0 = (SPLIT ? 2 * j + t : j) * kKeys, see = limit - key0;
                const bool masked = key0 + kKeys - 1 > warp_limit;
                const bool fresh = WINDOWS ? j % kWindow == 0 : j == 0;
                if (WINDOWS && fresh && j > 0) {   // (the scores' barrier also says that the products into O so far are complete)
#pragma unroll
                    for (int i = 0; i < kHd; i += 32) {
                        float o[32];
                        tmem_ld32(o_at + i, o);
                        tmem_wait_ld();
                        tmem_tie32(o);
#pragma unroll
                        for (int u = 0; u < 32; ++u) sum[WINDOWS ? i + u : 0] = fmaf(sum[WINDOWS ? i + u : 0], since, o[u]);
                    }
                    since = 1.0f;
                }
                // 32 scores at a time, twice (a read of tensor memory costs less than 128 registers): the maximum, then P
                float mx = -INFINITY;
#pragma unroll 1
                for (int i = 0; i < kKeys; i += 32) {
                    float s[32];
                    tmem_ld32(s_at + i, s);
                    tmem_wait_ld();
                    tmem_tie32(s);
                    if (masked) mask_keys(s, see - i);
                    float top[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
                    for (int u = 4; u < 28; u += 8) {
#pragma unroll
                        for (int w = 0; w < 4; ++w) top[w] = fmaxf(top[w], fmaxf(s[u + w], s[u + 4 + w]));
                    }
#pragma unroll
                    for (int w = 0; w < 4; ++w) top[w] = fmaxf(top[w], s[28 + w]);
                    mx = fmaxf(mx, fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])));
                }
                const bool moves = mx > m && (m == -INFINITY || (mx - m) * c > kSlack);
                if (__any_sync(0xffffffffu, moves)) {
                    const float f = moves ? (m == -INFINITY ? 0.0f : exp2_approx((m - mx) * c)) : 1.0f;
                    if (moves) m = mx;
                    l.x *= f; l.y *= f;
                    if (WINDOWS) since *= f;
                    if (!fresh) {
#pragma unroll 1
                        for (int i = 0; i < kHd; i += 16) {
                            float o[2][8];
                            tmem_ld8(o_at + i, o[0]);
                            tmem_ld8(o_at + i + 8, o[1]);
                            tmem_wait_ld();
                            tmem_tie(o[0]);
                            tmem_tie(o[1]);
                            uint32_t r[16];
#pragma unroll
                            for (int u = 0; u < 16; ++u) r[u] = __float_as_uint(o[u >> 3][u & 7] * f);
                            tmem_st16(o_at + i, r);
                        }
                    }
                }
                const float mc = m == -INFINITY ? 0.0f : m * c;
#pragma unroll 1
                for (int i = 0; i < kKeys; i += 32) {
                    float s[32];
                    tmem_ld32(s_at + i, s);
                    tmem_wait_ld();
                    tmem_tie32(s);
                    if (masked) mask_keys(s, see - i);
                    uint32_t hi[16], lo[16];
#pragma unroll
                    for (int u = 0; u < 16; ++u) {
                        const float2 x = __ffma2_rn(make_float2(s[2 * u], s[2 * u + 1]), make_float2(c, c), make_float2(-mc, -mc));
                        const float2 p = make_float2(exp2_approx(x.x), exp2_approx(x.y));
                        l = __fadd2_rn(l, p);
                        split2(p.x, p.y, hi[u], lo[u]);
                    }
                    tmem_st16(s_at + i, hi);   // over the 32 scores just read
                    tmem_st16(s_at + i + 16, lo);
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full + 8 * t);
            }
            if (alive) alive = mbar_wait(o_full + 8 * t, 0, a.error_flag, 126, kSpinLimit);
            tc_fence_after();
            // rows to memory as whole lines, through the shared memory that the queries have left (a warp's own 16 KB); SPLIT: the odd
            // tiles' sums, maximum and l come through the second tile's
            float total = l.x + l.y, f0 = 1.0f, f1 = 0.0f;
            const uint32_t stage = q_tile + row0 * (kHd * 4), other = q_at + 2 * kTileBytes + row0 * (kHd * 4), last_words = bars + 128 + row * 8;
            if (SPLIT && n[1] > 0) {
                if (t == 1) {
#pragma unroll 1
                    for (int i = 0; i < kHd; i += 32) {
                        float o[32];
                        tmem_ld32(o_at + i, o);
                        tmem_wait_ld();
                        tmem_tie32(o);
#pragma unroll
                        for (int u = 0; u < 32; u += 4) {
                            sts128(other + lane * (kHd * 4) + ((((i + u) >> 2) ^ (lane & 7)) << 4),
                                   make_uint4(__float_as_uint(o[u]), __float_as_uint(o[u + 1]), __float_as_uint(o[u + 2]), __float_as_uint(o[u + 3])));
                        }
                    }
                    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(last_words), "f"(m), "f"(total) : "memory");
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (t == 0) {
                    float m1, l1;
                    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(m1), "=f"(l1) : "r"(last_words) : "memory");
                    const float top = fmaxf(m, m1);
                    f0 = exp2_approx((m - top) * c);
                    f1 = exp2_approx((m1 - top) * c);   // 0 where the row sees no odd tile's key
                    total = total * f0 + l1 * f1;
                }
            }
            if (SPLIT && t == 1) live = 0;
            const float inv = 1.0f / total;
            auto over = [&](float o) { return quotient(o, total, inv); };
            if (!SPLIT || t == 0) {
#pragma unroll (WINDOWS ? kHd / 32 : 1)
                for (int i = 0; i < kHd; i += 32) {
                    float o[32];
                    tmem_ld32(o_at + i, o);
                    tmem_wait_ld();
                    tmem_tie32(o);
                    if (WINDOWS) {
#pragma unroll
                        for (int u = 0; u < 32; ++u) o[u] = fmaf(sum[WINDOWS ? i + u : 0], since, o[u]);
                    }
                    if (SPLIT && n[1] > 0) {
#pragma unroll
                        for (int u = 0; u < 32; u += 4) {
                            const uint4 v = lds128(other + lane * (kHd * 4) + ((((i + u) >> 2) ^ (lane & 7)) << 4));
                            o[u] = fmaf(__uint_as_float(v.x), f1, o[u] * f0); o[u + 1] = fmaf(__uint_as_float(v.y), f1, o[u + 1] * f0);
                            o[u + 2] = fmaf(__uint_as_float(v.z), f1, o[u + 2] * f0); o[u + 3] = fmaf(__uint_as_float(v.w), f1, o[u + 3] * f0);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 32; u += 4) {
                        sts128(stage + lane * (kHd * 4) + ((((i + u) >> 2) ^ (lane & 7)) << 4),
                               make_uint4(__float_as_uint(over(o[u])), __float_as_uint(over(o[u + 1])), __float_as_uint(over(o[u + 2])), __float_as_uint(over(o[u + 3]))));
                    }
                }
            }
            __syncwarp();
            if (a.operand.blocks != nullptr) {
                if (live > 0) write_wide_operand(a.operand, stage, a.q_heads / 2, kvh * q_per_kv / 2, q_per_kv, local[t] + row0 / q_per_kv, local[t] + tokens[t], lane);
                live = 0;
            }
#pragma unroll 4
            for (int r = 0; r < 32; ++r) {
                if (row0 + r >= live) break;
                const uint4 v = lds128(stage + r * (kHd * 4) + ((lane ^ (r & 7)) << 4));
                const int rr = row0 + r;
                float* to = a.out + ((long long)(a.first + local[t] + rr / q_per_kv) * a.q_heads + kvh * q_per_kv + rr % q_per_kv) * kHd;
                *reinterpret_cast<uint4*>(to + lane * 4) = v;
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

}  // namespace

cudaError_t launch_attention_tc(cudaStream_t stream, const PrefillAttention& a) {
    if (a.count <= 0 || a.q_heads % a.kv_heads != 0 || a.q_heads / a.kv_heads > 16) return cudaErrorInvalidValue;
    static bool configured[kMaxDevices] = {false};   // function attributes are per device
    static int sms[kMaxDevices] = {0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    if (!configured[dev]) {
        e = cudaFuncSetAttribute(attention_tc_kernel<kPairs>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(attention_tc_kernel<kWindows>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(attention_tc_kernel<kShared>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    const int tile_tokens = kRows / (a.q_heads / a.kv_heads), tiles = (a.count + tile_tokens - 1) / tile_tokens;
    // While every query tile can have an SM of its own, half of its key tiles per softmax group take half as long: 777 tokens of
    // the 0.6B model (7 key tiles) 37 -> 33 us a layer; with one or two key tiles there is nothing to share (65 tokens: 2 % of
    // the step slower).
    const bool split = tiles * a.kv_heads <= sms[dev] && a.keys > 2 * kKeys;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((split ? tiles : (tiles + 1) / 2) * a.kv_heads));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];   // barriers and tensor memory are set up under the kernel before
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, split ? attention_tc_kernel<kShared> : a.keys > kWindow * kKeys ? attention_tc_kernel<kWindows> : attention_tc_kernel<kPairs>,
                              a, tile_tokens);
}

}  // namespace ribn
