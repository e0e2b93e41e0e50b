// Dequant-GEMM over Q4_K / Q6_K weights with the converted weights in TENSOR MEMORY (tcgen05, A operand in TMEM).
//
//   y[m][n] = sum_k deq(W[n][k]) x[m][k]
//
// The tensor core multiplies the blocks' exact integers, as binary16, by the activations' binary16 hi + lo pairs:
// sc q (at most 945) for Q4_K, sc (q - 32) (up to 4096 in magnitude, as p1 = its value rounded to binary16 and the exact
// rest p2) for Q6_K.  Per 256 inputs the F32 sums leave tensor memory and are folded into F32 registers with the row's
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
// Tensor memory: main sums of k tile parity p at columns 64 p, minima sums at 128 + 64 p, A stages at 256 + 128 s (256
// inputs of Q4_K's one plane, 128 inputs of Q6_K's two).  Slots (unit, row group, k tile) are dealt to the CTAs evenly
// when another kernel finishes the sums, in whole items otherwise (StepSplit).  Every wait is bounded.
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "blocks.cuh"
#include "gemv.cuh"

namespace ribn {

namespace {

constexpr int kUnitTiles = 8;
constexpr int kRows = kUnitTiles * kTileRows;
constexpr int kEpilogueWarps = 8, kConvertWarp0 = 8, kConvertWarps = 8, kWeightWarp = 16, kMmaWarp = 17, kBlockWarp = 18;
constexpr int kThreads = 20 * 32;
// Register shares: the launch gives each thread 96 (61,440 in all); conversion 256 x 96, fold 256 x 112, the rest 128 x 64.
constexpr int kEpilogueRegs = 112, kOtherRegs = 64;
constexpr int kA2Bytes = kRows * 16 * 2;        // minima operand: 128 rows x (8 minima, twice) halves
constexpr int kA2Lbo = kRows / 8 * 128;         // bytes between its two 8-input column blocks
constexpr uint32_t kSpinLimit = 1u << 22;
constexpr size_t kSmemBudget = 224 * 1024;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* error_flag, int code, uint32_t limit) {
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
        if (ok) return true;
    }
    if (error_flag != nullptr) atomicExch(error_flag, code);
    return false;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void tiles_g2s(uint32_t dst, const void* map, int k_tile, int row_tile, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %2, %3, %4}], [%5];" ::"r"(dst),
                 "l"(map), "r"(0), "r"(k_tile), "r"(row_tile), "r"(bar) : "memory");
}
__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
    uint32_t v;
    asm volatile("{\n\t.reg .u16 t;\n\tld.shared.u16 t, [%1];\n\tcvt.u32.u16 %0, t;\n\t}" : "=r"(v) : "r"(addr));
    return v;
}
// (a & mask) | other in one LOP3
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t mask, uint32_t other) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(mask), "r"(other));
    return r;
}
__device__ __forceinline__ __half2 as_half2(uint32_t x) { return *reinterpret_cast<const __half2*>(&x); }
__device__ __forceinline__ uint32_t as_bits(__half2 x) { return *reinterpret_cast<const uint32_t*>(&x); }

// ---- tcgen05 ---------------------------------------------------------------------------------
// Shared-memory operand descriptor, K-major, no swizzle (8 rows x 16 bytes core matrices; see gemm_tc.cu).
__device__ __forceinline__ uint64_t umma_desc(uint32_t smem_addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// kind::f16: F32 accumulate, F16 x F16, M = 128
__host__ __device__ constexpr uint32_t umma_idesc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24); }
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 16 rows x 32 columns: register 2 i + h is row lane / 4 + 8 h, column 4 i + lane % 4
__device__ __forceinline__ void tmem_st_x8(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
        "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
        "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void tmem_st_x4(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.16x128b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]) : "r"(taddr));
}
// Waits for the thread's loads; the values are tied to the wait, so that nothing uses them before it.
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_tie(float (&x)[8]) {
    asm volatile("" : "+f"(x[0]), "+f"(x[1]), "+f"(x[2]), "+f"(x[3]), "+f"(x[4]), "+f"(x[5]), "+f"(x[6]), "+f"(x[7]) :: "memory");
}

struct UnitAt { int seg, rt0; };
__device__ __forceinline__ UnitAt unit_at(const StepGemm& a, int u) {
    UnitAt r{0, u * kUnitTiles};
    while (r.seg + 1 < a.n_segments) {
        const int tiles = (a.seg[r.seg].row_tiles + kUnitTiles - 1) / kUnitTiles * kUnitTiles;
        if (r.rt0 < tiles) break;
        r.rt0 -= tiles;
        ++r.seg;
    }
    return r;
}

// ---- conversion ------------------------------------------------------------------------------------------------
// Rows g and g + 8 of two row tiles (`tile`, `tile` + tile bytes) of one 64-input chunk c of Q4_K: A = sc q, exact.
// Chunk 0 also leaves the rows' (d, dmin) and the minima operand.
__device__ __forceinline__ void convert_q4k(uint32_t tile, int c, uint32_t a_tmem, uint32_t scales, uint32_t a2, int row0, int lane) {
    const int g = lane >> 2, t = lane & 3;
    const uint32_t sel_e = (c & 1) ? 0x4242u : 0x4040u, sel_o = (c & 1) ? 0x4343u : 0x4141u;   // scale bytes of groups 2c, 2c + 1
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint32_t at = tile + r * 2304;
        const uint4 w = lds128(at + c * 512 + lane * 16);
        uint32_t out[16];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint4 hd = lds128(at + 2048 + (g + 8 * h) * 16);
            const uint32_t s4 = c < 2 ? (hd.y & 0x3F3F3F3Fu) : and_or(hd.w, 0x0F0F0F0Fu, (hd.y >> 2) & 0x30303030u);
            if (c == 0) {
                const int row = row0 + r * 16 + g + 8 * h;
                if (t == 0) {
                    const float2 d = __half22float2(as_half2(hd.x));
                    asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(scales + row * 8), "f"(d.x), "f"(d.y) : "memory");
                }
                // minima of groups 2t, 2t + 1, once for the hi sums and once for the lo sums
                const uint32_t m_lo = hd.z & 0x3F3F3F3Fu, m_hi = and_or(hd.w >> 4, 0x0F0F0F0Fu, (hd.z >> 2) & 0x30303030u);
                const uint32_t mm = as_bits(__hsub2(as_half2(__byte_perm(t < 2 ? m_lo : m_hi, 0x64646464u, (t & 1) ? 0x4342u : 0x4140u)), __float2half2_rn(1024.0f)));
                const uint32_t to = a2 + (row >> 3) * 128 + (row & 7) * 16 + 4 * t;
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(to), "r"(mm) : "memory");
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(to + kA2Lbo), "r"(mm) : "memory");
            }
            const __half2 se = __hsub2(as_half2(__byte_perm(s4, 0x64646464u, sel_e)), __float2half2_rn(1024.0f));
            const __half2 so = __hfma2(as_half2(__byte_perm(s4, 0x64646464u, sel_o)), __float2half2_rn(0.0625f), __float2half2_rn(-64.0f));
            const __half2 k1024 = __float2half2_rn(-1024.0f), be = __hmul2(se, k1024), bo = __hmul2(so, k1024);
#pragma unroll
            for (int part = 0; part < 2; ++part) {
                const uint32_t word = h == 0 ? (part == 0 ? w.x : w.y) : (part == 0 ? w.z : w.w), up = word >> 8;
                // step 2 odd + part, pairs (b0, b2) and (b1, b3); 1024 + q, or 1024 + 16 q with sc / 16
                out[(2 * part + 0) * 2 + h] = as_bits(__hfma2(as_half2(and_or(word, 0x000F000Fu, 0x64006400u)), se, be));
                out[(2 * part + 1) * 2 + h] = as_bits(__hfma2(as_half2(and_or(up, 0x000F000Fu, 0x64006400u)), se, be));
                out[(4 + 2 * part + 0) * 2 + h] = as_bits(__hfma2(as_half2(and_or(word, 0x00F000F0u, 0x64006400u)), so, bo));
                out[(4 + 2 * part + 1) * 2 + h] = as_bits(__hfma2(as_half2(and_or(up, 0x00F000F0u, 0x64006400u)), so, bo));
            }
        }
        tmem_st_x8(a_tmem + ((uint32_t)(16 * r) << 16) + 32 * c, out);
    }
}

// One 128-input half `cc` of Q6_K for warp quarter c = kh + 2 hi: inputs 16 kh .. of the groups of variants 2 hi, 2 hi + 1.
// p = sc (q - 32): plane one holds p rounded to binary16, plane two (64 columns on) the exact rest.
__device__ __forceinline__ void convert_q6k(uint32_t tile, int cc, int c, uint32_t a_tmem, uint32_t scales, int row0, int lane) {
    const int g = lane >> 2, t = lane & 3, kh = c & 1, hi = c >> 1;
    const uint32_t sel0 = kh ? 0x4141u : 0x4040u, sel1 = kh ? 0x4343u : 0x4242u;
    const uint32_t lm = hi ? 0x00F000F0u : 0x000F000Fu, hm = hi ? 0x03000300u : 0x00300030u;
    // 1024 + q, or 1024 + 16 q: to q - 32
    const __half2 mul = __float2half2_rn(hi ? 0.0625f : 1.0f), bias = __float2half2_rn(hi ? -96.0f : -1056.0f);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint32_t at = tile + r * 3360;
        const uint4 w = lds128(at + (cc * 2 + kh) * 512 + lane * 16);
        const uint4 qh = lds128(at + 2048 + cc * 512 + lane * 16);
        uint32_t p1[8], p2[8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = g + 8 * h;
            const uint32_t s4 = lds32(at + 3072 + row * 16 + cc * 8 + 4 * hi) ^ 0x80808080u;
            if (cc == 0 && c == 0 && t == 0) {
                const float d = __half2float(__ushort_as_half((unsigned short)lds16(at + 3328 + row * 2)));
                asm volatile("st.shared.v2.f32 [%0], {%1,%2};" ::"r"(scales + (row0 + r * 16 + row) * 8), "f"(d), "f"(0.0f) : "memory");
            }
            const uint32_t high = h == 0 ? (kh == 0 ? qh.x : qh.z) : (kh == 0 ? qh.y : qh.w);
#pragma unroll
            for (int vv = 0; vv < 2; ++vv) {
                const __half2 sc = __hsub2(as_half2(__byte_perm(s4, 0x64646464u, vv ? sel1 : sel0)), __float2half2_rn(1152.0f));
                const uint32_t low = h == 0 ? (vv ? w.y : w.x) : (vv ? w.w : w.z);
                const uint32_t up = vv ? high << 2 : high << 4, down = vv ? high >> 6 : high >> 4;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t x = and_or(i ? low >> 8 : low, lm, and_or(i ? down : up, hm, 0x64006400u));
                    const __half2 v = __hfma2(as_half2(x), mul, bias), p = __hmul2(sc, v);
                    p1[(2 * vv + i) * 2 + h] = as_bits(p);
                    p2[(2 * vv + i) * 2 + h] = as_bits(__hfma2(sc, v, __hneg2(p)));
                }
            }
        }
        tmem_st_x4(a_tmem + ((uint32_t)(16 * r) << 16) + 16 * c, p1);
        tmem_st_x4(a_tmem + ((uint32_t)(16 * r) << 16) + 64 + 16 * c, p2);
    }
}

// Columns of a launch's operand: MP rows of activations per group.
template <int MP>
struct Cols {
    static constexpr bool kJoined = MP <= 32;               // hi and lo parts side by side in one MMA, or one after the other
    static constexpr int kSumCols = MP < 16 ? 16 : (MP + 15) / 16 * 16;
    static constexpr int kMain = 1024 * MP, kSums = 32 * kSumCols;
    static constexpr int kBlock = kMain + kSums + 4 * MP;
};

struct TaRings { int w_stages, b_stages, w_bytes; };

template <int MP>
__global__ void __launch_bounds__(kThreads, 1) gemm_ta_kernel(const StepGemm a, const StepSplit split, const TaRings rings) {
    using C = Cols<MP>;
    constexpr int kBBytes = (C::kBlock + 127) & ~127;
    extern __shared__ __align__(128) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t spin_limit = a.spin_limit ? a.spin_limit : kSpinLimit;
    const int nw = rings.w_stages, nb = rings.b_stages, k_tiles = split.k_tiles;
    const uint32_t w_ring = smem_u32(smem), b_ring = w_ring + nw * rings.w_bytes, a2_buf = b_ring + nb * kBBytes,
                   scales_ring = a2_buf + 2 * kA2Bytes, inv_at = scales_ring + 4 * kRows * 8, tmem_slot = inv_at + MP * 4, bars = tmem_slot + 16;
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
                const int item = s / k_tiles, end = min(s1, (item + 1) * k_tiles);
                const UnitAt at = unit_at(a, item / split.groups);
                const GemvSegment& seg = a.seg[at.seg];
                const uint32_t bytes = kUnitTiles * (uint32_t)packed_tile_bytes(seg.type);
                for (int kb = s - item * k_tiles; s < end; ++s, ++kb) {
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
                const int item = s / k_tiles, end = min(s1, (item + 1) * k_tiles);
                const unsigned char* from = a.blocks + ((size_t)(item % split.groups) * k_tiles + (s - item * k_tiles)) * C::kBlock;
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
        } else if (warp == kMmaWarp && lane == 0) {
            // ---------------- MMA issue ----------------
            constexpr uint32_t kBLbo = 2 * MP * 16;
            constexpr uint64_t kStep = 2 * kBLbo >> 4, kLo = MP * 16 >> 4;   // descriptor units: a k16 step, the lo columns
            constexpr uint32_t idesc_both = umma_idesc(2 * MP), idesc_one = umma_idesc(MP), idesc_sum = umma_idesc(C::kSumCols);
            const uint64_t b_desc0 = umma_desc(b_ring, kBLbo, 128), sum_desc0 = umma_desc(b_ring + C::kMain, C::kSumCols * 16, 128),
                           a2_desc0 = umma_desc(a2_buf, kA2Lbo, 128);
            int bs = 0, fold_slot = 0;
            uint32_t b_parity = 0, fold_parity = 0, a_count = 0, kt = 0, q6_count = 0;
            for (int s = s0; s < s1;) {
                const int item = s / k_tiles, end = min(s1, (item + 1) * k_tiles);
                const bool q4k = a.seg[unit_at(a, item / split.groups).seg].type == kQ4_K;
                for (; s < end; ++s, ++kt) {
                    const uint32_t p = kt & 1u, d_main = tmem + 64 * p, d_min = tmem + 128 + 64 * p;
                    if (kt >= 2) {   // the fold of k tile kt - 2 has left these sums
                        if (alive) alive = mbar_wait(folded + 8 * fold_slot, fold_parity, a.error_flag, 93, spin_limit);
                        if (++fold_slot == nb) { fold_slot = 0; fold_parity ^= 1u; }
                    }
                    if (alive) alive = mbar_wait(b_full + 8 * bs, b_parity, a.error_flag, 94, spin_limit);
                    const uint64_t b_desc = b_desc0 + (uint64_t)(bs * (kBBytes >> 4));
                    const uint32_t st = a_count & 1u, a_at = tmem + 256 + 128 * st;
                    if (alive) alive = mbar_wait(a_full + 8 * st, (a_count >> 1) & 1u, a.error_flag, 95, spin_limit);
                    tc_fence_after();
                    if (q4k) {
                        umma_ss(d_min, a2_desc0 + (uint64_t)(st * (kA2Bytes >> 4)), sum_desc0 + (uint64_t)(bs * (kBBytes >> 4)), idesc_sum, 0u);
                        if (C::kJoined) {
#pragma unroll
                            for (int i = 0; i < 16; ++i) umma_ts(d_main, a_at + 8 * i, b_desc + i * kStep, idesc_both, i != 0);
                        } else {   // lo parts first: the sums they join are still small
#pragma unroll
                            for (int i = 0; i < 16; ++i) umma_ts(d_main, a_at + 8 * i, b_desc + kLo + i * kStep, idesc_one, i != 0);
#pragma unroll
                            for (int i = 0; i < 16; ++i) umma_ts(d_main, a_at + 8 * i, b_desc + i * kStep, idesc_one, 1u);
                        }
                        ++a_count;
                    } else {
#pragma unroll 1
                        for (int half = 0; half < 2; ++half, ++a_count) {
                            const uint32_t hs = a_count & 1u, h_at = tmem + 256 + 128 * hs;
                            if (half == 1) {
                                umma_commit(half_done + 8 * (q6_count & 1u));
                                ++q6_count;
                                if (alive) alive = mbar_wait(a_full + 8 * hs, (a_count >> 1) & 1u, a.error_flag, 95, spin_limit);
                                tc_fence_after();
                            }
                            const uint64_t b_half = b_desc + 8 * half * kStep;
                            // position i of the stage holds step 4 (i >> 2) + 2 (i & 1) + ((i >> 1) & 1) of the half.
                            // p2 x lo is below F32's resolution: left out where it costs an MMA.
#pragma unroll
                            for (int pass = C::kJoined ? 1 : 0; pass < 3; ++pass) {   // (lo x p1 apart,) p1, p2
#pragma unroll
                                for (int i = 0; i < 8; ++i) {
                                    const uint64_t b = b_half + (4 * (i >> 2) + 2 * (i & 1) + ((i >> 1) & 1)) * kStep;
                                    const uint32_t acc = (i != 0 || pass != (C::kJoined ? 1 : 0)) ? 1u : (uint32_t)half;
                                    if (pass == 0) umma_ts(d_main, h_at + 8 * i, b + kLo, idesc_one, acc);
                                    else umma_ts(d_main, h_at + (pass == 2 ? 64 : 0) + 8 * i, b, C::kJoined ? idesc_both : idesc_one, acc);
                                }
                            }
                        }
                    }
                    umma_commit(done + 8 * bs);
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
            const int item = s / k_tiles, end = min(s1, (item + 1) * k_tiles);
            const int type = a.seg[unit_at(a, item / split.groups).seg].type;
            for (; s < end; ++s, ++kt) {
                if (alive) alive = mbar_wait(w_full + 8 * ws, parity, a.error_flag, 96, spin_limit);
                const uint32_t tile = w_ring + ws * rings.w_bytes + 2 * quadrant * packed_tile_bytes(type);
                const uint32_t scales = scales_ring + (kt & 3u) * (kRows * 8);
                const int halves = type == kQ4_K ? 1 : 2;
                for (int half = 0; half < halves; ++half, ++a_count) {
                    const uint32_t st = a_count & 1u, a_at = tmem + 256 + 128 * st + ((uint32_t)(32 * quadrant) << 16);
                    stage_free(st);
                    by_half = (by_half & ~(1u << st)) | ((uint32_t)(halves == 2 && half == 0) << st);
                    tc_fence_after();
                    if (type == kQ4_K) {
#pragma unroll 1
                        for (int c = 2 * part; c < 2 * part + 2; ++c) convert_q4k(tile, c, a_at, scales, a2_buf + st * kA2Bytes, 32 * quadrant, lane);
                    } else {
#pragma unroll 1
                        for (int hi = 0; hi < 2; ++hi) convert_q6k(tile, half, part + 2 * hi, a_at, scales, 32 * quadrant, lane);
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
        int bs = 0, inv_group = -1;
        uint32_t b_parity = 0, kt = 0;
        float* inv = reinterpret_cast<float*>(smem + (inv_at - w_ring));
        for (int s = s0; s < s1;) {
            const int item = s / k_tiles, unit = item / split.groups, group = item - unit * split.groups;
            const UnitAt at = unit_at(a, unit);
            const GemvSegment& seg = a.seg[at.seg];
            const bool q4k = seg.type == kQ4_K;
            const int end = min(s1, (item + 1) * k_tiles);
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
                float x[kChunks][8], y[kChunks][8], z[kChunks][8];
#pragma unroll
                for (int j = 0; j < kChunks; ++j) {
                    if (16 * j + mine < MP) {
                        tmem_ld8(t_main + 16 * j, x[j]);
                        if (C::kJoined) tmem_ld8(t_main + MP + 16 * j, y[j]);
                        if (q4k) tmem_ld8(t_min + 16 * j, z[j]);
                    }
                }
                float d, dmin;
                asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(d), "=f"(dmin) : "r"(scales_ring + (kt & 3u) * (kRows * 8) + row * 8));
                const uint32_t sx_at = b_ring + bs * kBBytes + C::kMain + C::kSums + mine * 4;
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < kChunks; ++j) {
                    if (16 * j + mine < MP) {
                        tmem_tie(x[j]);
                        if (C::kJoined) tmem_tie(y[j]);
                        if (q4k) tmem_tie(z[j]);
                        float sx[8];
#pragma unroll
                        for (int i = 0; i < 8; i += 4) {
                            asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(sx[i]), "=f"(sx[i + 1]), "=f"(sx[i + 2]), "=f"(sx[i + 3])
                                         : "r"(sx_at + (16 * j + i) * 4));
                        }
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            float v = d * (C::kJoined ? x[j][i] + y[j][i] : x[j][i]);
                            if (q4k) v = fmaf(-dmin, z[j][i], v);
                            acc[j][i] = fmaf(sx[i], v, acc[j][i]);
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(folded + 8 * bs);
                if (++bs == nb) { bs = 0; b_parity ^= 1u; }
            }
            if (a.partial == nullptr && group != inv_group) {
                inv_group = group;
                asm volatile("bar.sync 1, 256;" ::: "memory");   // the previous group's factors have been read
                for (int m = warp; m < MP; m += kEpilogueWarps) {
                    const int member = group * MP + m;
                    float sum = 0.0f;
                    if (a.ss != nullptr && member < a.members) for (int i = lane; i < k_tiles; i += 32) sum += a.ss[(size_t)member * k_tiles + i];
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                    if (lane == 0) inv[m] = a.ss != nullptr ? 1.0f / sqrtf(sum / (float)a.k + a.eps) : 1.0f;
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
            }
            const int n_index = at.rt0 * kTileRows + row;
            if (n_index < seg.n) {
                float* part = a.partial + (size_t)((int)blockIdx.x - split.first_worker(item)) * a.members * a.total_n + a.n_offset[at.seg] + n_index;
#pragma unroll
                for (int j = 0; j < kChunks; ++j) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int m = 16 * j + mine + i, member = group * MP + m;
                        if (m >= MP || member >= a.members) continue;
                        if (a.partial != nullptr) {
                            part[(size_t)member * a.total_n] = acc[j][i];
                        } else {
                            float* y = seg.y + (size_t)member * seg.n + n_index;
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

template <int MP>
cudaError_t launch_variant(cudaStream_t stream, const StepGemm& a, int w_bytes, bool programmatic) {
    static bool configured[kMaxDevices] = {false};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    if (!configured[dev]) {
        e = cudaFuncSetAttribute(gemm_ta_kernel<MP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    TaRings rings{};
    rings.w_bytes = (w_bytes + 127) & ~127;
    const size_t b_bytes = (size_t)((Cols<MP>::kBlock + 127) & ~127), fixed = 2 * kA2Bytes + 4 * kRows * 8 + MP * 4 + 16 + 352;
    rings.b_stages = MP <= 8 ? 5 : MP <= 16 ? 4 : MP <= 32 ? 3 : 2;
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
    return cudaLaunchKernelEx(&cfg, gemm_ta_kernel<MP>, a, split, rings);
}

}  // namespace

cudaError_t launch_gemm_ta(cudaStream_t stream, const StepGemm& a, int w_bytes, bool programmatic) {
    switch (step_shape(a.members, kColumnForm).ng) {
        case 1: return launch_variant<8>(stream, a, w_bytes, programmatic);
        case 2: return launch_variant<16>(stream, a, w_bytes, programmatic);
        case 3: return launch_variant<24>(stream, a, w_bytes, programmatic);
        case 4: return launch_variant<32>(stream, a, w_bytes, programmatic);
        case 6: return launch_variant<48>(stream, a, w_bytes, programmatic);
        default: return launch_variant<64>(stream, a, w_bytes, programmatic);
    }
}

}  // namespace ribn
