// What the step GEMMs share: barriers, copies and shared-memory loads, and, of the tcgen05 kernels with a tensor-memory A
// operand, tensor-memory accesses and the conversion of packed Q4_K / Q6_K / Q8_0 tiles to operand columns.
#pragma once
#include <cuda_fp16.h>

#include "blocks.cuh"
#include "gemv.cuh"

namespace ribn {

constexpr int kUnitRows = kUnitTiles * kTileRows;   // 128: tensor-memory lanes
constexpr int kA2Bytes = kUnitRows * 16 * 2;        // minima operand: 128 rows x (8 minima, twice) halves
constexpr int kA2Lbo = kUnitRows / 8 * 128;         // bytes between its two 8-input column blocks

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
// Shared-memory operand descriptor, K-major, no swizzle (8 rows x 16 bytes core matrices, 128 bytes between groups of
// eight rows; see gemm_tc.cu).  Only the low word differs between operands: start address and `lbo`, in 16-byte units.
__device__ __forceinline__ uint32_t umma_desc(uint32_t smem_addr, uint32_t lbo) { return ((smem_addr >> 4) & 0x3FFFu) | ((lbo >> 4) << 16); }
constexpr uint32_t kDescHigh = (128u >> 4) | (1u << 14);
// kind::f16: F32 accumulate, F16 x F16, M = 128
__host__ __device__ constexpr uint32_t umma_idesc(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kUnitRows >> 4) << 24); }
__device__ __forceinline__ void umma_ts(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 b, {%2, %6};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(kDescHigh) : "memory");
}
__device__ __forceinline__ void umma_ss(uint32_t d_tmem, uint32_t a_desc, uint32_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 a, {%1, %6};\n\t"
        "mov.b64 b, {%2, %6};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(d_tmem), "r"(a_desc), "r"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(kDescHigh) : "memory");
}
// The same with the lane's predicate on the instruction itself instead of a branch around it: 64 clocks at N = 128, where the
// branch form takes 74 (and 64 at every smaller N, where the branch form is the faster one).
__device__ __forceinline__ void umma_ts_if(bool leader, uint32_t d_tmem, uint32_t a_tmem, uint32_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .b64 b;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %7, 0;\n\t"
        "mov.b64 b, {%2, %6};\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(kDescHigh), "r"((uint32_t)leader) : "memory");
}
// One lane of the warp, for `if (leader)` around MMAs and commits.  The warp runs the issuing loop as a whole so that the
// compiler keeps addresses and descriptors in uniform registers: issued from a `threadIdx` branch an MMA cost 110 clocks of
// register moves whatever its size, against 22 (N = 16) to 74 (N = 128) this way.
__device__ __forceinline__ bool elect_one() {
    uint32_t leader;
    asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.u32 %0, 1, 0, P;\n\t}" : "=r"(leader));
    return leader != 0;
}
__device__ __forceinline__ int uniform_warp() { return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0); }
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
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float (&v)[4]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];" : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]) : "r"(taddr));
}
// Waits for the thread's loads; the values are tied to the wait, so that nothing uses them before it.
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_tie(float (&x)[8]) {
    asm volatile("" : "+f"(x[0]), "+f"(x[1]), "+f"(x[2]), "+f"(x[3]), "+f"(x[4]), "+f"(x[5]), "+f"(x[6]), "+f"(x[7]) :: "memory");
}
__device__ __forceinline__ void tmem_tie(float (&x)[4]) { asm volatile("" : "+f"(x[0]), "+f"(x[1]), "+f"(x[2]), "+f"(x[3]) :: "memory"); }

// The block type of a launch's matrices where it is one for all (the kernels are compiled for each: without the other types'
// branches they run 5 to 15 % faster), else kKQuants or kAnyType.
constexpr int kAnyType = -1, kKQuants = -2;
template <int TYPE>
__device__ __forceinline__ int type_of(const GemvSegment& s) { return TYPE < 0 ? s.type : TYPE; }
inline int common_type(const StepGemm& a) {
    bool same = true, k_quants = true;
    for (int i = 0; i < a.n_segments; ++i) {
        same = same && a.seg[i].type == a.seg[0].type;
        k_quants = k_quants && (a.seg[i].type == kQ4_K || a.seg[i].type == kQ6_K);
    }
    return same ? a.seg[0].type : k_quants ? kKQuants : kAnyType;
}

struct UnitAt { int seg, rt0; };
// Unit u of the launch: units of `tiles` row tiles, whole units per segment.
__device__ __forceinline__ UnitAt unit_at(const StepGemm& a, int u, int tiles) {
    UnitAt r{0, u * tiles};
    while (r.seg + 1 < a.n_segments) {
        const int have = (a.seg[r.seg].row_tiles + tiles - 1) / tiles * tiles;
        if (r.rt0 < have) break;
        r.rt0 -= have;
        ++r.seg;
    }
    return r;
}

// ---- conversion ------------------------------------------------------------------------------------------------
// Rows g and g + 8 of two row tiles (`tile`, `tile` + tile bytes) of one 64-input chunk c of Q4_K: A = sc q, exact, into
// 32 columns from a_tmem on.  Chunk 0 also leaves the rows' (d, dmin) binary16 pairs and the minima operand.
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
                if (t == 0) asm volatile("st.shared.u32 [%0], %1;" ::"r"(scales + row * 4), "r"(hd.x) : "memory");
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
        tmem_st_x8(a_tmem + ((uint32_t)(16 * r) << 16), out);
    }
}

// One 128-input half `cc` of Q6_K for warp quarter c = kh + 2 hi: inputs 16 kh .. of the groups of variants 2 hi, 2 hi + 1.
// p = sc (q - 32): 16 columns from a_tmem on hold p rounded to binary16, those `plane` columns further the exact rest.
__device__ __forceinline__ void convert_q6k(uint32_t tile, int cc, int c, uint32_t a_tmem, uint32_t plane, uint32_t scales, int row0, int lane) {
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
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(scales + (row0 + r * 16 + row) * 4), "r"(lds16(at + 3328 + row * 2)) : "memory");
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
        tmem_st_x4(a_tmem + ((uint32_t)(16 * r) << 16), p1);
        tmem_st_x4(a_tmem + ((uint32_t)(16 * r) << 16) + plane, p2);
    }
}

// The same quarter of a Q8_0 half: p = d' q with d' = d 2^s, s the power of two that brings the largest of the row's eight d
// of this tile into [128, 256) (so p stays below 65,504, and what binary16 cannot hold of the rest lies 2^-39 below the
// largest p); the row's scale for the fold is 2^-s.
__device__ __forceinline__ void convert_q8_0(uint32_t tile, int cc, int c, uint32_t a_tmem, uint32_t plane, uint32_t scales, int row0, int lane) {
    const int g = lane >> 2, t = lane & 3, kh = c & 1, hi = c >> 1;
    const __half2 bias = __float2half2_rn(1152.0f);   // 1024 + 128
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint32_t at = tile + r * 4352;
        uint32_t p1[8], p2[8];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int row = g + 8 * h;
            const uint4 d8 = lds128(at + 4096 + row * 16);
            uint32_t top = __vmaxu2(__vmaxu2(d8.x & 0x7FFF7FFFu, d8.y & 0x7FFF7FFFu), __vmaxu2(d8.z & 0x7FFF7FFFu, d8.w & 0x7FFF7FFFu));
            top = max(top & 0xffffu, top >> 16);
            const int s = 22 - (int)(top >> 10);
            if (cc == 0 && c == 0 && t == 0) {
                const uint32_t back = s <= 14 ? (uint32_t)(15 - s) << 10 : 1u << (24 - s);   // 2^-s as binary16
                asm volatile("st.shared.u32 [%0], %1;" ::"r"(scales + (row0 + r * 16 + row) * 4), "r"(back) : "memory");
            }
            const uint32_t two = cc == 0 ? (hi ? d8.y : d8.x) : (hi ? d8.w : d8.z);          // d of blocks 4 cc + 2 hi, + 1
            const float up = __int_as_float((s + 127) << 23);
            const float2 df = __half22float2(as_half2(two));
#pragma unroll
            for (int vv = 0; vv < 2; ++vv) {
                const __half2 sc = __float2half2_rn((vv ? df.y : df.x) * up);
                const uint32_t word = lds32(at + (cc * 4 + 2 * hi + vv) * 512 + lane * 16 + 8 * h + 4 * kh);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const __half2 v = __hsub2(as_half2(and_or(i ? word >> 8 : word, 0x00FF00FFu, 0x64006400u)), bias), p = __hmul2(sc, v);
                    p1[(2 * vv + i) * 2 + h] = as_bits(p);
                    p2[(2 * vv + i) * 2 + h] = as_bits(__hfma2(sc, v, __hneg2(p)));
                }
            }
        }
        tmem_st_x4(a_tmem + ((uint32_t)(16 * r) << 16), p1);
        tmem_st_x4(a_tmem + ((uint32_t)(16 * r) << 16) + plane, p2);
    }
}

}  // namespace ribn
