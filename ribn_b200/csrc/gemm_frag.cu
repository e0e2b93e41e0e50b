// Dequant-GEMM in MMA-fragment order for batches of 3 and more rows, any packed block type.
//
//   y[m][n] = sum_k deq(W[n][k]) x[m][k]
//
// The packed tiles already hold, per lane, the bytes of its MMA A fragments, so a weight never passes through
// shared memory a second time: a lane masks its bytes straight into binary16 SUBNORMALS (the bit pattern of an
// integer i below 1024 is the number i 2^-24), about one LOP3 per two weights, and `mma.sync.m16n8k16` adds them against
// the activations' binary16 hi + lo pairs.  By its errors the tensor core aligns a step's products as if a subnormal
// were a full-scale 2^-14 and cuts what falls below the sum's F32 resolution there, so an integer has to fill the ten bits to be added as
// exactly as a normal number: Q8_0's eight bits do (3e-7 of a row's results from the exact ones at K = 4,096), Q4_K's
// nibbles are taken four bits up (2.6e-7; as they lie 1.8e-6, and 5.6e-6 with the wide-ranging inputs that a gate leaves,
// against 7e-7 and 8e-7 of the kernel of gemm_tc.cu), and Q6_K's six bits become the signed normal number q - 32, which
// also spares the cancellation of an offset (1.3e-7; as they lie 5e-7, and 1.5e-6 with those inputs).  The shifts take 0.9 %
// of a step of 5 rows of the 8B model; without the offset's product a step of 16 rows is 0.6 % faster.
//
// One group of inputs that shares a block scale (32 inputs of Q4_K and Q8_0, 16 of Q6_K) is one chain of MMAs; its F32 sum
// is folded into the tile's sum with the group's exact F32 scale, and the tile's (256 inputs) into the row's sum with the
// activations' power-of-two scale, both round-to-nearest.  Offsets (Q4_K minima, Q8_0 -128) are one more MMA per tile
// against the activations' group sums.
//
// Why not a tcgen05 pipeline that converts its A operand through shared memory: at these row counts its hand-offs
// (packed ring -> registers -> shared memory -> MMA -> commit -> tensor memory -> registers) cost several
// microseconds per 128 x 256 tile, whatever the row count.  Here a warp has no hand-off between the copy of a tile
// and its sums.
//
// Execution: one persistent CTA per SM; a producer thread streams ring slots (the eight row tiles of a 128-row unit
// at one k tile, one tensor copy, and the activations' block of that k tile), weights before the programmatic
// dependency on the previous kernel resolves.  Two teams of four warps work on their own slots, a warp on two row
// tiles (so that an activation fragment read from shared memory serves two).  The launch's slots are dealt out to
// the teams in whole units when a unit's result is stored by this kernel, else evenly: a unit's partial sums are then
// added in worker order by the kernel that consumes them.  Sums are ordered; a row's result does not depend on what it
// is batched with.  Every wait is bounded and raises the caller's error word.
#include <cuda_fp16.h>

#include <algorithm>

#include "blocks.cuh"
#include "gemv.cuh"
#include "tmem.cuh"

namespace ribn {

namespace {

constexpr int kTeams = kFragTeams;
constexpr int kTeamWarps = 4;                    // warps per team, two row tiles each
constexpr int kWarps = kTeams * kTeamWarps;
constexpr int kThreads = (kTeams + 1) * kTeamWarps * 32;
constexpr uint32_t kSpinLimit = 1u << 22;
constexpr size_t kSmemBudget = 220 * 1024;

__device__ __forceinline__ uint2 lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ float2 lds64f(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void sts128f(uint32_t addr, float2 a, float2 b) {
    asm volatile("st.shared.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y) : "memory");
}
__device__ __forceinline__ void sts32f(uint32_t addr, float a) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(a) : "memory"); }
// D = A B (fresh accumulator) and D += A B
__device__ __forceinline__ void mma_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ void mma_next(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// bytes i and i + 1 of w as floats minus `bias` (exact), times f
__device__ __forceinline__ float2 bytes_scaled(uint32_t w, int i, float bias, float2 f) {
    const float2 raw = make_float2(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u | (uint32_t)i)),
                                   __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540u | (uint32_t)(i + 1))));
    return __fmul2_rn(__fadd2_rn(raw, make_float2(-bias, -bias)), f);
}
__device__ __forceinline__ float half_low(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w & 0xffffu))); }
__device__ __forceinline__ float half_high(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w >> 16))); }

constexpr float kTwo24 = 16777216.0f, kTwo20 = 1048576.0f;   // an integer masked into binary16 is that integer times 2^-24
// bytes i and j of w (selector 0x4j4i) as a pair of normal binary16 integers
__device__ __forceinline__ uint32_t bytes_half2(uint32_t w, uint32_t selector) {
    return as_bits(__hsub2(as_half2(__byte_perm(w, 0x64646464u, selector)), __float2half2_rn(1024.0f)));
}

// c: (row g, columns 2t, 2t + 1), (row g + 8, the same); s0 / s1: factors of rows g / g + 8
__device__ __forceinline__ void fold(float (&acc)[4], const float (&c)[4], float s0, float s1) {
    const float2 lo = __ffma2_rn(make_float2(s0, s0), make_float2(c[0], c[1]), make_float2(acc[0], acc[1]));
    const float2 hi = __ffma2_rn(make_float2(s1, s1), make_float2(c[2], c[3]), make_float2(acc[2], acc[3]));
    acc[0] = lo.x; acc[1] = lo.y; acc[2] = hi.x; acc[3] = hi.y;
}

// A fragments of one k16 step: registers 0 / 2 are row g's input pairs (4t, 4t + 2) and (4t + 1, 4t + 3), 1 / 3 row g + 8's.
struct Frag { uint32_t r[4]; };

// One scale group of both row tiles against every column group: lo parts first (the accumulator is still small), then
// hi parts; the 2 NG chains advance side by side.
template <int NG, int STEPS>
__device__ __forceinline__ void group_mma(float (&d)[2][NG][4], const Frag (&a)[2][STEPS], const uint4 (&b)[STEPS][NG]) {
#pragma unroll
    for (int s = 0; s < STEPS; ++s) {
#pragma unroll
        for (int n = 0; n < NG; ++n) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if (s == 0) mma_first(d[r][n], a[r][s].r[0], a[r][s].r[1], a[r][s].r[2], a[r][s].r[3], b[s][n].z, b[s][n].w);
                else mma_next(d[r][n], a[r][s].r[0], a[r][s].r[1], a[r][s].r[2], a[r][s].r[3], b[s][n].z, b[s][n].w);
            }
        }
    }
#pragma unroll
    for (int s = 0; s < STEPS; ++s) {
#pragma unroll
        for (int n = 0; n < NG; ++n) {
#pragma unroll
            for (int r = 0; r < 2; ++r) mma_next(d[r][n], a[r][s].r[0], a[r][s].r[1], a[r][s].r[2], a[r][s].r[3], b[s][n].x, b[s][n].y);
        }
    }
}

template <int NG>
using TileSums = float[2][NG][4];

// A warp's row records: its 32 rows' scales as F32 and the minima's A operand, written by lane = row (decoding a row's
// header once instead of in each of the four lanes that need it) and read back in fragment order.
//   words 0..7 scales, 8..11 Q4_K minima (binary16 pairs), 12 their factor; a pitch of 20 words is conflict-free
constexpr int kRecWords = 20;
struct Record {
    uint32_t wr, rd;   // this lane's row / row g of the warp's first row tile
};
__device__ __forceinline__ float2 rec_scales(const Record& rec, int r, int h, int pair) {   // scales 2 pair, 2 pair + 1
    return lds64f(rec.rd + (uint32_t)((r * 16 + h * 8) * kRecWords + 2 * pair) * 4u);
}
__device__ __forceinline__ uint32_t rec_word(const Record& rec, int r, int h, int word) {
    return lds32(rec.rd + (uint32_t)((r * 16 + h * 8) * kRecWords + word) * 4u);
}

// ---- Q4_K: w = d sc q - dmin m, groups of 32 --------------------------------------------------------------------
template <int NG>
__device__ __forceinline__ void slot_q4k(uint32_t tile, uint32_t b_at, const Record& rec, int lane, TileSums<NG>& sums) {
    constexpr int kUnroll = NG <= 2 ? 2 : 1;
    const int t = lane & 3;
    {
        const uint4 hd = lds128(tile + (lane >> 4) * 2304 + 2048 + (lane & 15) * 16);
        const float d = half_low(hd.x);
        const uint32_t s_lo = hd.y & 0x3F3F3F3Fu, s_hi = and_or(hd.w, 0x0F0F0F0Fu, (hd.y >> 2) & 0x30303030u);
        const uint32_t m_lo = hd.z & 0x3F3F3F3Fu, m_hi = and_or(hd.w >> 4, 0x0F0F0F0Fu, (hd.z >> 2) & 0x30303030u);
        const float2 dd = make_float2(d * kTwo20, d * kTwo20);   // the nibbles are taken 4 bits up
        sts128f(rec.wr, bytes_scaled(s_lo, 0, 8388608.0f, dd), bytes_scaled(s_lo, 2, 8388608.0f, dd));
        sts128f(rec.wr + 16, bytes_scaled(s_hi, 0, 8388608.0f, dd), bytes_scaled(s_hi, 2, 8388608.0f, dd));
        sts128(rec.wr + 32, bytes_half2(m_lo, 0x4140u), bytes_half2(m_lo, 0x4342u), bytes_half2(m_hi, 0x4140u), bytes_half2(m_hi, 0x4342u));
        sts32f(rec.wr + 48, -half_high(hd.x));
    }
    __syncwarp();
#pragma unroll kUnroll
    for (int j = 0; j < 4; ++j) {
        uint4 w[2];
        float2 f[2][2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            w[r] = lds128(tile + r * 2304 + j * 512 + lane * 16);
            f[r][0] = rec_scales(rec, r, 0, j);
            f[r][1] = rec_scales(rec, r, 1, j);
        }
#pragma unroll
        for (int odd = 0; odd < 2; ++odd) {
            uint4 b[2][NG];
#pragma unroll
            for (int part = 0; part < 2; ++part) {
#pragma unroll
                for (int n = 0; n < NG; ++n) b[part][n] = lds128(b_at + n * kFragBlockBytes + (4 * j + 2 * odd + part) * 512 + lane * 16);
            }
            constexpr uint32_t mask = 0x00F000F0u;
            Frag a[2][2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
#pragma unroll
                for (int part = 0; part < 2; ++part) {
                    const uint32_t top = part == 0 ? w[r].x : w[r].y, bottom = part == 0 ? w[r].z : w[r].w;   // rows g, g + 8
                    a[r][part].r[0] = (odd ? top : top << 4) & mask; a[r][part].r[2] = (odd ? top >> 8 : top >> 4) & mask;
                    a[r][part].r[1] = (odd ? bottom : bottom << 4) & mask; a[r][part].r[3] = (odd ? bottom >> 8 : bottom >> 4) & mask;
                }
            }
            float d[2][NG][4];
            group_mma<NG, 2>(d, a, b);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
#pragma unroll
                for (int n = 0; n < NG; ++n) fold(sums[r][n], d[r][n], odd ? f[r][0].y : f[r][0].x, odd ? f[r][1].y : f[r][1].x);
            }
        }
    }
    // minima (groups 2t, 2t + 1) x group sums: hi sums in the operand's first eight rows, lo sums in its last
#pragma unroll
    for (int n = 0; n < NG; ++n) {
        const uint2 s = lds64(b_at + n * kFragBlockBytes + kFragSumsAt + lane * 8);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t m0 = rec_word(rec, r, 0, 8 + t), m1 = rec_word(rec, r, 1, 8 + t);
            float d[4];
            mma_first(d, m0, m1, m0, m1, s.x, s.y);
            fold(sums[r][n], d, __uint_as_float(rec_word(rec, r, 0, 12)), __uint_as_float(rec_word(rec, r, 1, 12)));
        }
    }
    __syncwarp();   // the records are free again
}

// ---- Q8_0: w = d (u - 128), blocks of 32 ------------------------------------------------------------------------
template <int NG>
__device__ __forceinline__ void slot_q8_0(uint32_t tile, uint32_t b_at, const Record& rec, int lane, TileSums<NG>& sums) {
    constexpr int kUnroll = NG <= 2 ? 2 : 1;
    const int g = lane >> 2, t = lane & 3;
    {
        const uint4 hd = lds128(tile + (lane >> 4) * 4352 + 4096 + (lane & 15) * 16);
        const float2 up = make_float2(kTwo24, kTwo24);
        sts128f(rec.wr, __fmul2_rn(make_float2(half_low(hd.x), half_high(hd.x)), up), __fmul2_rn(make_float2(half_low(hd.y), half_high(hd.y)), up));
        sts128f(rec.wr + 16, __fmul2_rn(make_float2(half_low(hd.z), half_high(hd.z)), up), __fmul2_rn(make_float2(half_low(hd.w), half_high(hd.w)), up));
    }
    __syncwarp();
#pragma unroll kUnroll
    for (int j = 0; j < 4; ++j) {
        float2 f[2][2];
#pragma unroll
        for (int r = 0; r < 2; ++r) { f[r][0] = rec_scales(rec, r, 0, j); f[r][1] = rec_scales(rec, r, 1, j); }
#pragma unroll
        for (int odd = 0; odd < 2; ++odd) {
            const int blk = 2 * j + odd;
            uint4 b[2][NG];
#pragma unroll
            for (int part = 0; part < 2; ++part) {
#pragma unroll
                for (int n = 0; n < NG; ++n) b[part][n] = lds128(b_at + n * kFragBlockBytes + (2 * blk + part) * 512 + lane * 16);
            }
            Frag a[2][2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint4 w = lds128(tile + r * 4352 + blk * 512 + lane * 16);
#pragma unroll
                for (int part = 0; part < 2; ++part) {
                    const uint32_t top = part == 0 ? w.x : w.y, bottom = part == 0 ? w.z : w.w;
                    a[r][part].r[0] = top & 0x00FF00FFu; a[r][part].r[2] = (top >> 8) & 0x00FF00FFu;
                    a[r][part].r[1] = bottom & 0x00FF00FFu; a[r][part].r[3] = (bottom >> 8) & 0x00FF00FFu;
                }
            }
            float d[2][NG][4];
            group_mma<NG, 2>(d, a, b);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
#pragma unroll
                for (int n = 0; n < NG; ++n) fold(sums[r][n], d[r][n], odd ? f[r][0].y : f[r][0].x, odd ? f[r][1].y : f[r][1].x);
            }
        }
    }
    // 128 x d of blocks 2t, 2t + 1 (as they lie in the tile) x block sums
#pragma unroll
    for (int n = 0; n < NG; ++n) {
        const uint2 s = lds64(b_at + n * kFragBlockBytes + kFragSumsAt + lane * 8);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t at = tile + r * 4352 + 4096 + g * 16 + 4 * t;
            const uint32_t d0 = lds32(at), d1 = lds32(at + 128);
            float d[4];
            mma_first(d, d0, d1, d0, d1, s.x, s.y);
            fold(sums[r][n], d, -128.0f, -128.0f);
        }
    }
    __syncwarp();
}

// ---- Q6_K: w = d sc (q - 32), one scale per 16 inputs -----------------------------------------------------------
template <int NG>
__device__ __forceinline__ void slot_q6k(uint32_t tile, uint32_t b_at, const Record& rec, int lane, TileSums<NG>& sums) {
    const uint32_t own = tile + (lane >> 4) * 3360, own_scales = own + 3072 + (lane & 15) * 16;
    const float d = half_low(lds16(own + 3328 + (lane & 15) * 2));
#pragma unroll 1
    for (int c = 0; c < 2; ++c) {
        if (c == 1) __syncwarp();
        {
            // the eight 16-input scales of this half
            uint2 sc = lds64(own_scales + c * 8);
            sc.x ^= 0x80808080u; sc.y ^= 0x80808080u;
            const float2 dd = make_float2(d, d);
            sts128f(rec.wr, bytes_scaled(sc.x, 0, 8388736.0f, dd), bytes_scaled(sc.x, 2, 8388736.0f, dd));
            sts128f(rec.wr + 16, bytes_scaled(sc.y, 0, 8388736.0f, dd), bytes_scaled(sc.y, 2, 8388736.0f, dd));
        }
        __syncwarp();
        uint4 qh[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) qh[r] = lds128(tile + r * 3360 + 2048 + c * 512 + lane * 16);
#pragma unroll
        for (int kh = 0; kh < 2; ++kh) {       // inputs 0..15 / 16..31 of the groups
            uint4 w[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) w[r] = lds128(tile + r * 3360 + (c * 2 + kh) * 512 + lane * 16);
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                uint4 b[1][NG];
#pragma unroll
                for (int n = 0; n < NG; ++n) b[0][n] = lds128(b_at + n * kFragBlockBytes + ((c * 4 + v) * 2 + kh) * 512 + lane * 16);
                Frag a[2][1];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t low = h == 0 ? ((v & 1) ? w[r].y : w[r].x) : ((v & 1) ? w[r].w : w[r].z);
                        const uint32_t high = h == 0 ? (kh == 0 ? qh[r].x : qh[r].z) : (kh == 0 ? qh[r].y : qh[r].w);
                        // the variant's two high bits (bits 2v of each byte) go above its nibble: 1024 + q, or 1024 + 16 q
                        const uint32_t up = (v & 1) ? high << 2 : high << 4, down = (v & 1) ? high >> 6 : high >> 4;
                        const uint32_t lm = v < 2 ? 0x000F000Fu : 0x00F000F0u, hm = v < 2 ? 0x00300030u : 0x03000300u;
                        const __half2 mul = __float2half2_rn(v < 2 ? 1.0f : 0.0625f), bias = __float2half2_rn(v < 2 ? -1056.0f : -96.0f);
                        a[r][0].r[h] = as_bits(__hfma2(as_half2(and_or(low, lm, and_or(up, hm, 0x64006400u))), mul, bias));
                        a[r][0].r[h + 2] = as_bits(__hfma2(as_half2(and_or(low >> 8, lm, and_or(down, hm, 0x64006400u))), mul, bias));
                    }
                }
                float dsum[2][NG][4];
                group_mma<NG, 1>(dsum, a, b);
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const uint32_t f0 = rec_word(rec, r, 0, v * 2 + kh), f1 = rec_word(rec, r, 1, v * 2 + kh);
#pragma unroll
                    for (int n = 0; n < NG; ++n) fold(sums[r][n], dsum[r][n], __uint_as_float(f0), __uint_as_float(f1));
                }
            }
        }
    }
    __syncwarp();
}

// A slot: the tiles, then the activations' block; the tensor copy wants 128-byte aligned destinations.
__host__ __device__ inline int frag_slot_bytes(int w_bytes, int ng) { return (w_bytes + ng * kFragBlockBytes + 127) & ~127; }

// Register shares: the launch gives each of the 384 threads 168 registers (64,512 in all); the consumers' two warpgroups
// then take what the producer's warpgroup (one working thread) hands back: 256 x 232 + 128 x 40 = 64,512.
//
// A kernel for each common block type, as in the other forms: what bounds a team is the chain of one slot (a warp has no
// other work to hide it behind), and the branch between types stands in it.  Against one kernel for all types, 4 layers of
// the 8B model (Q4_K and Q6_K): 5 rows 0.464 -> 0.453 ms, 9 rows 0.576 -> 0.560, 16 rows 0.629 -> 0.617; 3 rows the same.
constexpr int kConsumerRegs = 232, kProducerRegs = 40;

template <int NG, int TYPE>
__global__ void __launch_bounds__(kThreads, 1) gemm_frag_kernel(const StepGemm a, const StepSplit split, const int depth, const int w_bytes) {
    extern __shared__ __align__(128) unsigned char smem[];
    constexpr int kCols = 8 * NG;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t spin_limit = a.spin_limit ? a.spin_limit : kSpinLimit;
    const int slot_bytes = frag_slot_bytes(w_bytes, NG), slots = kTeams * depth;   // team i's ring: slots i depth ..
    const uint32_t records0 = smem_u32(smem + (size_t)slots * slot_bytes);
    const uint32_t full = records0 + kWarps * 32 * kRecWords * 4, empty = full + 8 * slots;
    const int k_tiles = split.k_tiles;

    if (threadIdx.x == 0) {
        for (int i = 0; i < slots; ++i) { mbar_init(full + 8 * i, 1); mbar_init(empty + 8 * i, kTeamWarps); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (warp >= kWarps) {
        // ---------------- producer (one thread): the teams' rings in turn ----------------
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kProducerRegs));
        if (warp > kWarps || lane != 0) return;
        auto issue = [&](int s, int slot, bool weights, bool activations) {
            const int item = s / k_tiles, kb = s - item * k_tiles;
            const UnitAt at = unit_at(a, item / split.groups, kUnitTiles);
            const GemvSegment& seg = a.seg[at.seg];
            const uint32_t bar = full + 8 * slot;
            unsigned char* base = smem + (size_t)slot * slot_bytes;
            if (weights) {
                mbar_expect_tx(bar, kUnitTiles * (uint32_t)packed_tile_bytes(type_of<TYPE>(seg)) + NG * kFragBlockBytes);
                tiles_g2s(smem_u32(base), seg.map, kb, at.rt0, bar);
            }
            if (activations) {
                bulk_g2s(smem_u32(base + w_bytes), a.blocks + ((size_t)(item % split.groups) * k_tiles + kb) * (NG * kFragBlockBytes),
                         NG * kFragBlockBytes, bar);
            }
        };
        int begin[kTeams], end[kTeams], longest = 0;
#pragma unroll
        for (int i = 0; i < kTeams; ++i) {
            begin[i] = split.begin((int)blockIdx.x * kTeams + i);
            end[i] = split.begin((int)blockIdx.x * kTeams + i + 1);
            longest = max(longest, end[i] - begin[i]);
        }
        for (int q = 0; q < min(depth, longest); ++q) {
#pragma unroll
            for (int i = 0; i < kTeams; ++i) if (begin[i] + q < end[i]) issue(begin[i] + q, i * depth + q, true, false);
        }
        asm volatile("griddepcontrol.wait;" ::: "memory");   // the activations come from the previous kernel
        for (int q = 0; q < min(depth, longest); ++q) {
#pragma unroll
            for (int i = 0; i < kTeams; ++i) if (begin[i] + q < end[i]) issue(begin[i] + q, i * depth + q, false, true);
        }
        int slot = 0;
        uint32_t parity = 0;
        bool alive = true;
        for (int q = depth; q < longest && alive; ++q) {
#pragma unroll
            for (int i = 0; i < kTeams; ++i) {
                if (begin[i] + q >= end[i] || !alive) continue;
                alive = mbar_wait(empty + 8 * (i * depth + slot), parity, a.error_flag, 81, spin_limit);
                if (alive) issue(begin[i] + q, i * depth + slot, true, true);
            }
            if (++slot == depth) { slot = 0; parity ^= 1u; }
        }
        if (!alive) {
            // the teams stop waiting too: let what is still in flight land before the block can end
            for (int i = 0; i < slots; ++i) mbar_wait(full + 8 * i, 0, nullptr, 0, spin_limit);
            for (int i = 0; i < slots; ++i) mbar_wait(full + 8 * i, 1, nullptr, 0, spin_limit);
        }
        return;
    }

    // ---------------- a team: four warps, each two of the unit's row tiles, over its own slots ----------------
    // (its ring is its own too: its warps then see every phase of the ring's barriers; a one-bit parity wait for a phase
    // that follows one the warp has not seen complete would pass too early)
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kConsumerRegs));
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int g = lane >> 2, t = lane & 3, team = warp / kTeamWarps, pair = warp % kTeamWarps;
    const int worker = (int)blockIdx.x * kTeams + team;
    const uint32_t records = records0 + (uint32_t)(warp * 32 * kRecWords * 4);
    const Record rec{records + (uint32_t)lane * kRecWords * 4u, records + (uint32_t)g * kRecWords * 4u};
    bool alive = true;
    int slot = 0, inv_group = -1;
    uint32_t parity = 0;
    float inv[NG][2];
#pragma unroll
    for (int n = 0; n < NG; ++n) inv[n][0] = inv[n][1] = 1.0f;
    const int s1 = split.begin(worker + 1);
    for (int s = split.begin(worker); s < s1;) {
        const int item = s / k_tiles, unit = item / split.groups, group = item - unit * split.groups;
        const UnitAt at = unit_at(a, unit, kUnitTiles);
        const GemvSegment& seg = a.seg[at.seg];
        const int type = type_of<TYPE>(seg);
        const bool present = at.rt0 + 2 * pair < seg.row_tiles;   // a pair's absent second tile reads as zeros and is never stored
        const int end = min(s1, (item + 1) * k_tiles);
        float acc[2][NG][4];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
#pragma unroll
            for (int n = 0; n < NG; ++n) acc[r][n][0] = acc[r][n][1] = acc[r][n][2] = acc[r][n][3] = 0.0f;
        }
        for (; s < end; ++s) {
            const uint32_t bar = 8 * (uint32_t)(team * depth + slot);
            if (alive) alive = mbar_wait(full + bar, parity, a.error_flag, 82, spin_limit);
            if (present) {
                const uint32_t base = smem_u32(smem) + (uint32_t)((team * depth + slot) * slot_bytes), b_at = base + w_bytes;
                TileSums<NG> sums;
#pragma unroll
                for (int r = 0; r < 2; ++r) {
#pragma unroll
                    for (int n = 0; n < NG; ++n) sums[r][n][0] = sums[r][n][1] = sums[r][n][2] = sums[r][n][3] = 0.0f;
                }
                const uint32_t tile = base + (uint32_t)(2 * pair * packed_tile_bytes(type));
                if (type == kQ4_K) slot_q4k<NG>(tile, b_at, rec, lane, sums);
                else if (TYPE == kKQuants || type == kQ6_K) slot_q6k<NG>(tile, b_at, rec, lane, sums);
                else slot_q8_0<NG>(tile, b_at, rec, lane, sums);
#pragma unroll
                for (int n = 0; n < NG; ++n) {
                    const float2 sx = lds64f(b_at + n * kFragBlockBytes + kFragScaleAt + 8 * t);
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        acc[r][n][0] = fmaf(sums[r][n][0], sx.x, acc[r][n][0]);
                        acc[r][n][1] = fmaf(sums[r][n][1], sx.y, acc[r][n][1]);
                        acc[r][n][2] = fmaf(sums[r][n][2], sx.x, acc[r][n][2]);
                        acc[r][n][3] = fmaf(sums[r][n][3], sx.y, acc[r][n][3]);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(empty + bar);
            if (++slot == depth) { slot = 0; parity ^= 1u; }
        }
        if (a.partial == nullptr && a.ss != nullptr && group != inv_group) {
            // RMSNorm factors of this lane's columns: the eight lanes of a column share its k tiles' sums of squares
            inv_group = group;
#pragma unroll
            for (int n = 0; n < NG; ++n) {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int m = group * kCols + n * 8 + 2 * t + c;
                    float sum = 0.0f;
                    if (m < a.members) for (int i = g; i < k_tiles; i += 8) sum += a.ss[(size_t)m * k_tiles + i];
#pragma unroll
                    for (int o = 4; o < 32; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                    inv[n][c] = 1.0f / sqrtf(sum / (float)a.k + a.eps);
                }
            }
        }
        const int part = a.partial != nullptr && !split.whole ? worker - split.first_worker(item) : 0;
        const StepSums to = step_sums(a, split, worker, part, group, 2 * t, at.seg, (at.rt0 + 2 * pair) * kTileRows + g);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int n_index = (at.rt0 + 2 * pair + r) * kTileRows + g + 8 * h;
                if (n_index >= seg.n) continue;
#pragma unroll
                for (int n = 0; n < NG; ++n) {
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int m = group * kCols + n * 8 + 2 * t + c;
                        if (m >= a.members) continue;
                        const float v = acc[r][n][2 * h + c];
                        if (a.partial != nullptr) {
                            to.at[(n * 8 + c) * to.stride + r * kTileRows + 8 * h] = v;
                        } else {
                            float* y = seg.y + (size_t)m * seg.n + n_index;
                            *y = a.epilogue == kResidual ? *y + v * inv[n][c] : v * inv[n][c];
                        }
                    }
                }
            }
        }
    }
}

template <int NG, int TYPE>
cudaError_t launch_variant(cudaStream_t stream, const StepGemm& a, int w_bytes, bool programmatic) {
    static bool configured[kMaxDevices] = {false};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    if (!configured[dev]) {
        e = cudaFuncSetAttribute(gemm_frag_kernel<NG, TYPE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBudget);
        if (e != cudaSuccess) return e;
        configured[dev] = true;
    }
    const int slot_bytes = frag_slot_bytes(w_bytes, NG);
    const size_t fixed = (size_t)kWarps * 32 * kRecWords * sizeof(float);
    const int depth = (int)std::min<size_t>(6, (kSmemBudget - fixed) / (slot_bytes + 16) / kTeams);
    if (depth < 1) return cudaErrorInvalidValue;
    const StepSplit split = step_split(a, a.partial == nullptr);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((split.workers + kTeams - 1) / kTeams));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = fixed + (size_t)kTeams * depth * (slot_bytes + 16);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, gemm_frag_kernel<NG, TYPE>, a, split, depth, w_bytes);
}

template <int TYPE>
cudaError_t launch_typed(cudaStream_t stream, const StepGemm& a, int w_bytes, bool programmatic) {
    switch (step_shape(a.members, kFragmentForm).ng) {
        case 1: return launch_variant<1, TYPE>(stream, a, w_bytes, programmatic);
        case 2: return launch_variant<2, TYPE>(stream, a, w_bytes, programmatic);
        case 3: return launch_variant<3, TYPE>(stream, a, w_bytes, programmatic);
        default: return launch_variant<4, TYPE>(stream, a, w_bytes, programmatic);
    }
}

}  // namespace

cudaError_t launch_gemm_frag(cudaStream_t stream, const StepGemm& a, int w_bytes, bool programmatic) {
    switch (common_type(a)) {
        case kQ4_K: return launch_typed<kQ4_K>(stream, a, w_bytes, programmatic);
        case kQ6_K: return launch_typed<kQ6_K>(stream, a, w_bytes, programmatic);
        case kQ8_0: return launch_typed<kQ8_0>(stream, a, w_bytes, programmatic);
        case kKQuants: return launch_typed<kKQuants>(stream, a, w_bytes, programmatic);
        default: return launch_typed<kAnyType>(stream, a, w_bytes, programmatic);
    }
}

}  // namespace ribn
