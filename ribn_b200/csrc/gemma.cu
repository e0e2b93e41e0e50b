// Gemma-4 text decoder for B200: the reference host decoder's arithmetic policy (BF16 storage, FP32
// arithmetic, one BF16 round-to-nearest-even after every operation; crates/gemma4/src/cpu) run as CUDA
// kernels over rows of any number of sequences at once, so every weight matrix is read once per step.
//
// All of this work is BF16 streaming: projections are row-tile GEMVs with 128-bit loads; normalisation,
// rotary, GeGLU and the per-layer-embedding steps are fused per row around them; attention reads each
// owner layer's cache once per (row, head).  Every FP32 sum keeps the reference's source order (see the
// note above the kernels), which is what keeps the BF16-rounded results equal to the reference's.  Rotary
// cos / sin factors are tabulated on the host with the same libm calls the reference makes, so they are
// bit-identical to its BF16 factors.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <map>
#include <string>
#include <vector>

#include "../../include/ribn_b200_gemma.h"

namespace {

typedef uint16_t bf16_t;

__host__ __device__ __forceinline__ float bf_load(bf16_t bits) {
#ifdef __CUDA_ARCH__
    return __uint_as_float((uint32_t)bits << 16);
#else
    uint32_t u = (uint32_t)bits << 16;
    float f;
    memcpy(&f, &u, 4);
    return f;
#endif
}

// crates/gemma4/src/cpu/linear.rs:10-16
__host__ __device__ __forceinline__ bf16_t bf_round(float value) {
#ifdef __CUDA_ARCH__
    const uint32_t bits = __float_as_uint(value);
#else
    uint32_t bits;
    memcpy(&bits, &value, 4);
#endif
    if ((bits & 0x7fffffffu) > 0x7f800000u) return 0x7fc0;
    return (bf16_t)((bits + 0x7fffu + ((bits >> 16) & 1u)) >> 16);
}

// The reference rounds to BF16 after every operation and leaves attention scores unscaled, so a single
// FP32 ULP in a sum can move a rounded score by a whole BF16 step and, through the softmax, the output by
// tens of percent.  Every FP32 sum below therefore adds its terms in the reference's own (source) order:
// one thread owns each sum, and parallelism comes from the many independent sums (output columns, keys,
// channels, rows), not from splitting one.  A product of two BF16 values is exact in FP32, so an FMA
// equals the reference's multiply-then-add.  Transcendentals are evaluated in double and rounded once,
// which is what the host libm's float routines return in all but rare cases.

__device__ __forceinline__ float bf_half(const uint4& v, int e) {   // value e of eight BF16 values; e is a constant after unrolling
    const uint32_t w = e < 2 ? v.x : e < 4 ? v.y : e < 6 ? v.z : v.w;
    return __uint_as_float(e & 1 ? w & 0xffff0000u : w << 16);
}

__device__ __forceinline__ float block_max(float v, float* scratch) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float m = scratch[0];
    for (int w = 1; w < warps; ++w) m = fmaxf(m, scratch[w]);
    return m;
}

// values[0 .. n) added in index order by one thread: 4 cycles per addition when the next 128-bit reads are under way
// while the last ones are added.
__device__ __forceinline__ float ordered_sum(const float* values, int n) {
    constexpr int kBatch = 8;
    const float4* quads = reinterpret_cast<const float4*>(values);
    const int whole = n / (4 * kBatch) * kBatch;
    float total = 0.0f;
    float4 now[kBatch];
    if (whole > 0) {
#pragma unroll
        for (int u = 0; u < kBatch; ++u) now[u] = quads[u];
    }
    for (int i = 0; i < whole; i += kBatch) {
        float4 next[kBatch];
        const float4* ahead = quads + min(i + kBatch, whole - kBatch);
#pragma unroll
        for (int u = 0; u < kBatch; ++u) next[u] = ahead[u];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) { total += now[u].x; total += now[u].y; total += now[u].z; total += now[u].w; }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) now[u] = next[u];
    }
    for (int i = 4 * whole; i < n; ++i) total += values[i];
    return total;
}

// Sum of squares of values[0 .. n) in index order by thread 0, broadcast to the block.  `squares` is a
// shared staging array of n floats the whole block fills first (each square is exact).
__device__ __forceinline__ float ordered_energy(const float* squares, int n, float* slot) {
    __syncthreads();
    if (threadIdx.x == 0) *slot = ordered_sum(squares, n);
    __syncthreads();
    return *slot;
}

// x^(-1/2) rounded once from double (norm.rs:66 calls powf(mean + eps, -0.5)).
__device__ __forceinline__ float inverse_root(float x) { return (float)(1.0 / sqrt((double)x)); }

// elementwise.rs:66-83
__device__ __forceinline__ bf16_t gelu_round(bf16_t v) {
    const float x = bf_load(v);
    // separately rounded operations, as the reference's source-order FP32 expression (no contraction to FMA)
    const float cubic = __fadd_rn(1.0f, __fmul_rn(__fmul_rn(0.044715f, x), x));
    const float inner = __fmul_rn(__fmul_rn(0.7978846f, x), cubic);
    const float hyperbolic = (float)tanh((double)inner);
    return bf_round(__fmul_rn(__fmul_rn(0.5f, x), __fadd_rn(1.0f, hyperbolic)));
}

// ---------------------------------------------------------------------------------------------
// Embedding rows: hidden = bf16(embed[token] * sqrt(H) as BF16), identity = bf16(ple_embed[token] * sqrt(P) as BF16)
// (decoder.rs:346-360).  One block per row.
// ---------------------------------------------------------------------------------------------
__global__ void gm_embed_kernel(const uint32_t* tokens, const bf16_t* __restrict__ embed, const bf16_t* __restrict__ ple_embed, int hidden, int packed,
                                float embed_scale, float ple_scale, bf16_t* __restrict__ out_hidden, bf16_t* __restrict__ out_identity) {
    const int row = blockIdx.x;
    const size_t token = tokens[row];
#pragma unroll 4
    for (int i = threadIdx.x; i < hidden; i += blockDim.x) {
        out_hidden[(size_t)row * hidden + i] = bf_round(bf_load(embed[token * hidden + i]) * embed_scale);
    }
#pragma unroll 4
    for (int i = threadIdx.x; i < packed; i += blockDim.x) {
        out_identity[(size_t)row * packed + i] = bf_round(bf_load(ple_embed[token * packed + i]) * ple_scale);
    }
}

// ---------------------------------------------------------------------------------------------
// Projection: out[r][n] = bf16(sum_k in[r][k] * w[n][k]) (linear.rs:23-66), the sum in k order.  A block is a
// feeder warp and GR x GC consumer warps.  A consumer owns 32 * C output columns for R rows: a thread walks C weight
// rows and keeps R * C independent accumulation chains, fed with BF16 operands as they lie (`fma_half`).  The feeder
// brings tiles of the weights and of the blocks' input rows by cp.async into a ring of stages (rows pitched 16 bytes
// apart from a multiple of 128, so the 128-bit reads of a quarter-warp fall in distinct banks).  Named barriers hand
// the stages over; their ids are constants because an SM has 64 barriers and a block whose ids are computed is given
// 16 of them.  Four consumer warps per block fall on the four schedulers; two-warp blocks leave two without one.
//
// What bounds it: the chain of dependent additions, 4 cycles per input (14.4 us for the 6,912 inputs of a down
// projection), or, with several chains per scheduler, issue and the shared-memory reads (a 128-bit read occupies a
// scheduler's return path about 12 cycles, broadcast or not).  One warp per 32 columns that copied for itself and
// unpacked every operand took 24 cycles per input of four rows.  Measured on a 1,152-wide model, before -> now: a layer's
// three projections to 1,152 columns (1,024, 6,912 and 256 inputs) 105 -> 35 us at 4 rows, 162 -> 64 at 35, 179 -> 87 at
// 113; gate|up 18.6 -> 12.1 us at 4 rows (4.9 of HBM time), 205 -> 113 at 113.
// ---------------------------------------------------------------------------------------------
struct ProjectNarrow { static constexpr int R = 1, C = 1, GR = 1, GC = 1, tile = 256, stages = 4; };   // a few rows: chains spread over blocks
struct ProjectWide { static constexpr int R = 4, C = 1, GR = 1, GC = 4, tile = 128, stages = 3; };     // up to four rows of a wide projection
struct ProjectRows { static constexpr int R = 4, C = 1, GR = 4, GC = 1, tile = 128, stages = 3; };     // a few tens of rows
struct ProjectChunk { static constexpr int R = 4, C = 2, GR = 4, GC = 1, tile = 128, stages = 3; };    // prefill
template <typename V>
struct ProjectShape {
    static constexpr int consumers = V::GR * V::GC, threads = 32 * (1 + consumers);
    static constexpr int cols = 32 * V::C * V::GC, rows = V::R * V::GR;
    static constexpr int chunks = V::tile / 8, pitch = V::tile * 2 + 16;        // 16-byte chunks, and bytes between rows of a tile
    static constexpr int x_offset = cols * pitch, x_bytes = rows * pitch;
    static constexpr int stage_bytes = x_offset + x_bytes, smem_bytes = V::stages * stage_bytes;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// Barrier of stage `slot`: 1 + slot when it is filled, 1 + STAGES + slot when it has been read.
template <int ID, int THREADS>
__device__ __forceinline__ void stage_barrier(bool wait) {
    if (wait) asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(THREADS) : "memory");
    else asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(THREADS) : "memory");
}
template <int FIRST, int STAGES, int THREADS>
__device__ __forceinline__ void stage_barrier(int slot, bool wait) {
    if (slot == 0) stage_barrier<FIRST, THREADS>(wait);
    else if (STAGES <= 2 || slot == 1) stage_barrier<FIRST + 1, THREADS>(wait);
    else if (STAGES <= 3 || slot == 2) stage_barrier<FIRST + (STAGES > 2 ? 2 : 0), THREADS>(wait);
    else stage_barrier<FIRST + (STAGES > 3 ? 3 : 0), THREADS>(wait);
}

// sum + a.e * b.e for value e of eight BF16 values, one rounding (the product of two BF16 values is exact in FP32):
// the instruction takes the halves of a register as they are, so nothing is unpacked.
__device__ __forceinline__ float fma_half(const uint4& a, const uint4& b, float sum, int e) {
    const uint32_t x = e < 2 ? a.x : e < 4 ? a.y : e < 6 ? a.z : a.w, y = e < 2 ? b.x : e < 4 ? b.y : e < 6 ? b.z : b.w;
    float out;
    if (e & 1) asm("{.reg .b16 al, ah, bl, bh; mov.b32 {al, ah}, %1; mov.b32 {bl, bh}, %2; fma.rn.f32.bf16 %0, ah, bh, %3;}" : "=f"(out) : "r"(x), "r"(y), "f"(sum));
    else asm("{.reg .b16 al, ah, bl, bh; mov.b32 {al, ah}, %1; mov.b32 {bl, bh}, %2; fma.rn.f32.bf16 %0, al, bl, %3;}" : "=f"(out) : "r"(x), "r"(y), "f"(sum));
    return out;
}

// Up to three matrices that read the same input rows share one launch (q | k | v, gate | up): their
// column blocks are laid side by side in the grid.
struct ProjectTargets {
    const bf16_t* w[3];
    bf16_t* out[3];
    int n[3];
    int first_block[3];  // first column block of each matrix
    int count;
};

template <typename V>
__global__ void __launch_bounds__(ProjectShape<V>::threads, 4) gm_project_kernel(const bf16_t* __restrict__ in, int rows,
                                                                              const __grid_constant__ ProjectTargets targets, int k) {
    extern __shared__ __align__(16) unsigned char project_smem[];
    using S = ProjectShape<V>;
    constexpr int R = V::R, C = V::C, kStages = V::stages, kThreads = S::threads;
    const int lane = threadIdx.x & 31;
    int which = 0;
    if (targets.count > 1 && (int)blockIdx.x >= targets.first_block[1]) which = 1;
    if (targets.count > 2 && (int)blockIdx.x >= targets.first_block[2]) which = 2;
    const int n = targets.n[which];
    const int col0 = ((int)blockIdx.x - targets.first_block[which]) * S::cols;
    const int r0 = blockIdx.y * S::rows;
    const int live_cols = min(S::cols, n - col0);
    const int chunks = k / 8;  // 16-byte chunks per row
    const int tiles = (chunks + S::chunks - 1) / S::chunks;

    if (threadIdx.x < 32) {   // feeder
        constexpr int kRowsPerIssue = 32 / S::chunks;              // rows one warp-wide copy instruction covers
        const int piece = lane % S::chunks, sub_row = lane / S::chunks;
        const uint4* wsrc = reinterpret_cast<const uint4*>(targets.w[which] + (size_t)(col0 + sub_row) * k) + piece;
        const uint32_t wdst = (uint32_t)__cvta_generic_to_shared(project_smem) + (uint32_t)(sub_row * S::pitch + piece * 16);
        auto copy_weights = [&](int tile, int slot) {
            const int c = tile * S::chunks;
            if (tile >= tiles || c + piece >= chunks) return;
            const uint4* src = wsrc + c;
            uint32_t dst = wdst + (uint32_t)(slot * S::stage_bytes);
#pragma unroll 8
            for (int j = sub_row; j < live_cols; j += kRowsPerIssue, dst += kRowsPerIssue * S::pitch, src += (size_t)kRowsPerIssue * chunks) {
                cp_async16(dst, src);
            }
        };
        auto copy_rows = [&](int tile, int slot) {
            const int c = tile * S::chunks + piece;
            if (tile >= tiles || c >= chunks) return;
            const uint32_t dst = wdst + (uint32_t)(slot * S::stage_bytes + S::x_offset);
#pragma unroll
            for (int j = 0; j < S::rows; j += kRowsPerIssue) {
                if (j + sub_row < S::rows) {
                    cp_async16(dst + (uint32_t)(j * S::pitch), reinterpret_cast<const uint4*>(in) + (size_t)min(r0 + j + sub_row, rows - 1) * chunks + c);
                }
            }
        };
        auto copy = [&](int tile, int slot) {
            copy_weights(tile, slot);
            copy_rows(tile, slot);
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll
        for (int t = 0; t < kStages - 1; ++t) copy(t, t);
        int slot = 0, ahead = kStages - 1;   // slots of tile t and of tile t + kStages - 1
        for (int t = 0; t < tiles; ++t) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");   // tile t; younger copies stay in flight
            __syncwarp();
            stage_barrier<1, kStages, kThreads>(slot, false);
            if (t > 0 && t - 1 + kStages < tiles) stage_barrier<1 + kStages, kStages, kThreads>(ahead, true);   // the consumers have left tile t - 1
            copy(t + kStages - 1, ahead);
            slot = slot + 1 == kStages ? 0 : slot + 1;
            ahead = ahead + 1 == kStages ? 0 : ahead + 1;
        }
        return;
    }

    const int gr = ((int)threadIdx.x / 32 - 1) % V::GR, gc = ((int)threadIdx.x / 32 - 1) / V::GR;
    float sum[C][R];
#pragma unroll
    for (int c = 0; c < C; ++c) {
#pragma unroll
        for (int r = 0; r < R; ++r) sum[c][r] = 0.0f;
    }
    int slot = 0;
    for (int t = 0; t < tiles; ++t) {
        stage_barrier<1, kStages, kThreads>(slot, true);
        const unsigned char* stage = project_smem + (size_t)slot * S::stage_bytes;
        const unsigned char* ws = stage + (gc * 32 * C + lane) * S::pitch;
        const unsigned char* xs = stage + S::x_offset + gr * R * S::pitch;
        const int count = min(S::chunks, chunks - t * S::chunks);
        struct Group { uint4 w[C], x[R]; };   // eight inputs
        auto fetch = [&](Group& to, int i) {
#pragma unroll
            for (int c = 0; c < C; ++c) to.w[c] = *reinterpret_cast<const uint4*>(ws + c * 32 * S::pitch + i * 16);
#pragma unroll
            for (int r = 0; r < R; ++r) to.x[r] = *reinterpret_cast<const uint4*>(xs + r * S::pitch + i * 16);
        };
        auto add = [&](const Group& from) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
#pragma unroll
                for (int c = 0; c < C; ++c) {
#pragma unroll
                    for (int r = 0; r < R; ++r) sum[c][r] = fma_half(from.x[r], from.w[c], sum[c][r], e);
                }
            }
        };
        if (R == 1 && count == S::chunks) {
#pragma unroll 8
            for (int i = 0; i < S::chunks; ++i) { Group one; fetch(one, i); add(one); }
        } else {   // the next group's reads are under way while this one is added
            Group now, next;
            fetch(now, 0);
#pragma unroll 2
            for (int i = 0; i < count; ++i) {
                fetch(next, min(i + 1, count - 1));
                add(now);
                now = next;
            }
        }
        if (t + kStages < tiles) stage_barrier<1 + kStages, kStages, kThreads>(slot, false);
        slot = slot + 1 == kStages ? 0 : slot + 1;
    }
#pragma unroll
    for (int c = 0; c < C; ++c) {
        const int col = gc * 32 * C + lane + 32 * c;
        if (col >= live_cols) break;
        bf16_t* out = targets.out[which] + col0 + col;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int row = r0 + gr * R + r;
            if (row < rows) out[(size_t)row * n] = bf_round(sum[c][r]);
        }
    }
}

// Which variant: the one whose busiest scheduler finishes first, by cycles per input of a consumer warp, alone and for
// each that shares its scheduler (measured for one row, 4.8 and 3.1; for the others near the reads they make).  A narrow
// projection of a few rows goes to one warp per row and 32 columns (1,152 columns x four rows: 144 warps), many rows
// or columns to the variants that spend less per product and read the weights fewer times.
int project_variant(const int* n, int count, int rows, int sms) {
    constexpr int kCols[4] = {64, 32, 128, 32}, kRows[4] = {16, 16, 4, 1};
    constexpr float kAlone[4] = {11.0f, 8.0f, 8.0f, 4.8f}, kShared[4] = {9.5f, 7.5f, 7.5f, 3.1f};
    int best = 0;
    float best_cost = 0.0f;
    for (int v = 0; v < 4; ++v) {
        int blocks = 0;
        for (int i = 0; i < count; ++i) blocks += (n[i] + kCols[v] - 1) / kCols[v];
        blocks *= (rows + kRows[v] - 1) / kRows[v];
        const int per_sm = (blocks + sms - 1) / sms, per_scheduler = v == 3 ? (per_sm + 1) / 2 : per_sm;
        const float cost = std::max(kAlone[v], kShared[v] * (float)per_scheduler);
        if (v == 0 || cost < best_cost) { best = v; best_cost = cost; }
    }
    return best;
}

// ---------------------------------------------------------------------------------------------
// The same projection on the tensor cores, for passes of many rows when the model was created with
// RIBN_B200_GEMMA_FLAG_TENSOR_CORE_PREFILL: BF16 x BF16 products (exact in FP32) accumulated in FP32 by
// `mma.sync.m16n8k16`, one BF16 rounding of each output.  The sums are no longer in source order, so a result
// can differ from the host decoder's by a rounding step of the FP32 sum before the BF16 rounding; the
// ordered kernel above stays the default.  A block of four warps owns 64 rows x 64 columns; warp w owns rows
// 16 w .. 16 w + 15 against all 64 columns.  Inputs and weights arrive in 32-input stages (rows pitched by 80
// bytes: conflict-free matrix loads) through a two-stage cp.async pipeline.  k must be a multiple of 32.
// ---------------------------------------------------------------------------------------------
constexpr int kMmaTile = 64;           // rows and columns per block
constexpr int kMmaStageK = 32;         // inputs per stage
constexpr int kMmaPitch = kMmaStageK * 2 + 16;   // bytes between rows of a stage
constexpr int kMmaStageBytes = 2 * kMmaTile * kMmaPitch;  // input rows, then weight rows

__global__ void __launch_bounds__(128) gm_project_mma_kernel(const bf16_t* __restrict__ in, const int* __restrict__ row_index,
                                                             int rows, const ProjectTargets targets, int k) {
    __shared__ __align__(16) unsigned char stage_smem[2 * kMmaStageBytes];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int which = 0;
    if (targets.count > 1 && (int)blockIdx.x >= targets.first_block[1]) which = 1;
    if (targets.count > 2 && (int)blockIdx.x >= targets.first_block[2]) which = 2;
    const bf16_t* __restrict__ w = targets.w[which];
    bf16_t* __restrict__ out = targets.out[which];
    const int n = targets.n[which];
    const int col0 = ((int)blockIdx.x - targets.first_block[which]) * kMmaTile;
    const int r0 = blockIdx.y * kMmaTile;
    const uint32_t smem = (uint32_t)__cvta_generic_to_shared(stage_smem);
    // copies: a stage holds 64 + 64 rows of 64 bytes = 512 pieces of 16 bytes, four per thread
    const unsigned char* src[4];
    uint32_t dst[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int piece = (int)threadIdx.x + 128 * j, row = piece >> 2, part = piece & 3;   // rows 0..63 inputs, 64..127 weights
        if (row < kMmaTile) {
            const int r = min(r0 + row, rows - 1);
            src[j] = reinterpret_cast<const unsigned char*>(in + (size_t)(row_index ? row_index[r] : r) * k) + part * 16;
        } else {
            const int c = min(col0 + row - kMmaTile, n - 1);
            src[j] = reinterpret_cast<const unsigned char*>(w + (size_t)c * k) + part * 16;
        }
        dst[j] = (uint32_t)(row * kMmaPitch + part * 16);
    }
    const int stages = k / kMmaStageK;
    auto issue = [&](int st) {
        if (st < stages) {
#pragma unroll
            for (int j = 0; j < 4; ++j) cp_async16(smem + (uint32_t)((st & 1) * kMmaStageBytes) + dst[j], src[j] + (size_t)st * (kMmaStageK * 2));
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[8][4];
#pragma unroll
    for (int t = 0; t < 8; ++t) { acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.0f; }
    // matrix-load offsets: A = this warp's 16 input rows; B = weight rows (the MMA's columns), two column tiles per load
    const uint32_t a_off = (uint32_t)((warp * 16 + (lane & 15)) * kMmaPitch + (lane >> 4) * 16);
    const uint32_t b_off = (uint32_t)((kMmaTile + (lane & 7) + (lane >> 4) * 8) * kMmaPitch + ((lane >> 3) & 1) * 16);
    issue(0);
    for (int st = 0; st < stages; ++st) {
        issue(st + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const uint32_t base = smem + (uint32_t)((st & 1) * kMmaStageBytes);
#pragma unroll
        for (int ks = 0; ks < kMmaStageK / 16; ++ks) {
            uint32_t a[4];
            asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                         : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(base + a_off + ks * 32));
#pragma unroll
            for (int t2 = 0; t2 < 4; ++t2) {
                uint32_t b[4];
                asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                             : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(base + b_off + t2 * (16 * kMmaPitch) + ks * 32));
                asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                             : "+f"(acc[2 * t2][0]), "+f"(acc[2 * t2][1]), "+f"(acc[2 * t2][2]), "+f"(acc[2 * t2][3])
                             : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
                asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                             : "+f"(acc[2 * t2 + 1][0]), "+f"(acc[2 * t2 + 1][1]), "+f"(acc[2 * t2 + 1][2]), "+f"(acc[2 * t2 + 1][3])
                             : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[2]), "r"(b[3]));
            }
        }
        __syncthreads();  // every warp has read this stage before the copies of stage st + 2 land in it
    }
    // accumulator layout: rows g and g + 8 of the warp's 16, columns 8 t + 2 t4 + {0, 1}
    const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        const int c = col0 + t * 8 + 2 * t4;
        const int ra = r0 + warp * 16 + g, rb = ra + 8;
        if (ra < rows) {
            if (c < n) out[(size_t)ra * n + c] = bf_round(acc[t][0]);
            if (c + 1 < n) out[(size_t)ra * n + c + 1] = bf_round(acc[t][1]);
        }
        if (rb < rows) {
            if (c < n) out[(size_t)rb * n + c] = bf_round(acc[t][2]);
            if (c + 1 < n) out[(size_t)rb * n + c + 1] = bf_round(acc[t][3]);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Row RMS normalisation (norm.rs:38-82) with the decoder's follow-ups fused:
//   mode 0: out = bf16(x * inverse * scale)
//   mode 1: out = bf16(residual + mode 0)                         (post-norm + residual add)
//   mode 2: out = bf16(mode 1 * scalar)                           (end of a layer: layer scalar)
// row_index gathers input rows (the rows that want logits).  With `next_scale` the block goes on to normalise the row
// that it has just written (mode 0, into next_out): the norm that follows a post-norm needs no launch of its own.
// Bound by the ordered sum, 4 cycles per value.  Dynamic shared memory: width floats.
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) gm_rms_kernel(const bf16_t* in, const int* row_index, int width, float eps,
                                                     const bf16_t* scale, const bf16_t* residual, const bf16_t* scalar,
                                                     int mode, bf16_t* out, const bf16_t* next_scale, bf16_t* next_out) {
    extern __shared__ __align__(16) float squares[];
    __shared__ float slot;
    const int row = blockIdx.x;
    const uint4* x = reinterpret_cast<const uint4*>(in + (size_t)(row_index ? row_index[row] : row) * width);
    const uint4* res = reinterpret_cast<const uint4*>(residual + (mode >= 1 ? (size_t)row * width : 0));
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t)row * width);
    const int chunks = width / 8;
    const float factor = mode == 2 ? bf_load(scalar[0]) : 1.0f;
    for (int pass = 0; pass < (next_scale ? 2 : 1); ++pass) {
        const uint4* sc = reinterpret_cast<const uint4*>(pass ? next_scale : scale);
        if (pass) { x = dst; dst = reinterpret_cast<uint4*>(next_out + (size_t)row * width); }   // a thread reads back what it wrote
        const int how = pass ? 0 : mode;
        // Eight values per thread per trip; everything a trip needs is requested before the sum starts.
        for (int c = threadIdx.x; c < chunks; c += blockDim.x) {
            const uint4 v = x[c];
            float4* to = reinterpret_cast<float4*>(squares + c * 8);
            float f[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] = bf_half(v, e) * bf_half(v, e);
            to[0] = make_float4(f[0], f[1], f[2], f[3]);
            to[1] = make_float4(f[4], f[5], f[6], f[7]);
        }
        const float energy = ordered_energy(squares, width, &slot);
        const float inverse = inverse_root(energy / (float)width + eps);
        for (int c = threadIdx.x; c < chunks; c += blockDim.x) {
            const uint4 v = x[c];
            const uint4 sv = sc ? __ldg(sc + c) : make_uint4(0, 0, 0, 0);
            const uint4 rv = how >= 1 ? res[c] : make_uint4(0, 0, 0, 0);
            uint32_t ow[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                bf16_t pair[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float value = bf_half(v, 2 * j + e) * inverse;
                    if (sc) value *= bf_half(sv, 2 * j + e);
                    bf16_t r = bf_round(value);
                    if (how >= 1) r = bf_round(bf_half(rv, 2 * j + e) + bf_load(r));
                    if (how == 2) r = bf_round(bf_load(r) * factor);
                    pair[e] = r;
                }
                ow[j] = (uint32_t)pair[0] | ((uint32_t)pair[1] << 16);
            }
            dst[c] = make_uint4(ow[0], ow[1], ow[2], ow[3]);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Per-head normalisation, rotary and cache append (decoder.rs:488-530).  One block per (row, head slot):
// slots [0, heads) are queries (scaled norm + rotary -> q buffer), [heads, heads + kv) keys (scaled norm +
// rotary -> key cache at the row's position), the rest values (scale-free norm -> value cache).  Layers
// that do not own their cache launch only the query slots.
// Rotary (rotary.rs:95-140): each product rounds to BF16, the FP32 sum rounds to BF16; cos / sin come
// from the host-built BF16 table of this layer kind, [position][width / 2].
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) gm_head_kernel(const bf16_t* q_in, const bf16_t* k_in, const bf16_t* v_in,
                                                      const bf16_t* q_scale, const bf16_t* k_scale, const int* slot,
                                                      const int* position, const bf16_t* cosine, const bf16_t* sine,
                                                      int heads, int kv_heads, int width, float eps, int context,
                                                      bf16_t* q_out, bf16_t* key_cache, bf16_t* value_cache) {
    __shared__ __align__(16) float squares[512];
    __shared__ float energy_slot;
    __shared__ bf16_t normed[512];
    const int row = blockIdx.x, h = blockIdx.y, half = width / 2, pos = position[row];
    const bf16_t* x;
    const bf16_t* scale = nullptr;
    bf16_t* out;
    bool rotate = true;
    if (h < heads) {
        x = q_in + ((size_t)row * heads + h) * width;
        scale = q_scale;
        out = q_out + ((size_t)row * heads + h) * width;
    } else {
        const int kh = (h - heads) % kv_heads;
        const size_t at = (((size_t)slot[row] * context + pos) * kv_heads + kh) * width;
        if (h < heads + kv_heads) {
            x = k_in + ((size_t)row * kv_heads + kh) * width;
            scale = k_scale;
            out = key_cache + at;
        } else {
            x = v_in + ((size_t)row * kv_heads + kh) * width;
            out = value_cache + at;
            rotate = false;
        }
    }
    for (int i = threadIdx.x; i < width; i += blockDim.x) {
        const float v = bf_load(x[i]);
        squares[i] = v * v;
    }
    const float energy = ordered_energy(squares, width, &energy_slot);
    const float inverse = inverse_root(energy / (float)width + eps);
    for (int i = threadIdx.x; i < width; i += blockDim.x) {
        float v = bf_load(x[i]) * inverse;
        if (scale) v *= bf_load(scale[i]);
        const bf16_t r = bf_round(v);
        if (rotate) normed[i] = r; else out[i] = r;
    }
    if (!rotate) return;
    __syncthreads();
    const bf16_t* c = cosine + (size_t)pos * half;
    const bf16_t* s = sine + (size_t)pos * half;
    for (int j = threadIdx.x; j < half; j += blockDim.x) {
        const float a = bf_load(normed[j]), b = bf_load(normed[j + half]);
        const float cj = bf_load(c[j]), sj = bf_load(s[j]);
        const float first = bf_load(bf_round(a * cj)) + bf_load(bf_round(-b * sj));
        const float second = bf_load(bf_round(b * cj)) + bf_load(bf_round(a * sj));
        out[j] = bf_round(first);
        out[j + half] = bf_round(second);
    }
}

// ---------------------------------------------------------------------------------------------
// Attention (attention.rs:203-277).  One block per (row, query head).  Keys, then values, pass through two shared
// memory tiles of TILE positions: while a tile is used, cp.async brings the next one (the first values arrive during
// the softmax).  Scores: one thread per key, the dot product in channel order, BF16 rounded, scaling 1.0.  Softmax in
// FP32 with the total added in key order; weights rounded to BF16; the output accumulates weight x value in FP32 over
// the keys in position order, one thread per channel.  window 0 = full attention.
// Bound by chains of dependent additions: the channels of a score once per tile, the keys of the total and of the
// output.  A step of a few rows takes tiles of 128 positions, so that the scores of 128 keys run side by side; more
// blocks than SMs take 64, which leaves room for three blocks per SM.  Tiles of 64 loaded between barriers, with
// nothing in flight while a tile was used, took 36 us for 331 keys of four rows.
// Dynamic shared memory: one float per visible key (rounded up to 16 bytes), then the tiles.
// ---------------------------------------------------------------------------------------------
constexpr size_t kAttnSmemLimit = 200 * 1024;

__host__ __device__ inline size_t attention_smem_bytes(int tile, int visible, int width) {
    return (((size_t)visible * sizeof(float) + 15) & ~(size_t)15) + 2 * (size_t)tile * ((size_t)width * 2 + 16);
}
// Tiles of 32 positions are for contexts whose scores leave no room for more.
inline int attention_tile(int visible, int width, int blocks, int sms) {
    if (blocks <= sms && attention_smem_bytes(128, visible, width) <= kAttnSmemLimit) return 128;
    return attention_smem_bytes(64, visible, width) <= kAttnSmemLimit ? 64 : 32;
}

// query . key over 8 * chunks channels, in channel order
__device__ __forceinline__ float ordered_dot(const uint4* query, const uint4* key, int chunks) {
    float sum = 0.0f;
    uint4 kv[2] = {key[0], key[min(1, chunks - 1)]}, qq[2] = {query[0], query[min(1, chunks - 1)]};
#pragma unroll 2
    for (int i = 0; i < chunks; i += 2) {   // two chunks read ahead of the two in use
        uint4 next_k[2], next_q[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int at = min(i + 2 + u, chunks - 1);
            next_k[u] = key[at];
            next_q[u] = query[at];
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            if (i + u < chunks) {
#pragma unroll
                for (int e = 0; e < 8; ++e) sum = fma_half(qq[u], kv[u], sum, e);
            }
            kv[u] = next_k[u];
            qq[u] = next_q[u];
        }
    }
    return sum;
}

// The same attention with a cluster of four blocks per (row, head), for steps of so few rows that the blocks still fit
// the GPU once.  Each block scores a quarter of the keys, writes its scores into the shared memory of all four, does
// the softmax (the same in each) and sums a quarter of the channels, whose values it requested at the start.  Against
// one block the keys and values arrive over four SMs and the scores take one pass instead of one per 128 keys.
// Dynamic shared memory: one float per visible key, the block's keys, its quarter of every value row.
constexpr int kAttnCluster = 4;
__host__ __device__ inline size_t attention_split_bytes(int visible, int width) {
    return (((size_t)visible * sizeof(float) + 15) & ~(size_t)15) +
           (size_t)((visible + kAttnCluster - 1) / kAttnCluster) * ((size_t)width * 2 + 16) + (size_t)visible * (width / kAttnCluster * 2 + 16);
}
inline bool attention_splits(int visible, int width, int blocks, int sms) {
    return blocks * kAttnCluster <= sms && width % (8 * kAttnCluster) == 0 && attention_split_bytes(visible, width) <= kAttnSmemLimit;
}

__global__ void __launch_bounds__(256, 1) __cluster_dims__(1, 1, kAttnCluster)
    gm_attention_split_kernel(const bf16_t* q, const int* slot, const int* position, const bf16_t* key_cache, const bf16_t* value_cache,
                              int heads, int kv_heads, int width, int window, int context, bf16_t* out) {
    extern __shared__ __align__(16) unsigned char attention_smem[];
    __shared__ float scratch[8];
    __shared__ float total_slot;
    __shared__ uint4 query[64];  // up to 512 BF16 channels
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // this block runs: its scores can be written
    const int row = blockIdx.x, h = blockIdx.y, rank = blockIdx.z, pos = position[row];
    const int kv_head = h / (heads / kv_heads);
    const int last = pos, first = window > 0 ? max(0, pos - (window - 1)) : 0;
    const int visible = last - first + 1;
    const int share = (visible + kAttnCluster - 1) / kAttnCluster, key0 = rank * share, keys = max(0, min(share, visible - key0));
    float* scores = reinterpret_cast<float*>(attention_smem);
    unsigned char* key_tile = attention_smem + (((size_t)visible * sizeof(float) + 15) & ~(size_t)15);
    const int key_pitch = width * 2 + 16, part = width / kAttnCluster, value_pitch = part * 2 + 16;
    unsigned char* value_tile = key_tile + (size_t)share * key_pitch;
    const size_t stride = (size_t)kv_heads * width;
    const bf16_t* kbase = key_cache + ((size_t)slot[row] * context + first) * stride + (size_t)kv_head * width;
    const bf16_t* vbase = value_cache + ((size_t)slot[row] * context + first) * stride + (size_t)kv_head * width + rank * part;
    const int chunks = width / 8, part_chunks = part / 8;
    const uint32_t key_dst = (uint32_t)__cvta_generic_to_shared(key_tile), value_dst = (uint32_t)__cvta_generic_to_shared(value_tile);
#pragma unroll 4
    for (int key = (int)threadIdx.x / 32; key < keys; key += 8) {
        for (int c = (int)threadIdx.x % 32; c < chunks; c += 32) {
            cp_async16(key_dst + (uint32_t)(key * key_pitch + c * 16), reinterpret_cast<const uint4*>(kbase + (size_t)(key0 + key) * stride) + c);
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll 4
    for (int i = threadIdx.x; i < visible * part_chunks; i += 256) {
        const int key = i / part_chunks, c = i - key * part_chunks;
        cp_async16(value_dst + (uint32_t)(key * value_pitch + c * 16), reinterpret_cast<const uint4*>(vbase + (size_t)key * stride) + c);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int i = threadIdx.x; i < chunks; i += blockDim.x) {
        query[i] = reinterpret_cast<const uint4*>(q + ((size_t)row * heads + h) * width)[i];
    }
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    for (int key = threadIdx.x; key < keys; key += blockDim.x) {
        const float score = bf_load(bf_round(ordered_dot(query, reinterpret_cast<const uint4*>(key_tile + (size_t)key * key_pitch), chunks)));
        const uint32_t own = (uint32_t)__cvta_generic_to_shared(scores + key0 + key);
#pragma unroll
        for (int r = 0; r < kAttnCluster; ++r) {
            uint32_t there;
            asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(own), "r"(r));
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(there), "f"(score) : "memory");
        }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");   // the last access to another block's memory is before it
    float maximum = -INFINITY;
    for (int t = threadIdx.x; t < visible; t += blockDim.x) maximum = fmaxf(maximum, scores[t]);
    maximum = block_max(maximum, scratch);
    for (int t = threadIdx.x; t < visible; t += blockDim.x) scores[t] = (float)exp((double)(scores[t] - maximum));
    __syncthreads();
    if (threadIdx.x == 0) total_slot = ordered_sum(scores, visible);
    __syncthreads();
    const float total = total_slot;
    for (int t = threadIdx.x; t < visible; t += blockDim.x) scores[t] = bf_load(bf_round(scores[t] / total));
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if ((int)threadIdx.x < part) {
        const bf16_t* column = reinterpret_cast<const bf16_t*>(value_tile) + threadIdx.x;
        float acc = 0.0f;
#pragma unroll 16
        for (int t = 0; t < visible; ++t) acc = fmaf(scores[t], bf_load(column[(size_t)t * (value_pitch / 2)]), acc);
        out[((size_t)row * heads + h) * width + rank * part + threadIdx.x] = bf_round(acc);
    }
}

template <int TILE>
__global__ void __launch_bounds__(256, 1) gm_attention_kernel(const bf16_t* q, const int* slot, const int* position,
                                                              const bf16_t* key_cache, const bf16_t* value_cache, int heads,
                                                              int kv_heads, int width, int window, int context, bf16_t* out) {
    extern __shared__ __align__(16) unsigned char attention_smem[];
    __shared__ float scratch[8];
    __shared__ float total_slot;
    __shared__ uint4 query[64];  // up to 512 BF16 channels
    const int row = blockIdx.x, h = blockIdx.y, pos = position[row];
    const int kv_head = h / (heads / kv_heads);
    const int last = pos, first = window > 0 ? max(0, pos - (window - 1)) : 0;
    const int visible = last - first + 1;
    float* scores = reinterpret_cast<float*>(attention_smem);
    unsigned char* tiles = attention_smem + (((size_t)visible * sizeof(float) + 15) & ~(size_t)15);
    const int pitch = width * 2 + 16;
    const size_t stride = (size_t)kv_heads * width;
    const bf16_t* kbase = key_cache + ((size_t)slot[row] * context + first) * stride + (size_t)kv_head * width;
    const bf16_t* vbase = value_cache + ((size_t)slot[row] * context + first) * stride + (size_t)kv_head * width;
    const int chunks = width / 8, steps = (visible + TILE - 1) / TILE;
    // steps 0 .. steps - 1 bring the keys, the next as many the values; a warp copies whole positions
    auto copy = [&](int step) {
        if (step < 2 * steps) {
            const int t0 = (step < steps ? step : step - steps) * TILE, count = min(TILE, visible - t0);
            const bf16_t* base = (step < steps ? kbase : vbase) + (size_t)t0 * stride;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(tiles) + (uint32_t)((step & 1) * TILE * pitch);
#pragma unroll 4
            for (int key = (int)threadIdx.x / 32; key < count; key += 8) {
                for (int c = (int)threadIdx.x % 32; c < chunks; c += 32) {
                    cp_async16(dst + (uint32_t)(key * pitch + c * 16), reinterpret_cast<const uint4*>(base + (size_t)key * stride) + c);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // the tile of `step` is in place and the one before it, whose place step + 1 takes, has been used
    auto next_tile = [&](int step) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        copy(step + 1);
        return tiles + (size_t)(step & 1) * TILE * pitch;
    };
    copy(0);
    for (int i = threadIdx.x; i < chunks; i += blockDim.x) {
        query[i] = reinterpret_cast<const uint4*>(q + ((size_t)row * heads + h) * width)[i];
    }
    float maximum = -INFINITY;
    for (int step = 0; step < steps; ++step) {
        const unsigned char* tile = next_tile(step);
        const int t0 = step * TILE;
        if ((int)threadIdx.x < min(TILE, visible - t0)) {
            const float sum = ordered_dot(query, reinterpret_cast<const uint4*>(tile + (size_t)threadIdx.x * pitch), chunks);
            const float score = bf_load(bf_round(sum));
            scores[t0 + threadIdx.x] = score;
            maximum = fmaxf(maximum, score);
        }
    }
    maximum = block_max(maximum, scratch);  // its barriers also order the score writes before the reads below
    for (int t = threadIdx.x; t < visible; t += blockDim.x) scores[t] = (float)exp((double)(scores[t] - maximum));
    __syncthreads();
    if (threadIdx.x == 0) total_slot = ordered_sum(scores, visible);
    __syncthreads();
    const float total = total_slot;
    for (int t = threadIdx.x; t < visible; t += blockDim.x) scores[t] = bf_load(bf_round(scores[t] / total));
    // weight x value, two channels per thread at most (width <= 512)
    float acc[2] = {0.0f, 0.0f};
    for (int step = 0; step < steps; ++step) {
        const unsigned char* tile = next_tile(steps + step);   // its barrier also follows the last write of a weight
        const int t0 = step * TILE, count = min(TILE, visible - t0);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const int c = threadIdx.x + u * 256;
            if (c < width) {
                const bf16_t* column = reinterpret_cast<const bf16_t*>(tile) + c;
#pragma unroll 16
                for (int t = 0; t < count; ++t) acc[u] = fmaf(scores[t0 + t], bf_load(column[(size_t)t * (pitch / 2)]), acc[u]);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int c = threadIdx.x + u * 256;
        if (c < width) out[((size_t)row * heads + h) * width + c] = bf_round(acc[u]);
    }
}

// out = bf16(bf16(gelu(gate)) * other)   (decoder.rs:592-593 and 608-609)
__global__ void gm_gelu_mul_kernel(const bf16_t* gate, const bf16_t* other, size_t n, bf16_t* out) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = bf_round(bf_load(gelu_round(gate[i])) * bf_load(other[i]));
}

// Per-layer inputs (decoder.rs:361-385): projection slice * 1/sqrt(H) (rounded), RMS with the shared
// per-layer norm (rounded), + token identity (rounded), * 2^-1/2 (rounded).  One block per (row, layer);
// out is [layer][row][ple].
__global__ void __launch_bounds__(256) gm_ple_kernel(const bf16_t* projection, const bf16_t* identity, const bf16_t* norm,
                                                     int rows, int ple, int packed, float projection_scale, float eps,
                                                     bf16_t* out) {
    __shared__ __align__(16) float squares[1024];
    __shared__ float energy_slot;
    __shared__ bf16_t scaled[1024];
    const int row = blockIdx.x, layer = blockIdx.y;
    const bf16_t* p = projection + (size_t)row * packed + (size_t)layer * ple;
    const bf16_t* id = identity + (size_t)row * packed + (size_t)layer * ple;
    for (int i = threadIdx.x; i < ple; i += blockDim.x) {
        const bf16_t s = bf_round(bf_load(p[i]) * projection_scale);
        scaled[i] = s;
        const float v = bf_load(s);
        squares[i] = v * v;
    }
    const float energy = ordered_energy(squares, ple, &energy_slot);
    const float inverse = inverse_root(energy / (float)ple + eps);
    for (int i = threadIdx.x; i < ple; i += blockDim.x) {
        float v = bf_load(scaled[i]) * inverse;
        v *= bf_load(norm[i]);
        const bf16_t context = bf_round(v);
        const bf16_t sum = bf_round(bf_load(context) + bf_load(id[i]));
        out[((size_t)layer * rows + row) * ple + i] = bf_round(bf_load(sum) * 0.70710678118654752440f);
    }
}

// Soft cap (elementwise.rs:85-107): divide, tanh, multiply, each rounded.
__global__ void gm_softcap_kernel(bf16_t* logits, size_t n, float cap) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const bf16_t divided = bf_round(__fdiv_rn(bf_load(logits[i]), cap));
    const bf16_t hyperbolic = bf_round((float)tanh((double)bf_load(divided)));
    logits[i] = bf_round(bf_load(hyperbolic) * cap);
}

// Greedy choice (decoder.rs:316-332): the first maximum; a NaN never beats the incumbent, and a NaN in
// element 0 is never replaced.  One block per row.
__global__ void __launch_bounds__(1024) gm_argmax_kernel(const bf16_t* logits, int vocab, uint32_t* out) {
    __shared__ float best_value[32];
    __shared__ int best_index[32];
    const bf16_t* x = logits + (size_t)blockIdx.x * vocab;
    const float head = bf_load(x[0]);
    if (head != head) {  // nothing compares greater than a NaN incumbent
        if (threadIdx.x == 0) out[blockIdx.x] = 0;
        return;
    }
    float value = -INFINITY;
    int index = 0x7fffffff;
    // four 128-bit loads in flight per thread (one value at a time took 20 us for 32,768)
    const int vectors = vocab % 8 == 0 ? vocab / 8 : 0;
#pragma unroll 4
    for (int c = threadIdx.x; c < vectors; c += blockDim.x) {
        const uint4 eight = reinterpret_cast<const uint4*>(x)[c];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float v = bf_half(eight, e);
            if (v > value || (v == value && c * 8 + e < index)) { value = v; index = c * 8 + e; }
        }
    }
    for (int i = vectors * 8 + threadIdx.x; i < vocab; i += blockDim.x) {
        const float v = bf_load(x[i]);
        if (v > value || (v == value && i < index)) { value = v; index = i; }
    }
    // -inf everywhere keeps index 0 (the incumbent), as the sequential scan does
    if (index == 0x7fffffff) index = 0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, value, o);
        const int oi = __shfl_xor_sync(0xffffffffu, index, o);
        if (ov > value || (ov == value && oi < index)) { value = ov; index = oi; }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) { best_value[warp] = value; best_index[warp] = index; }
    __syncthreads();
    if (warp == 0) {
        const int warps = blockDim.x >> 5;
        value = lane < warps ? best_value[lane] : -INFINITY;
        index = lane < warps ? best_index[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, value, o);
            const int oi = __shfl_xor_sync(0xffffffffu, index, o);
            if (ov > value || (ov == value && oi < index)) { value = ov; index = oi; }
        }
        if (lane == 0) out[blockIdx.x] = (uint32_t)index;
    }
}

// Seeded N(0, sigma) values rounded to BF16 (counter-based: SplitMix64 of (seed, index), Box-Muller).
__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
__global__ void gm_normal_kernel(bf16_t* out, size_t n, uint64_t seed, float sigma) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t r = splitmix64(seed ^ splitmix64(i));
    const float u1 = ((float)(uint32_t)(r >> 40) + 1.0f) * (1.0f / 16777217.0f);
    const float u2 = (float)(uint32_t)((r >> 8) & 0xffffffu) * (1.0f / 16777216.0f);
    out[i] = bf_round(sigma * sqrtf(-2.0f * logf(u1)) * cospif(2.0f * u2));
}
__global__ void gm_fill_kernel(bf16_t* out, size_t n, bf16_t value) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = value;
}

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
enum { G_EMBED, G_PLE_EMBED, G_PLE_PROJ, G_PLE_NORM, G_NORM, G_COUNT };
enum { L_Q, L_K, L_V, L_O, L_QNORM, L_KNORM, L_IN, L_POST_ATTN, L_PRE_FFN, L_POST_FFN, L_GATE, L_UP, L_DOWN, L_PLE_GATE,
       L_PLE_PROJ, L_POST_PLE, L_SCALAR, L_COUNT };
const char* const kGlobalNames[G_COUNT] = {"embed_tokens", "embed_tokens_per_layer", "per_layer_model_projection",
                                           "per_layer_projection_norm", "norm"};
const char* const kLayerNames[L_COUNT] = {"q_proj", "k_proj", "v_proj", "o_proj", "q_norm", "k_norm", "input_layernorm",
                                          "post_attention_layernorm", "pre_feedforward_layernorm",
                                          "post_feedforward_layernorm", "gate_proj", "up_proj", "down_proj",
                                          "per_layer_input_gate", "per_layer_projection", "post_per_layer_input_norm",
                                          "layer_scalar"};

struct Tensor {
    bf16_t* data = nullptr;
    size_t count = 0;
    bool loaded = false;
};

struct Sequence {
    bool open = false;
    uint32_t position = 0;
};

}  // namespace

struct ribn_b200_gemma {
    ribn_b200_gemma_config cfg;
    int owner[RIBN_B200_GEMMA_MAX_LAYERS];
    int cache_of[RIBN_B200_GEMMA_MAX_LAYERS];  // owner layer -> index of its cache pair, -1 for consumers
    Tensor g[G_COUNT];
    Tensor l[RIBN_B200_GEMMA_MAX_LAYERS][L_COUNT];
    std::vector<bf16_t*> key_cache, value_cache;  // per owner: [max_sequences][context][kv_heads][width]
    bf16_t* cosine[2] = {nullptr, nullptr};       // [kind: 0 sliding, 1 full][context][width / 2]
    bf16_t* sine[2] = {nullptr, nullptr};
    std::vector<Sequence> seq;
    bool finalized = false;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    // per-pass device buffers (rows = max_batch_tokens)
    uint32_t* d_tokens = nullptr;
    int *d_slot = nullptr, *d_position = nullptr, *d_out_rows = nullptr;
    bf16_t *hidden = nullptr, *mid = nullptr, *normed = nullptr, *q = nullptr, *q2 = nullptr, *k = nullptr, *v = nullptr,
           *attended = nullptr, *projected = nullptr, *gate = nullptr, *up = nullptr, *identity = nullptr,
           *projection = nullptr, *per_layer = nullptr, *ple_gate = nullptr, *logits = nullptr;
    uint32_t* d_choice = nullptr;
    // pinned staging
    uint32_t* h_tokens = nullptr;
    int *h_slot = nullptr, *h_position = nullptr, *h_out_rows = nullptr;
    uint32_t* h_choice = nullptr;
    int max_outputs = 0;
    int sms = 1;
    std::string error;
    float last_ms = 0.0f;
    uint32_t last_launches = 0;
    // passes of a recurring shape (rows, outputs, context bucket) replay a captured graph
    struct PassGraph { cudaGraphExec_t exec = nullptr; uint32_t launches = 0; };
    std::map<uint64_t, PassGraph> graphs;
    std::map<uint64_t, int> graph_seen;
};

namespace {

int fail(ribn_b200_gemma* m, int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (m) m->error = buf;
    return code;
}

int width_of(const ribn_b200_gemma_config& c, int layer) { return c.full[layer] ? c.global_head_dim : c.head_dim; }

size_t global_count(const ribn_b200_gemma_config& c, int id) {
    const size_t packed = (size_t)c.layers * c.ple;
    switch (id) {
        case G_EMBED: return (size_t)c.vocab * c.hidden;
        case G_PLE_EMBED: return (size_t)c.ple_vocab * packed;
        case G_PLE_PROJ: return packed * c.hidden;
        case G_PLE_NORM: return (size_t)c.ple;
        default: return (size_t)c.hidden;
    }
}

size_t layer_count(const ribn_b200_gemma_config& c, int layer, int id) {
    const size_t w = (size_t)width_of(c, layer), h = (size_t)c.hidden;
    switch (id) {
        case L_Q: case L_O: return (size_t)c.heads * w * h;
        case L_K: case L_V: return (size_t)c.kv_heads * w * h;
        case L_QNORM: case L_KNORM: return w;
        case L_GATE: case L_UP: case L_DOWN: return (size_t)c.ffn * h;
        case L_PLE_GATE: case L_PLE_PROJ: return (size_t)c.ple * h;
        case L_SCALAR: return 1;
        default: return h;
    }
}

bool is_matrix(int layer_id) {
    switch (layer_id) {
        case L_Q: case L_K: case L_V: case L_O: case L_GATE: case L_UP: case L_DOWN: case L_PLE_GATE: case L_PLE_PROJ: return true;
        default: return false;
    }
}

// name -> tensor slot and the element count the configuration implies; nullptr for an unknown name
Tensor* find_tensor(ribn_b200_gemma* m, const char* name, size_t* expect) {
    for (int i = 0; i < G_COUNT; ++i) {
        if (strcmp(name, kGlobalNames[i]) == 0) { *expect = global_count(m->cfg, i); return &m->g[i]; }
    }
    if (strncmp(name, "layers.", 7) == 0) {
        char* end = nullptr;
        const long layer = strtol(name + 7, &end, 10);
        if (end && *end == '.' && layer >= 0 && layer < m->cfg.layers) {
            for (int i = 0; i < L_COUNT; ++i) {
                if (strcmp(end + 1, kLayerNames[i]) == 0) {
                    const bool kv_only = i == L_K || i == L_V || i == L_KNORM;
                    if (kv_only && m->owner[layer] != (int)layer) return nullptr;  // consumers hold no key / value weights
                    *expect = layer_count(m->cfg, (int)layer, i);
                    return &m->l[layer][i];
                }
            }
        }
    }
    return nullptr;
}

#define GM_CUDA(m, call)                                                                           \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) return fail((m), RIBN_B200_ERROR, "%s: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

template <typename T>
cudaError_t dev_alloc(T** p, size_t count) { return cudaMalloc((void**)p, sizeof(T) * (count ? count : 1)); }

int ensure_tensor(ribn_b200_gemma* m, Tensor* t, size_t count) {
    if (t->data == nullptr) {
        GM_CUDA(m, dev_alloc(&t->data, count));
        t->count = count;
    }
    return RIBN_B200_OK;
}

}  // namespace

extern "C" {

RIBN_B200_API int ribn_b200_gemma_create(const ribn_b200_gemma_config* config, ribn_b200_gemma** out, char* error,
                                         size_t error_capacity) {
    auto refuse = [&](const char* why) {
        if (error && error_capacity) snprintf(error, error_capacity, "%s", why);
        return RIBN_B200_ERROR;
    };
    if (!config || !out) return refuse("null argument");
    const ribn_b200_gemma_config& c = *config;
    if (c.layers <= 0 || c.layers > RIBN_B200_GEMMA_MAX_LAYERS || c.kv_shared < 0 || c.kv_shared >= c.layers) {
        return refuse("layer count or shared-layer count is invalid");
    }
    if (c.hidden <= 0 || c.heads <= 0 || c.kv_heads <= 0 || c.heads % c.kv_heads || c.ffn <= 0 || c.vocab <= 0 ||
        c.ple <= 0 || c.ple_vocab < c.vocab || c.window <= 0 || c.context <= 0 || c.max_sequences <= 0 ||
        c.max_batch_tokens <= 0) {
        return refuse("a model dimension or limit is not positive");
    }
    if (c.hidden % 8 || c.ffn % 8 || c.ple % 8 || c.head_dim % 8 || c.global_head_dim % 8 || c.head_dim > 512 ||
        c.global_head_dim > 512 || c.ple > 1024 || c.hidden > 12288) {
        return refuse("widths must be multiples of 8 (head widths at most 512, per-layer width at most 1024, hidden at most 12288)");
    }
    if (!(c.eps > 0.0f) || !(c.softcap > 0.0f) || !(c.theta_local > 0.0f) || !(c.theta_global > 0.0f)) {
        return refuse("epsilon, soft cap and rotary bases must be positive");
    }
    if (!c.full[c.layers - 1]) return refuse("the last layer must be full attention");
    if (c.context >= (1 << 24)) return refuse("positions must convert to FP32 exactly");
    int devices = 0;
    if (cudaGetDeviceCount(&devices) != cudaSuccess || devices <= 0 || c.device < 0 || c.device >= devices) {
        return refuse("no usable CUDA device (this library has no CPU path)");
    }
    if (cudaSetDevice(c.device) != cudaSuccess) return refuse("cudaSetDevice failed");
    ribn_b200_gemma* m = new ribn_b200_gemma();
    m->cfg = c;
    const int owners = c.layers - c.kv_shared;
    int caches = 0;
    for (int i = 0; i < c.layers; ++i) {
        int owner = i;
        if (i >= owners) {
            owner = -1;
            for (int j = owners - 1; j >= 0; --j) {
                if ((c.full[j] != 0) == (c.full[i] != 0)) { owner = j; break; }
            }
            if (owner < 0) { delete m; return refuse("a shared layer has no owner of its attention kind"); }
        }
        m->owner[i] = owner;
        m->cache_of[i] = owner == i ? caches++ : -1;
    }
    m->seq.resize((size_t)c.max_sequences);
    auto ok = [&](cudaError_t e) { return e == cudaSuccess; };
    const size_t R = (size_t)c.max_batch_tokens, H = (size_t)c.hidden, packed = (size_t)c.layers * c.ple;
    const size_t W = (size_t)(c.head_dim > c.global_head_dim ? c.head_dim : c.global_head_dim);
    m->max_outputs = c.max_sequences < c.max_batch_tokens ? c.max_sequences : c.max_batch_tokens;
    bool good = ok(cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking)) && ok(cudaEventCreate(&m->ev0)) &&
                ok(cudaEventCreate(&m->ev1));
    good = good && ok(dev_alloc(&m->d_tokens, R)) && ok(dev_alloc(&m->d_slot, R)) && ok(dev_alloc(&m->d_position, R)) &&
           ok(dev_alloc(&m->d_out_rows, R)) && ok(dev_alloc(&m->hidden, R * H)) && ok(dev_alloc(&m->mid, R * H)) &&
           ok(dev_alloc(&m->normed, R * H)) && ok(dev_alloc(&m->q, R * c.heads * W)) &&
           ok(dev_alloc(&m->q2, R * c.heads * W)) && ok(dev_alloc(&m->k, R * c.kv_heads * W)) &&
           ok(dev_alloc(&m->v, R * c.kv_heads * W)) && ok(dev_alloc(&m->attended, R * c.heads * W)) &&
           ok(dev_alloc(&m->projected, R * H)) && ok(dev_alloc(&m->gate, R * c.ffn)) && ok(dev_alloc(&m->up, R * c.ffn)) &&
           ok(dev_alloc(&m->identity, R * packed)) && ok(dev_alloc(&m->projection, R * packed)) &&
           ok(dev_alloc(&m->per_layer, R * packed)) && ok(dev_alloc(&m->ple_gate, R * c.ple)) &&
           ok(dev_alloc(&m->logits, (size_t)m->max_outputs * c.vocab)) && ok(dev_alloc(&m->d_choice, (size_t)m->max_outputs));
    good = good && ok(cudaMallocHost((void**)&m->h_tokens, sizeof(uint32_t) * R)) &&
           ok(cudaMallocHost((void**)&m->h_slot, sizeof(int) * R)) && ok(cudaMallocHost((void**)&m->h_position, sizeof(int) * R)) &&
           ok(cudaMallocHost((void**)&m->h_out_rows, sizeof(int) * R)) &&
           ok(cudaMallocHost((void**)&m->h_choice, sizeof(uint32_t) * (size_t)m->max_outputs));
    for (int i = 0; i < c.layers && good; ++i) {
        if (m->cache_of[i] < 0) continue;
        const size_t n = (size_t)c.max_sequences * c.context * c.kv_heads * width_of(c, i);
        bf16_t *kc = nullptr, *vc = nullptr;
        good = ok(dev_alloc(&kc, n)) && ok(dev_alloc(&vc, n));
        m->key_cache.push_back(kc);
        m->value_cache.push_back(vc);
    }
    if (!good) {
        const char* why = cudaGetErrorString(cudaGetLastError());
        if (error && error_capacity) snprintf(error, error_capacity, "device allocation failed: %s", why);
        ribn_b200_gemma_destroy(m);
        return RIBN_B200_ERROR;
    }
    *out = m;
    return RIBN_B200_OK;
}

RIBN_B200_API int ribn_b200_gemma_destroy(ribn_b200_gemma* m) {
    if (!m) return RIBN_B200_OK;
    if (m->stream) cudaStreamSynchronize(m->stream);
    for (auto& g : m->graphs) cudaGraphExecDestroy(g.second.exec);
    for (auto& t : m->g) cudaFree(t.data);
    for (auto& layer : m->l) for (auto& t : layer) cudaFree(t.data);
    for (bf16_t* p : m->key_cache) cudaFree(p);
    for (bf16_t* p : m->value_cache) cudaFree(p);
    for (int i = 0; i < 2; ++i) { cudaFree(m->cosine[i]); cudaFree(m->sine[i]); }
    void* dev[] = {m->d_tokens, m->d_slot, m->d_position, m->d_out_rows, m->hidden, m->mid, m->normed, m->q, m->q2, m->k,
                   m->v, m->attended, m->projected, m->gate, m->up, m->identity, m->projection, m->per_layer, m->ple_gate,
                   m->logits, m->d_choice};
    for (void* p : dev) cudaFree(p);
    void* host[] = {m->h_tokens, m->h_slot, m->h_position, m->h_out_rows, m->h_choice};
    for (void* p : host) if (p) cudaFreeHost(p);
    if (m->ev0) cudaEventDestroy(m->ev0);
    if (m->ev1) cudaEventDestroy(m->ev1);
    if (m->stream) cudaStreamDestroy(m->stream);
    delete m;
    return RIBN_B200_OK;
}

RIBN_B200_API const char* ribn_b200_gemma_last_error(const ribn_b200_gemma* m) { return m ? m->error.c_str() : "null model"; }

RIBN_B200_API int ribn_b200_gemma_load_tensor(ribn_b200_gemma* m, const char* name, const uint16_t* values, size_t count) {
    if (!m || !name || !values) return RIBN_B200_ERROR;
    if (m->finalized) return fail(m, RIBN_B200_ERROR, "tensors cannot change after finalize");
    size_t expect = 0;
    Tensor* t = find_tensor(m, name, &expect);
    if (!t) return fail(m, RIBN_B200_ERROR, "unknown tensor name '%s'", name);
    if (count != expect) return fail(m, RIBN_B200_ERROR, "tensor '%s' has %zu elements, the configuration implies %zu", name, count, expect);
    if (int rc = ensure_tensor(m, t, expect)) return rc;
    GM_CUDA(m, cudaMemcpy(t->data, values, sizeof(bf16_t) * count, cudaMemcpyHostToDevice));
    t->loaded = true;
    return RIBN_B200_OK;
}

RIBN_B200_API int ribn_b200_gemma_init_synthetic(ribn_b200_gemma* m, uint64_t seed) {
    if (!m) return RIBN_B200_ERROR;
    if (m->finalized) return fail(m, RIBN_B200_ERROR, "tensors cannot change after finalize");
    uint64_t index = 0;
    auto fill = [&](Tensor* t, size_t count, bool matrix) -> int {
        if (int rc = ensure_tensor(m, t, count)) return rc;
        const unsigned blocks = (unsigned)((count + 255) / 256);
        if (matrix) gm_normal_kernel<<<blocks, 256, 0, m->stream>>>(t->data, count, seed * 0x100000001B3ull + (++index) * 0x9E3779B97F4A7C15ull, 0.02f);
        else gm_fill_kernel<<<blocks, 256, 0, m->stream>>>(t->data, count, (bf16_t)0x3f80);
        t->loaded = true;
        return RIBN_B200_OK;
    };
    for (int i = 0; i < G_COUNT; ++i) {
        if (int rc = fill(&m->g[i], global_count(m->cfg, i), i == G_EMBED || i == G_PLE_EMBED || i == G_PLE_PROJ)) return rc;
    }
    for (int l = 0; l < m->cfg.layers; ++l) {
        for (int i = 0; i < L_COUNT; ++i) {
            const bool kv_only = i == L_K || i == L_V || i == L_KNORM;
            if (kv_only && m->owner[l] != l) continue;
            if (int rc = fill(&m->l[l][i], layer_count(m->cfg, l, i), is_matrix(i))) return rc;
        }
    }
    GM_CUDA(m, cudaStreamSynchronize(m->stream));
    GM_CUDA(m, cudaGetLastError());
    return RIBN_B200_OK;
}

RIBN_B200_API int ribn_b200_gemma_read_tensor(ribn_b200_gemma* m, const char* name, uint16_t* out, size_t capacity,
                                              size_t* count) {
    if (!m || !name) return RIBN_B200_ERROR;
    size_t expect = 0;
    Tensor* t = find_tensor(m, name, &expect);
    if (!t || !t->loaded) return fail(m, RIBN_B200_ERROR, "tensor '%s' is not loaded", name);
    if (count) *count = expect;
    if (!out) return RIBN_B200_OK;
    if (capacity < expect) return fail(m, RIBN_B200_ERROR, "buffer holds %zu elements, '%s' has %zu", capacity, name, expect);
    GM_CUDA(m, cudaMemcpy(out, t->data, sizeof(bf16_t) * expect, cudaMemcpyDeviceToHost));
    return RIBN_B200_OK;
}

RIBN_B200_API int ribn_b200_gemma_finalize(ribn_b200_gemma* m) {
    if (!m) return RIBN_B200_ERROR;
    if (m->finalized) return RIBN_B200_OK;
    const ribn_b200_gemma_config& c = m->cfg;
    for (int i = 0; i < G_COUNT; ++i) {
        if (!m->g[i].loaded) return fail(m, RIBN_B200_ERROR, "missing tensor '%s'", kGlobalNames[i]);
    }
    for (int l = 0; l < c.layers; ++l) {
        for (int i = 0; i < L_COUNT; ++i) {
            const bool kv_only = i == L_K || i == L_V || i == L_KNORM;
            if (kv_only && m->owner[l] != l) continue;
            if (!m->l[l][i].loaded) return fail(m, RIBN_B200_ERROR, "missing tensor 'layers.%d.%s'", l, kLayerNames[i]);
        }
    }
    // Rotary factor tables (rotary.rs:33-93, config.rs:200-247), with the host libm the reference's CPU path uses.
    for (int kind = 0; kind < 2; ++kind) {
        const int width = kind ? c.global_head_dim : c.head_dim, half = width / 2;
        const float theta = kind ? c.theta_global : c.theta_local;
        const int active = kind ? half / 4 : half;
        std::vector<float> frequency((size_t)half, 0.0f);
        for (int p = 0; p < active; ++p) {
            const float exponent = (float)(p * 2) / (float)width;
            frequency[(size_t)p] = 1.0f / powf(theta, exponent);
        }
        std::vector<bf16_t> cs((size_t)c.context * half), sn((size_t)c.context * half);
        for (int pos = 0; pos < c.context; ++pos) {
            for (int p = 0; p < half; ++p) {
                const float phase = (float)pos * frequency[(size_t)p];
                cs[(size_t)pos * half + p] = bf_round(cosf(phase));
                sn[(size_t)pos * half + p] = bf_round(sinf(phase));
            }
        }
        GM_CUDA(m, dev_alloc(&m->cosine[kind], cs.size()));
        GM_CUDA(m, dev_alloc(&m->sine[kind], sn.size()));
        GM_CUDA(m, cudaMemcpy(m->cosine[kind], cs.data(), sizeof(bf16_t) * cs.size(), cudaMemcpyHostToDevice));
        GM_CUDA(m, cudaMemcpy(m->sine[kind], sn.data(), sizeof(bf16_t) * sn.size(), cudaMemcpyHostToDevice));
    }
    {
        GM_CUDA(m, cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, m->cfg.device));
        const cudaFuncAttribute at = cudaFuncAttributeMaxDynamicSharedMemorySize;
        GM_CUDA(m, cudaFuncSetAttribute(gm_project_kernel<ProjectNarrow>, at, ProjectShape<ProjectNarrow>::smem_bytes));
        GM_CUDA(m, cudaFuncSetAttribute(gm_project_kernel<ProjectWide>, at, ProjectShape<ProjectWide>::smem_bytes));
        GM_CUDA(m, cudaFuncSetAttribute(gm_project_kernel<ProjectRows>, at, ProjectShape<ProjectRows>::smem_bytes));
        GM_CUDA(m, cudaFuncSetAttribute(gm_project_kernel<ProjectChunk>, at, ProjectShape<ProjectChunk>::smem_bytes));
    }
    const int widest = c.head_dim > c.global_head_dim ? c.head_dim : c.global_head_dim;
    if (attention_smem_bytes(32, c.context, widest) > kAttnSmemLimit) {
        return fail(m, RIBN_B200_ERROR, "context %d exceeds the attention kernel's score buffer", c.context);
    }
    GM_CUDA(m, cudaFuncSetAttribute(gm_attention_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAttnSmemLimit));
    GM_CUDA(m, cudaFuncSetAttribute(gm_attention_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAttnSmemLimit));
    GM_CUDA(m, cudaFuncSetAttribute(gm_attention_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAttnSmemLimit));
    GM_CUDA(m, cudaFuncSetAttribute(gm_attention_kernel<32>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAttnSmemLimit));
    m->finalized = true;
    return RIBN_B200_OK;
}

}  // extern "C"

namespace {

struct Pass {
    ribn_b200_gemma* m;
    int rows;
    uint32_t launches = 0;

    template <typename... Params, typename... Args>
    void launch(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, Args... args) {
        kernel<<<grid, threads, smem, m->stream>>>(static_cast<Params>(args)...);   // its error is read at the end of the pass
        ++launches;
    }
    void project_many(const bf16_t* in, int n_rows, int k, int count, const bf16_t* const* w,
                      const int* n, bf16_t* const* out) {
        ProjectTargets t{};
        t.count = count;
        for (int i = 0; i < count; ++i) { t.w[i] = w[i]; t.out[i] = out[i]; t.n[i] = n[i]; }
        if ((m->cfg.flags & RIBN_B200_GEMMA_FLAG_TENSOR_CORE_PREFILL) && n_rows >= 16 && k % kMmaStageK == 0) {
            unsigned tile_blocks = 0;
            for (int i = 0; i < count; ++i) {
                t.first_block[i] = (int)tile_blocks;
                tile_blocks += (unsigned)((n[i] + kMmaTile - 1) / kMmaTile);
            }
            gm_project_mma_kernel<<<dim3(tile_blocks, (unsigned)((n_rows + kMmaTile - 1) / kMmaTile)), 128, 0, m->stream>>>(in, nullptr, n_rows, t, k);
            ++launches;
            return;
        }
        switch (project_variant(n, count, n_rows, m->sms)) {
            case 0: launch_project<ProjectChunk>(in, n_rows, t, k); break;
            case 1: launch_project<ProjectRows>(in, n_rows, t, k); break;
            case 2: launch_project<ProjectWide>(in, n_rows, t, k); break;
            default: launch_project<ProjectNarrow>(in, n_rows, t, k); break;
        }
    }
    template <typename V>
    void launch_project(const bf16_t* in, int n_rows, ProjectTargets& t, int k) {
        using S = ProjectShape<V>;
        unsigned col_blocks = 0;
        for (int i = 0; i < t.count; ++i) {
            t.first_block[i] = (int)col_blocks;
            col_blocks += (unsigned)((t.n[i] + S::cols - 1) / S::cols);
        }
        launch(gm_project_kernel<V>, dim3(col_blocks, (unsigned)((n_rows + S::rows - 1) / S::rows)), S::threads, S::smem_bytes, in, n_rows,
               (const ProjectTargets)t, k);
    }
    void project(const bf16_t* in, int n_rows, const bf16_t* w, int n, int k, bf16_t* out) {
        project_many(in, n_rows, k, 1, &w, &n, &out);
    }
    void rms(const bf16_t* in, const int* row_index, int n_rows, int width, const bf16_t* scale, const bf16_t* residual,
             const bf16_t* scalar, int mode, bf16_t* out, const bf16_t* next_scale = nullptr, bf16_t* next_out = nullptr) {
        launch(gm_rms_kernel, dim3((unsigned)n_rows), 256, sizeof(float) * (size_t)width, in, row_index, width, m->cfg.eps, scale, residual,
               scalar, mode, out, next_scale, next_out);
    }
    void gelu_mul(const bf16_t* gate, const bf16_t* other, size_t n, bf16_t* out) {
        launch(gm_gelu_mul_kernel, dim3((unsigned)((n + 255) / 256)), 256, 0, gate, other, n, out);
    }
};

// One pass over `rows` flattened tokens already staged in the model's pinned arrays; n_out of them (their
// indices in h_out_rows) produce logits and a greedy token.
int enqueue_pass(ribn_b200_gemma* m, int rows, int n_out, int max_position, uint32_t* launches) {
    const ribn_b200_gemma_config& c = m->cfg;
    cudaStream_t s = m->stream;
    GM_CUDA(m, cudaMemcpyAsync(m->d_tokens, m->h_tokens, sizeof(uint32_t) * (size_t)rows, cudaMemcpyHostToDevice, s));
    GM_CUDA(m, cudaMemcpyAsync(m->d_slot, m->h_slot, sizeof(int) * (size_t)rows, cudaMemcpyHostToDevice, s));
    GM_CUDA(m, cudaMemcpyAsync(m->d_position, m->h_position, sizeof(int) * (size_t)rows, cudaMemcpyHostToDevice, s));
    if (n_out > 0) GM_CUDA(m, cudaMemcpyAsync(m->d_out_rows, m->h_out_rows, sizeof(int) * (size_t)n_out, cudaMemcpyHostToDevice, s));
    Pass p{m, rows};
    const int H = c.hidden, P = c.ple, packed = c.layers * c.ple;
    // decoder.rs:78-92: the embedding scales are BF16-rounded square roots; the projection scale is plain FP32
    const float embed_scale = bf_load(bf_round(sqrtf((float)H)));
    const float ple_scale = bf_load(bf_round(sqrtf((float)P)));
    const float projection_scale = 1.0f / sqrtf((float)H);
    p.launch(gm_embed_kernel, dim3((unsigned)rows), 256, 0, m->d_tokens, m->g[G_EMBED].data, m->g[G_PLE_EMBED].data, H, packed,
                                                    embed_scale, ple_scale, m->hidden, m->identity);
    p.project(m->hidden, rows, m->g[G_PLE_PROJ].data, packed, H, m->projection);
    p.launch(gm_ple_kernel, dim3((unsigned)rows, (unsigned)c.layers), 256, 0, m->projection, m->identity, m->g[G_PLE_NORM].data, rows,
                                                                           P, packed, projection_scale, c.eps, m->per_layer);
    for (int l = 0; l < c.layers; ++l) {
        Tensor* L = m->l[l];
        const int w = width_of(c, l), kind = c.full[l] ? 1 : 0, owner = m->owner[l], cache = m->cache_of[owner];
        const bool owns = owner == l;
        if (l == 0) p.rms(m->hidden, nullptr, rows, H, L[L_IN].data, nullptr, nullptr, 0, m->normed);   // later layers: with the layer before
        {
            const bf16_t* ws[3] = {L[L_Q].data, L[L_K].data, L[L_V].data};
            const int ns[3] = {c.heads * w, c.kv_heads * w, c.kv_heads * w};
            bf16_t* outs[3] = {m->q, m->k, m->v};
            p.project_many(m->normed, rows, H, owns ? 3 : 1, ws, ns, outs);
        }
        p.launch(gm_head_kernel, dim3((unsigned)rows, (unsigned)(c.heads + (owns ? 2 * c.kv_heads : 0))), 128, 0,
            m->q, m->k, m->v, L[L_QNORM].data, owns ? L[L_KNORM].data : nullptr, m->d_slot, m->d_position, m->cosine[kind],
            m->sine[kind], c.heads, c.kv_heads, w, c.eps, c.context, m->q2, m->key_cache[(size_t)cache],
            m->value_cache[(size_t)cache]);
        const int window = kind ? 0 : c.window;
        const int visible = window > 0 && window < max_position + 1 ? window : max_position + 1;
        const auto attend = [&](auto kernel, dim3 grid, size_t smem) {
            p.launch(kernel, grid, 256, smem, m->q2, m->d_slot, m->d_position, m->key_cache[(size_t)cache], m->value_cache[(size_t)cache],
                     c.heads, c.kv_heads, w, window, c.context, m->attended);
        };
        const dim3 grid((unsigned)rows, (unsigned)c.heads);
        const int tile = attention_tile(visible, w, rows * c.heads, m->sms);
        const size_t smem = attention_smem_bytes(tile, visible, w);
        if (attention_splits(visible, w, rows * c.heads, m->sms)) attend(gm_attention_split_kernel, dim3(grid.x, grid.y, kAttnCluster), attention_split_bytes(visible, w));
        else if (tile == 128) attend(gm_attention_kernel<128>, grid, smem);
        else if (tile == 64) attend(gm_attention_kernel<64>, grid, smem);
        else attend(gm_attention_kernel<32>, grid, smem);
        p.project(m->attended, rows, L[L_O].data, H, c.heads * w, m->projected);
        p.rms(m->projected, nullptr, rows, H, L[L_POST_ATTN].data, m->hidden, nullptr, 1, m->mid, L[L_PRE_FFN].data, m->normed);
        // feed-forward (decoder.rs:570-600)
        {
            const bf16_t* ws[2] = {L[L_GATE].data, L[L_UP].data};
            const int ns[2] = {c.ffn, c.ffn};
            bf16_t* outs[2] = {m->gate, m->up};
            p.project_many(m->normed, rows, H, 2, ws, ns, outs);
        }
        p.gelu_mul(m->gate, m->up, (size_t)rows * c.ffn, m->gate);
        p.project(m->gate, rows, L[L_DOWN].data, H, c.ffn, m->projected);
        p.rms(m->projected, nullptr, rows, H, L[L_POST_FFN].data, m->mid, nullptr, 1, m->hidden);
        // per-layer embedding gate, layer scalar (decoder.rs:602-626)
        p.project(m->hidden, rows, L[L_PLE_GATE].data, P, H, m->ple_gate);
        p.gelu_mul(m->ple_gate, m->per_layer + (size_t)l * rows * P, (size_t)rows * P, m->ple_gate);
        p.project(m->ple_gate, rows, L[L_PLE_PROJ].data, H, P, m->projected);
        p.rms(m->projected, nullptr, rows, H, L[L_POST_PLE].data, m->hidden, L[L_SCALAR].data, 2, m->hidden,
              l + 1 < c.layers ? m->l[l + 1][L_IN].data : nullptr, m->normed);
    }
    if (n_out > 0) {
        // decoder.rs:410-428: final norm, tied head, soft cap; then the greedy choice
        p.rms(m->hidden, m->d_out_rows, n_out, H, m->g[G_NORM].data, nullptr, nullptr, 0, m->normed);
        p.project(m->normed, n_out, m->g[G_EMBED].data, c.vocab, H, m->logits);
        const size_t n = (size_t)n_out * c.vocab;
        p.launch(gm_softcap_kernel, dim3((unsigned)((n + 255) / 256)), 256, 0, m->logits, n, c.softcap);
        p.launch(gm_argmax_kernel, dim3((unsigned)n_out), 1024, 0, m->logits, c.vocab, m->d_choice);
        GM_CUDA(m, cudaMemcpyAsync(m->h_choice, m->d_choice, sizeof(uint32_t) * (size_t)n_out, cudaMemcpyDeviceToHost, s));
    }
    GM_CUDA(m, cudaGetLastError());
    *launches += p.launches;
    return RIBN_B200_OK;
}

// A pass reads its rows (tokens, slots, positions, output rows) from the pinned staging arrays, so passes of one
// shape differ only in data: from the third time a shape (rows, outputs, context bucket of 128) comes up it is
// captured into a CUDA graph, which closes the gaps between its ~100 short launches.
int run_pass(ribn_b200_gemma* m, int rows, int n_out, int max_position, uint32_t* launches) {
    constexpr size_t kMaxPassGraphs = 128;
    const int bucket_end = std::min(((max_position + 1 + 127) / 128) * 128, m->cfg.context);
    const uint64_t key = (uint64_t)rows | ((uint64_t)n_out << 20) | ((uint64_t)bucket_end << 40);
    auto found = m->graphs.find(key);
    if (found == m->graphs.end()) {
        if (++m->graph_seen[key] < 3 || m->graphs.size() >= kMaxPassGraphs) return enqueue_pass(m, rows, n_out, max_position, launches);
        cudaGraph_t graph = nullptr;
        uint32_t captured = 0;
        GM_CUDA(m, cudaStreamBeginCapture(m->stream, cudaStreamCaptureModeThreadLocal));
        const int rc = enqueue_pass(m, rows, n_out, bucket_end - 1, &captured);
        const cudaError_t end = cudaStreamEndCapture(m->stream, &graph);
        if (rc != RIBN_B200_OK) { if (graph) cudaGraphDestroy(graph); return rc; }
        GM_CUDA(m, end);
        ribn_b200_gemma::PassGraph entry;
        entry.launches = captured;
        const cudaError_t inst = cudaGraphInstantiate(&entry.exec, graph, 0);
        cudaGraphDestroy(graph);
        GM_CUDA(m, inst);
        found = m->graphs.emplace(key, entry).first;
    }
    GM_CUDA(m, cudaGraphLaunch(found->second.exec, m->stream));
    *launches += found->second.launches;
    return RIBN_B200_OK;
}

Sequence* find_sequence(ribn_b200_gemma* m, uint64_t id) {
    if (id == 0 || id > m->seq.size() || !m->seq[(size_t)id - 1].open) return nullptr;
    return &m->seq[(size_t)id - 1];
}

}  // namespace

extern "C" {

RIBN_B200_API int ribn_b200_gemma_open(ribn_b200_gemma* m, uint64_t* sequence) {
    if (!m || !sequence) return RIBN_B200_ERROR;
    if (!m->finalized) return fail(m, RIBN_B200_ERROR, "finalize the model before opening a sequence");
    for (size_t i = 0; i < m->seq.size(); ++i) {
        if (!m->seq[i].open) {
            m->seq[i].open = true;
            m->seq[i].position = 0;
            *sequence = (uint64_t)i + 1;
            return RIBN_B200_OK;
        }
    }
    return fail(m, RIBN_B200_DEFERRED, "all %zu sequence slots are open", m->seq.size());
}

RIBN_B200_API int ribn_b200_gemma_close(ribn_b200_gemma* m, uint64_t sequence) {
    if (!m) return RIBN_B200_ERROR;
    if (sequence == 0 || sequence > m->seq.size()) return fail(m, RIBN_B200_ERROR, "unknown sequence %llu", (unsigned long long)sequence);
    // every step call completes its device work before it returns, so nothing is in flight here; idempotent
    m->seq[(size_t)sequence - 1].open = false;
    m->seq[(size_t)sequence - 1].position = 0;
    return RIBN_B200_OK;
}

RIBN_B200_API int ribn_b200_gemma_position(const ribn_b200_gemma* m, uint64_t sequence, uint32_t* position) {
    if (!m || !position || sequence == 0 || sequence > m->seq.size() || !m->seq[(size_t)sequence - 1].open) return RIBN_B200_ERROR;
    *position = m->seq[(size_t)sequence - 1].position;
    return RIBN_B200_OK;
}

RIBN_B200_API int ribn_b200_gemma_step(ribn_b200_gemma* m, const ribn_b200_gemma_row* rows, uint32_t n_rows,
                                       uint32_t* tokens_out, uint16_t* logits_out) {
    if (!m || !rows || n_rows == 0) return m ? fail(m, RIBN_B200_ERROR, "empty step") : RIBN_B200_ERROR;
    if (!m->finalized) return fail(m, RIBN_B200_ERROR, "finalize the model before stepping");
    const ribn_b200_gemma_config& c = m->cfg;
    // Validate everything before any state changes (decoder.rs:139-160: a failed step leaves the continuation as it was).
    size_t total = 0;
    for (uint32_t i = 0; i < n_rows; ++i) {
        const ribn_b200_gemma_row& r = rows[i];
        Sequence* s = find_sequence(m, r.sequence);
        if (!s) return fail(m, RIBN_B200_REJECTED, "row %u: unknown sequence %llu", i, (unsigned long long)r.sequence);
        for (uint32_t j = 0; j < i; ++j) {
            if (rows[j].sequence == r.sequence) return fail(m, RIBN_B200_REJECTED, "row %u: sequence appears twice in one step", i);
        }
        if (r.n_tokens == 0 || !r.tokens || (uint64_t)s->position + r.n_tokens > (uint64_t)c.context) {
            return fail(m, RIBN_B200_REJECTED, "row %u: empty or overlong token chunk", i);
        }
        for (uint32_t t = 0; t < r.n_tokens; ++t) {
            if (r.tokens[t] >= (uint32_t)c.vocab) return fail(m, RIBN_B200_REJECTED, "row %u: token %u outside the vocabulary", i, r.tokens[t]);
        }
        if (r.want_output && !tokens_out) return fail(m, RIBN_B200_ERROR, "row %u wants output but tokens_out is null", i);
        total += r.n_tokens;
    }
    GM_CUDA(m, cudaSetDevice(c.device));
    GM_CUDA(m, cudaEventRecord(m->ev0, m->stream));
    uint32_t launches = 0;
    // Flatten rows into passes of at most max_batch_tokens tokens, in row order.
    uint32_t row = 0, offset = 0;  // next token to stage
    size_t logits_row = 0;         // next slot of logits_out
    std::vector<uint32_t> out_owner;  // pass-local: which step row each output belongs to
    while (row < n_rows) {
        int staged = 0, n_out = 0, max_position = 0;
        out_owner.clear();
        while (row < n_rows && staged < c.max_batch_tokens && n_out < m->max_outputs) {
            const ribn_b200_gemma_row& r = rows[row];
            Sequence* s = find_sequence(m, r.sequence);
            const uint32_t take = std::min<uint32_t>(r.n_tokens - offset, (uint32_t)(c.max_batch_tokens - staged));
            for (uint32_t t = 0; t < take; ++t) {
                m->h_tokens[staged] = r.tokens[offset + t];
                m->h_slot[staged] = (int)(r.sequence - 1);
                m->h_position[staged] = (int)(s->position + offset + t);
                max_position = std::max(max_position, m->h_position[staged]);
                ++staged;
            }
            offset += take;
            if (offset == r.n_tokens) {
                if (r.want_output) {
                    m->h_out_rows[n_out++] = staged - 1;
                    out_owner.push_back(row);
                }
                ++row;
                offset = 0;
            }
        }
        if (int rc = run_pass(m, staged, n_out, max_position, &launches)) return rc;
        GM_CUDA(m, cudaStreamSynchronize(m->stream));
        for (int o = 0; o < n_out; ++o) {
            tokens_out[out_owner[(size_t)o]] = m->h_choice[o];
            if (logits_out) {
                GM_CUDA(m, cudaMemcpy(logits_out + logits_row * (size_t)c.vocab, m->logits + (size_t)o * c.vocab,
                                      sizeof(bf16_t) * (size_t)c.vocab, cudaMemcpyDeviceToHost));
                ++logits_row;
            }
        }
    }
    GM_CUDA(m, cudaEventRecord(m->ev1, m->stream));
    GM_CUDA(m, cudaEventSynchronize(m->ev1));
    cudaEventElapsedTime(&m->last_ms, m->ev0, m->ev1);
    m->last_launches = launches;
    for (uint32_t i = 0; i < n_rows; ++i) find_sequence(m, rows[i].sequence)->position += rows[i].n_tokens;
    (void)total;
    return RIBN_B200_OK;
}

RIBN_B200_API int ribn_b200_gemma_advance_prefill(ribn_b200_gemma* m, uint64_t sequence, const uint32_t* tokens, uint32_t n_tokens) {
    const ribn_b200_gemma_row row = {sequence, tokens, n_tokens, 0};
    return ribn_b200_gemma_step(m, &row, 1, nullptr, nullptr);
}

RIBN_B200_API int ribn_b200_gemma_prefill(ribn_b200_gemma* m, uint64_t sequence, const uint32_t* tokens, uint32_t n_tokens,
                                          uint16_t* logits, uint32_t* token) {
    const ribn_b200_gemma_row row = {sequence, tokens, n_tokens, 1};
    uint32_t choice = 0;
    const int rc = ribn_b200_gemma_step(m, &row, 1, &choice, logits);
    if (rc == RIBN_B200_OK && token) *token = choice;
    return rc;
}

RIBN_B200_API int ribn_b200_gemma_decode(ribn_b200_gemma* m, uint64_t sequence, uint32_t input, uint16_t* logits, uint32_t* token) {
    return ribn_b200_gemma_prefill(m, sequence, &input, 1, logits, token);
}

RIBN_B200_API int ribn_b200_gemma_synchronize(ribn_b200_gemma* m) {
    if (!m) return RIBN_B200_ERROR;
    GM_CUDA(m, cudaStreamSynchronize(m->stream));
    return RIBN_B200_OK;
}

RIBN_B200_API int ribn_b200_gemma_last_step_stats(const ribn_b200_gemma* m, float* milliseconds, uint32_t* launches) {
    if (!m) return RIBN_B200_ERROR;
    if (milliseconds) *milliseconds = m->last_ms;
    if (launches) *launches = m->last_launches;
    return RIBN_B200_OK;
}

}  // extern "C"
