// The operand form of a step's GEMMs (StepOperand), written by the kernel that produces the values.
#pragma once
#include <cuda_fp16.h>
#include <math.h>

#include "gemv.cuh"

namespace ribn {

struct StepStage {
    float tops[16], squares[16];
    uint4 pieces[32][2][8];   // [8-input block][hi, lo][member ^ step % 8]: conflict-free both ways
};

// x / den from a reciprocal r of den: the remainder of x r, which a fused multiply-add gives exactly, times r is folded back
// (P. Markstein, Computation of elementary functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990).  With r
// good to a unit in the last place the result is x / den but for near ties.  An infinite x or den leaves no remainder: x r.
__device__ __forceinline__ float quotient(float x, float den, float r) {
    const float q = x * r, rest = fmaf(-q, den, x);
    return fabsf(rest) < INFINITY ? fmaf(rest, r, q) : q;
}
// 1 / x to a unit in the last place; a result below 2^-126 is zero
__device__ __forceinline__ float reciprocal(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// 2^k, k in [-126, 127]
__device__ __forceinline__ float power2(int k) { return __int_as_float((k + 127) << 23); }

// One block of 512 threads: k tile `kt` (256 values of the row) of the eight members from 8 `eight` on, 64 threads each, four
// neighbouring values per thread: lane t of fragment step s holds inputs 16 s + 4 t .. + 3, so a thread writes its member's 16
// bytes of the step.  `v`: the thread's values (zeros where the member does not exist: `have`), `square`: its share of the row's
// sum of squares.
__device__ __forceinline__ void write_step_operand(const StepOperand& out, int kt, int k_tiles, int eight, bool have, const float4 v, float square, StepStage& stage) {
    const int tid = threadIdx.x, g = tid >> 6, i = tid & 63, lane = tid & 31;
    // the tile's largest magnitude and, for a norm's consumer, its sum of squares, over the member's 64 threads
    float top = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (out.ss != nullptr) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) square += __shfl_xor_sync(0xffffffffu, square, o);
    }
    if (lane == 0) { stage.tops[tid >> 5] = top; stage.squares[tid >> 5] = square; }
    __syncthreads();
    top = fmaxf(stage.tops[2 * g], stage.tops[2 * g + 1]);
    // a power of two that brings the largest value into [512, 1024): sums of 32 such values still fit binary16
    const int biased = (int)(__float_as_uint(top) >> 23);   // top is not negative
    const int e = biased == 255 ? 10 : max(-126, min(126, 136 - biased));
    const float scale = power2(e);
    if (i == 0 && have && out.ss != nullptr) out.ss[(size_t)(eight * 8 + g) * k_tiles + kt] = stage.squares[2 * g] + stage.squares[2 * g + 1];
    // hi and lo of inputs 0, 2 and 1, 3; the sum of what the tensor core will see
    const __half2 h02 = __floats2half2_rn(v.x * scale, v.z * scale), h13 = __floats2half2_rn(v.y * scale, v.w * scale);
    const float2 b02 = __half22float2(h02), b13 = __half22float2(h13);
    const __half2 l02 = __floats2half2_rn(v.x * scale - b02.x, v.z * scale - b02.y), l13 = __floats2half2_rn(v.y * scale - b13.x, v.w * scale - b13.y);
    const float2 r02 = __half22float2(l02), r13 = __half22float2(l13);
    float sum = (((b02.x + r02.x) + (b13.x + r13.x)) + (b02.y + r02.y)) + (b13.y + r13.y);
    auto bits = [](const __half2& x) { return *reinterpret_cast<const uint32_t*>(&x); };
    const int group = eight / out.ng, ng = eight - group * out.ng;
    const int s = i >> 2, t = i & 3;
    const float inv_scale = power2(-e);
    if (out.form != kFragmentForm) {
        const int mp = 8 * out.ng, sum_cols = (mp + 15) / 16 * 16, col = ng * 8 + g;
        const bool wide = out.form == kWideForm;   // 64 rows of a block at a time, and 128 inputs of them
        unsigned char* blk = out.blocks + ((size_t)group * k_tiles + kt) * (1028 * mp + 32 * sum_cols);
        // The eight members' 16-byte pieces of an 8-input block lie side by side: through shared memory, so that a warp's
        // stores are whole 128-byte lines.  stage.pieces[8-input block][hi, lo][member ^ step % 8]: conflict-free both ways.
        {
            uint32_t* at = reinterpret_cast<uint32_t*>(&stage.pieces[2 * s][0][g ^ (s & 7)]) + t;
            at[0] = bits(h02);
            at[32] = bits(l02);
            at[64] = bits(h13);          // the next 8-input block
            at[96] = bits(l13);
        }
        __syncthreads();
        {
            const int kb = tid >> 4, half = (tid >> 3) & 1, member = tid & 7;
            const int c = ng * 8 + member;
            const int at = wide ? (((c >> 6) * 2 + (kb >> 4)) * 2 + half) * 1024 + (kb & 15) * 64 + (c & 63) : (kb * 2 + half) * mp + c;
            *reinterpret_cast<uint4*>(blk + (size_t)at * 16) = stage.pieces[kb][half][member ^ ((kb >> 1) & 7)];
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if ((i & 7) == 0) {
            const __half h = __float2half_rn(sum), l = __float2half_rn(sum - __half2float(h));
            const int cols = wide ? 64 : sum_cols, at = wide ? (col >> 6) * 128 + (col & 63) : col;
            __half* to = reinterpret_cast<__half*>(blk + 1024 * mp + at * 16) + (i >> 3);
            to[0] = h;
            to[8 * cols] = l;
        }
        if (i == 0) reinterpret_cast<float*>(blk + 1024 * mp + 32 * sum_cols)[col] = inv_scale;
        return;
    }
    unsigned char* blk = out.blocks + (((size_t)group * k_tiles + kt) * out.ng + ng) * kFragBlockBytes;
    *reinterpret_cast<uint4*>(blk + s * 512 + (g * 4 + t) * 16) = make_uint4(bits(h02), bits(h13), bits(l02), bits(l13));
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    sum += __shfl_xor_sync(0xffffffffu, sum, 4);
    if ((i & 7) == 0) {
        const int q = i >> 3;
        const __half h = __float2half_rn(sum), l = __float2half_rn(sum - __half2float(h));
        __half* at = reinterpret_cast<__half*>(blk + kFragSumsAt + (g * 4 + (q >> 1)) * 8) + (q & 1);
        at[0] = h;
        at[2] = l;
    }
    if (i == 0) reinterpret_cast<float*>(blk + kFragScaleAt)[g] = inv_scale;
}

}  // namespace ribn
