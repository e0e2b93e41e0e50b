// Around the GEMMs of a step (gemm_frag.cu, gemm_ta.cu, gemm_pf.cu): how their work is dealt out, the tensor maps of the
// packed matrices, and the kernels that finish a split launch's partial sums (residual add, SwiGLU) and write the next
// projection's operand in the same pass.
#include <cuda.h>
#include <cuda_fp16.h>
#include <string.h>

#include <algorithm>
#include <type_traits>

#include "blocks.cuh"
#include "gemv.cuh"
#include "step_operand.cuh"

namespace ribn {

namespace {

// RMSNorm factor of one row from the sums of squares of its k tiles (every lane of the warp gets it).
__device__ __forceinline__ float norm_factor(const float* ss, int tiles, float eps, int lane) {
    float sum = 0.0f;
    for (int i = lane; i < tiles; i += 32) sum += ss[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    return 1.0f / sqrtf(sum / (float)(tiles * kTileCols) + eps);
}

// ---- consumers of partial sums, producers of operands -----------------------------------------------------------

// The parts of outputs n .. n + 3 (inside segment `seg`) of member m: where the first lies, how many there are, and the slots
// of the further ones, counted from the first's worker.
struct Parts { const float* at; int count; const float* slots; };
__device__ __forceinline__ Parts parts_of(const StepFinish& a, int seg, int m, int n) {
    const int unit = a.unit0[seg] + (n >> a.split.unit_shift), group = m / a.split.group_members, item = a.split.item_of(unit, group);
    Parts p{a.partial + (size_t)m * a.total_n + a.n_offset[seg] + n, a.split.parts(item), nullptr};
    if (p.count > 1) {
        p.slots = a.further + a.split.slot_of(group, a.split.first_worker(item)) +
                  ((m - group * a.split.group_members) << a.split.unit_shift) + (n & ((1 << a.split.unit_shift) - 1));
    }
    return p;
}
// Their sum in worker order, `s` holding the first, BATCH at a time in flight.  Prefill-sized launches have one or two parts
// and want threads (two in flight: 40 registers, SwiGLU of 2,048 x 12,288 in 124 us; eight: 199 us), small ones up to a
// dozen and want the round trips back (eight in flight: 3.5 us against 5.4).
template <int BATCH>
__device__ __forceinline__ float4 add_parts(const StepFinish& a, const Parts& p, float4 s) {
    const int slot = a.split.slot_floats();
    for (int i = 1; i < p.count; i += BATCH) {
        float4 v[BATCH];
#pragma unroll
        for (int j = 0; j < BATCH; ++j) v[j] = i + j < p.count ? *reinterpret_cast<const float4*>(p.slots + (i + j) * slot) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int j = 0; j < BATCH; ++j) {
            if (i + j < p.count) { s.x += v[j].x; s.y += v[j].y; s.z += v[j].z; s.w += v[j].w; }
        }
    }
    return s;
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// One block: a k tile of eight members (write_step_operand).  MODE: where the values come from (StepFinishMode).
template <int MODE, int BATCH>
__global__ void __launch_bounds__(512, BATCH > 4 ? 1 : BATCH > 2 ? 2 : 3) step_finish_kernel(const StepFinish a) {
    __shared__ StepStage stage;
    __shared__ float factors[8];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int kt = blockIdx.x, tid = threadIdx.x, g = tid >> 6, i = tid & 63, lane = tid & 31;
    const int m = blockIdx.y * 8 + g, n = kt * kTileCols + 4 * i, k_tiles = gridDim.x, width = k_tiles * kTileCols;
    // What depends on no earlier kernel comes before the wait: where the parts lie (divisions) and the norm's weights.  A
    // prefill-sized launch has other blocks to hide them and no registers to hold them.
    constexpr bool kAhead = MODE == kFinishRows || BATCH > 2;
    Parts p0{}, p1{};
    float4 w = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
    if (kAhead && m < a.members) {
        if (MODE != kFinishRows) p0 = parts_of(a, 0, m, n);
        if (MODE == kFinishSwiGLU) p1 = parts_of(a, 1, m, n);
        if (a.norm_weight != nullptr) w = load4(a.norm_weight + n);
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f), gt = v, up = v;
    float square = 0.0f;
    if (m < a.members) {
        if (MODE == kFinishRows) {
            v = *reinterpret_cast<const float4*>(a.x + (size_t)(a.index ? a.index[m] : m) * width + n);
        } else if (MODE == kFinishResidual) {
            float4* h = reinterpret_cast<float4*>(a.y[0] + (size_t)m * width + n);
            if (!kAhead) p0 = parts_of(a, 0, m, n);
            const float4 before = *h, first = load4(p0.at), s = add_parts<BATCH>(a, p0, first);
            v = make_float4(before.x + s.x, before.y + s.y, before.z + s.z, before.w + s.w);
            *h = v;
        } else {
            if (!kAhead) { p0 = parts_of(a, 0, m, n); p1 = parts_of(a, 1, m, n); }
            const float4 first_g = load4(p0.at), first_u = load4(p1.at);
            if (tid < 32) {
                // the eight members' RMSNorm factors, four lanes each, once for the block: in every warp they were a third of its instructions
                const int row = blockIdx.y * 8 + (lane >> 2);
                float sum = 0.0f;
                if (a.ss != nullptr && row < a.members) for (int j = lane & 3; j < a.split.k_tiles; j += 4) sum += a.ss[(size_t)row * a.split.k_tiles + j];
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                if ((lane & 3) == 0) factors[lane >> 2] = a.ss != nullptr ? 1.0f / sqrtf(sum / (float)(a.split.k_tiles * kTileCols) + a.eps) : 1.0f;
            }
            gt = add_parts<BATCH>(a, p0, first_g);
            up = add_parts<BATCH>(a, p1, first_u);
        }
    }
    if (MODE == kFinishSwiGLU) {
        __syncthreads();
        const float inv = factors[g];
        // silu(x) u, a quarter of x by a quarter of 1 + e^-x: the reciprocal of any finite denominator is a normal number
        auto act = [&](float x, float u) {
            x *= inv;
            const float den = fmaf(expf(-x), 0.25f, 0.25f);
            return quotient(0.25f * x, den, reciprocal(den)) * (u * inv);
        };
        // rows past the last one stay zero; a block without any row has no factors either
        if (m < a.members) v = make_float4(act(gt.x, up.x), act(gt.y, up.y), act(gt.z, up.z), act(gt.w, up.w));
    }
    if (m < a.members) {
        square = fmaf(v.x, v.x, fmaf(v.y, v.y, fmaf(v.z, v.z, v.w * v.w)));
        if (a.norm_weight != nullptr) {
            if (!kAhead) w = load4(a.norm_weight + n);
            v.x *= w.x; v.y *= w.y; v.z *= w.z; v.w *= w.w;
        }
    }
    write_step_operand(a.out, kt, k_tiles, (int)blockIdx.y, m < a.members, v, square, stage);
}

// Plain outputs of a split launch: y = (sum of the parts) x the RMSNorm factor, four values per thread; blockIdx.y = member.
template <int BATCH>
__global__ void __launch_bounds__(256) step_store_kernel(const StepFinish a) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int m = blockIdx.y, lane = threadIdx.x & 31;
    int n = 4 * (int)(blockIdx.x * blockDim.x + threadIdx.x), seg = 0;
    while (seg < a.n_segments && n >= a.n[seg]) { n -= a.n[seg]; ++seg; }
    Parts p{};
    if (seg < a.n_segments) p = parts_of(a, seg, m, n);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const float4 first = seg < a.n_segments ? load4(p.at) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float inv = a.ss != nullptr ? norm_factor(a.ss + (size_t)m * a.split.k_tiles, a.split.k_tiles, a.eps, lane) : 1.0f;
    if (seg >= a.n_segments) return;
    const float4 s = add_parts<BATCH>(a, p, first);
    *reinterpret_cast<float4*>(a.y[seg] + (size_t)m * a.n[seg] + n) = make_float4(s.x * inv, s.y * inv, s.z * inv, s.w * inv);
}

// One block per token: the rotation's factors once for all its heads, then a warp per head, four neighbouring dimensions per
// thread; the next head's first sums are requested under the present one.  (A store of q, k and v and a warp per token and
// head behind it took 15.5 + 16.5 us at 777 tokens of the 0.6B model, 35 + 41 us at 2,048 of the 8B model; this 17 and 34 us,
// with eight or sixteen warps 18 to 19 and 36 to 41 us.)
constexpr int kQkvHead = 128;
template <int WARPS>
__global__ void __launch_bounds__(WARPS * 32) step_qkv_kernel(const StepFinish a, const StepQkv c) {
    __shared__ float4 turn[kQkvHead / 4];   // (cosine, sine) of two neighbouring dimensions
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, heads = c.q_heads + 2 * c.kv_heads;
    if (threadIdx.x < kQkvHead / 2) {   // positions are older than the projection
        const float theta = (float)c.token_pos[t] * c.inv_freq[threadIdx.x];
        reinterpret_cast<float2*>(turn)[threadIdx.x] = make_float2(cosf(theta), sinf(theta));
    }
    const long long slot = c.token_slot[t];
    const float4 wq = load4(c.q_norm + 4 * lane), wk = load4(c.k_norm + 4 * lane);
    auto place = [&](int h) {
        const int seg = h < c.q_heads ? 0 : h < c.q_heads + c.kv_heads ? 1 : 2;
        return parts_of(a, seg, t, (h - (seg == 0 ? 0 : seg == 1 ? c.q_heads : c.q_heads + c.kv_heads)) * kQkvHead + 4 * lane);
    };
    Parts p{};
    if (warp < heads) p = place(warp);
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float4 first = warp < heads ? load4(p.at) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float inv = a.ss != nullptr ? norm_factor(a.ss + (size_t)t * a.split.k_tiles, a.split.k_tiles, a.eps, lane) : 1.0f;
    for (int h = warp; h < heads; h += WARPS) {
        Parts next{};
        float4 next_first = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (h + WARPS < heads) { next = place(h + WARPS); next_first = load4(next.at); }
        float4 x = add_parts<2>(a, p, first);
        x.x *= inv; x.y *= inv; x.z *= inv; x.w *= inv;
        auto append = [&](__half* cache, int head) {
            const __half2 lo = __floats2half2_rn(x.x, x.y), hi = __floats2half2_rn(x.z, x.w);
            *reinterpret_cast<uint2*>(cache + (slot * c.kv_heads + head) * kQkvHead + 4 * lane) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        };
        if (h >= c.q_heads + c.kv_heads) {
            append(c.cache_v, h - c.q_heads - c.kv_heads);
        } else {
            float sum = fmaf(x.x, x.x, fmaf(x.y, x.y, fmaf(x.z, x.z, x.w * x.w)));
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            const float r = 1.0f / sqrtf(sum / (float)kQkvHead + c.eps);
            const float4 w = h < c.q_heads ? wq : wk;
            x.x = x.x * r * w.x; x.y = x.y * r * w.y; x.z = x.z * r * w.z; x.w = x.w * r * w.w;
            // dimension d turns with d + 64, sixteen lanes further
            const float4 o = make_float4(__shfl_xor_sync(0xffffffffu, x.x, 16), __shfl_xor_sync(0xffffffffu, x.y, 16),
                                         __shfl_xor_sync(0xffffffffu, x.z, 16), __shfl_xor_sync(0xffffffffu, x.w, 16));
            const float4 t0 = turn[2 * (lane & 15)], t1 = turn[2 * (lane & 15) + 1];
            auto rotate = [&](float mine, float other, float cosine, float sine) { return lane < 16 ? mine * cosine - other * sine : other * sine + mine * cosine; };
            x = make_float4(rotate(x.x, o.x, t0.x, t0.y), rotate(x.y, o.y, t0.z, t0.w), rotate(x.z, o.z, t1.x, t1.y), rotate(x.w, o.w, t1.z, t1.w));
            if (h < c.q_heads) *reinterpret_cast<float4*>(c.q + ((size_t)t * c.q_heads + h) * kQkvHead + 4 * lane) = x;
            else append(c.cache_k, h - c.q_heads);
        }
        p = next;
        first = next_first;
    }
}

int device_sms() {
    static int counts[kMaxDevices] = {0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 148;
    if (counts[dev] == 0) {
        if (cudaDeviceGetAttribute(&counts[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || counts[dev] <= 0) counts[dev] = 148;
    }
    return counts[dev];
}

template <typename... Params>
cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, int threads, size_t smem, cudaStream_t stream, bool programmatic,
                       const std::common_type_t<Params>&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace

StepShape step_shape(int members, int form) {
    const int eights = (members + 7) / 8;
    if (form == kWideForm) return StepShape{(eights + 15) / 16, 16};
    if (form == kColumnForm) {
        // one group of up to 64 rows: 24, 32, 48 or 64 columns
        return StepShape{1, eights <= 3 ? 3 : eights <= 4 ? 4 : eights <= 6 ? 6 : 8};
    }
    const int groups = (eights + 3) / 4;
    return StepShape{groups, (eights + groups - 1) / groups};
}

namespace {
size_t column_block_bytes(int mp) { return (size_t)1028 * mp + 32 * (size_t)((mp + 15) / 16 * 16); }
}  // namespace

size_t step_operand_bytes(int members, int k, int form) {
    const StepShape s = step_shape(members, form);
    return (size_t)s.groups * (size_t)(k / kTileCols) * (form != kFragmentForm ? column_block_bytes(8 * s.ng) : (size_t)s.ng * kFragBlockBytes);
}

cudaError_t make_tile_map(int type, const unsigned char* packed, long long rows, long long cols, void* host_map) {
    static_assert(sizeof(CUtensorMap) == kTileMapBytes, "tensor map size");
    if (!packable(type, rows, cols) || ((uintptr_t)packed & 15) != 0) return cudaErrorInvalidValue;
    using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static Encode encode = nullptr;
    if (encode == nullptr) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &found);
        if (e != cudaSuccess) return e;
        if (found != cudaDriverEntryPointSuccess || fn == nullptr) return cudaErrorNotSupported;
        encode = (Encode)fn;
    }
    // a tile as lines of 224 (Q6_K) or 256 bytes: box dimensions are limited to 256 elements of 8 bytes
    const cuuint64_t tile = (cuuint64_t)packed_tile_bytes(type), line = type == kQ6_K ? 224 : 256;
    const cuuint64_t k_tiles = (cuuint64_t)(cols / kTileCols), row_tiles = (cuuint64_t)((rows + kTileRows - 1) / kTileRows);
    const cuuint64_t dims[4] = {line / 8, tile / line, k_tiles, row_tiles};
    const cuuint64_t strides[3] = {line, tile, tile * k_tiles};
    const cuuint32_t box[4] = {(cuuint32_t)(line / 8), (cuuint32_t)(tile / line), 1, kUnitTiles}, steps[4] = {1, 1, 1, 1};
    CUtensorMap map;
    const CUresult r = encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 4, (void*)packed, dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    memcpy(host_map, &map, sizeof(map));
    return cudaSuccess;
}

StepSplit step_split(const StepGemm& a, bool whole_items) {
    const StepShape shape = step_shape(a.members, a.form);
    StepSplit s{};
    const int tiles = a.form == kWideForm ? 2 * kUnitTiles : kUnitTiles;
    s.unit_shift = a.form == kWideForm ? 8 : 7;
    s.k_tiles = a.k / kTileCols;
    s.groups = shape.groups;
    s.group_members = shape.ng * 8;
    s.joint_shift = a.form == kWideForm ? 1 : 0;
    s.unit_items = (s.groups + s.joint_shift) >> s.joint_shift;
    for (int i = 0; i < a.n_segments; ++i) s.items += (a.seg[i].row_tiles + tiles - 1) / tiles * s.unit_items;
    if ((unsigned long long)s.items * s.k_tiles * (device_sms() * kFragTeams) >> 32) whole_items = true;
    s.whole = whole_items ? 1 : 0;
    const int workers = a.form == kWideForm ? device_sms() / 2 : device_sms() * (a.form == kFragmentForm ? kFragTeams : 1);
    s.workers = std::min(std::max(1, workers), whole_items ? s.items : s.items * s.k_tiles);
    // With three groups every other item is of one group, 0.62 of the time of those of two, and in rounds every other worker
    // would get the long ones only: all even slots (300 rows, 4 layers of the 8B model: 1.96 -> 1.89 ms; with more groups the
    // shares are like enough, and rounds are faster: 1,047 rows 4.55 against 4.76 ms).
    s.rounds = a.form == kWideForm && s.groups != 3 ? s.items / s.workers : 0;
    if (s.rounds * s.workers == s.items && s.rounds > 0) s.whole = 1;   // nothing is left to deal out evenly
    s.spread = std::max(1, s.whole ? std::min(s.workers, s.even()) : std::min(s.workers, s.even() * s.k_tiles));
    s.even_magic = (uint32_t)std::min<unsigned long long>(0xFFFFFFFFull, (1ull << 32) / (unsigned long long)std::max(1, s.even() * s.k_tiles));
    return s;
}

size_t step_partial_floats(const StepGemm& a) {
    size_t total_n = 0;
    for (int i = 0; i < a.n_segments; ++i) total_n += a.seg[i].n;
    return (size_t)a.members * total_n;
}

size_t step_further_floats(const StepGemm& a) {
    const StepSplit s = step_split(a, false);
    return s.whole ? 0 : s.slot_of((1 << s.joint_shift) - 1, s.spread);
}

cudaError_t launch_step_gemm(cudaStream_t stream, const StepGemm& args, bool programmatic) {
    if (args.members < 1 || args.k % kTileCols != 0 || args.blocks == nullptr) return cudaErrorInvalidValue;
    if (args.epilogue != kStore && args.epilogue != kResidual) return cudaErrorInvalidValue;
    StepGemm a = args;
    int w_bytes = 0;
    a.total_n = 0;
    for (int i = 0; i < a.n_segments; ++i) {
        const int b = packed_tile_bytes(a.seg[i].type);
        if (b == 0 || a.seg[i].map == nullptr) return cudaErrorInvalidValue;
        w_bytes = std::max(w_bytes, kUnitTiles * b);
        a.n_offset[i] = a.total_n;
        a.total_n += a.seg[i].n;
    }
    if (a.total_n <= 0) return cudaSuccess;
    if (a.form == kWideForm) return launch_gemm_pf(stream, a, w_bytes, programmatic);
    return a.form == kColumnForm ? launch_gemm_ta(stream, a, w_bytes, programmatic) : launch_gemm_frag(stream, a, w_bytes, programmatic);
}

namespace {
// The fields that come from a split launch; false where its outputs are not multiples of four.
bool fill_parts(const StepGemm& gemm, StepFinish& a) {
    a.split = step_split(gemm, false);
    a.partial = gemm.partial;
    a.further = gemm.further;
    a.members = gemm.members;
    a.n_segments = gemm.n_segments;
    a.ss = gemm.ss;
    a.eps = gemm.eps;
    int units = 0;
    a.total_n = 0;
    for (int i = 0; i < gemm.n_segments; ++i) {
        a.y[i] = gemm.seg[i].y;
        a.n[i] = gemm.seg[i].n;
        a.unit0[i] = units;
        a.n_offset[i] = a.total_n;
        units += (gemm.seg[i].n + (1 << a.split.unit_shift) - 1) >> a.split.unit_shift;
        a.total_n += gemm.seg[i].n;
        if (gemm.seg[i].n % 4 != 0) return false;
    }
    return true;
}
}  // namespace

cudaError_t launch_step_qkv(cudaStream_t stream, const StepGemm& gemm, const StepQkv& args, bool programmatic) {
    StepFinish a{};
    if (gemm.members < 1 || gemm.n_segments != 3 || gemm.seg[0].n != args.q_heads * kQkvHead || gemm.seg[1].n != args.kv_heads * kQkvHead ||
        gemm.seg[2].n != gemm.seg[1].n || !fill_parts(gemm, a)) {
        return cudaErrorInvalidValue;
    }
    // two blocks per SM or less: the heads side by side (47 tokens, 4 layers of the 8B model: 0.66 ms against 0.71 with four warps)
    if (gemm.members <= 2 * device_sms()) return launch_pdl(step_qkv_kernel<16>, dim3((unsigned)gemm.members), 16 * 32, 0, stream, programmatic, a, args);
    return launch_pdl(step_qkv_kernel<4>, dim3((unsigned)gemm.members), 4 * 32, 0, stream, programmatic, a, args);
}

cudaError_t launch_step_finish(cudaStream_t stream, int mode, const StepGemm* gemm, StepFinish a, int width, bool programmatic) {
    a.n_segments = 0;
    if (gemm != nullptr && !fill_parts(*gemm, a)) return cudaErrorInvalidValue;
    if (a.members < 1) return cudaErrorInvalidValue;
    if (mode == kFinishStore) {
        return launch_pdl(a.members <= kColumnMaxMembers ? step_store_kernel<7> : step_store_kernel<2>, dim3((unsigned)((a.total_n / 4 + 255) / 256), (unsigned)a.members), 256, 0, stream, programmatic, a);
    }
    if (width % kTileCols != 0 || (a.out.form == kColumnForm && a.members > kColumnMaxMembers)) return cudaErrorInvalidValue;
    const StepShape shape = step_shape(a.members, a.out.form);
    a.out.ng = shape.ng;
    const dim3 grid((unsigned)(width / kTileCols), (unsigned)(shape.groups * shape.ng));
    // one block per SM while that is a single wave of blocks, two less deep ones, then three (see add_parts; the middle form: 300
    // tokens of the 0.6B model 3.57 -> 3.46 ms; for all larger launches 1 % slower at 2,048 tokens of the 8B model)
    const unsigned blocks = grid.x * grid.y, sms = (unsigned)device_sms();
    const int deep = blocks <= sms ? 7 : blocks <= 3 * sms ? 4 : 2;
    switch (mode) {
        case kFinishRows: return launch_pdl(step_finish_kernel<kFinishRows, 2>, grid, 512, 0, stream, programmatic, a);
        case kFinishResidual:
            return launch_pdl(deep == 7 ? step_finish_kernel<kFinishResidual, 7> : deep == 4 ? step_finish_kernel<kFinishResidual, 4> : step_finish_kernel<kFinishResidual, 2>,
                              grid, 512, 0, stream, programmatic, a);
        case kFinishSwiGLU:
            return launch_pdl(deep == 7 ? step_finish_kernel<kFinishSwiGLU, 7> : deep == 4 ? step_finish_kernel<kFinishSwiGLU, 4> : step_finish_kernel<kFinishSwiGLU, 2>,
                              grid, 512, 0, stream, programmatic, a);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ribn
