// rf_common.cuh — shared device helpers and host-side error plumbing of the CUDA library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/realflare_gb300.h"

#define RF_MPI_F 3.14159274101257324f  // OpenCL M_PI_F

namespace rf {

// ---------------------------------------------------------------- host error plumbing
void set_cuda_error(cudaError_t e);
void set_error_text(const char* text);
void count_launch();
// Called after every kernel launch: counts it and reports a launch error.
inline int launch_status() {
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_cuda_error(e);
        return RF_ERR_CUDA;
    }
    return RF_OK;
}
inline int cuda_status(cudaError_t e) {
    if (e != cudaSuccess) {
        set_cuda_error(e);
        return RF_ERR_CUDA;
    }
    return RF_OK;
}
#define RF_TRY(expr)                  \
    do {                              \
        int rf_s_ = (expr);           \
        if (rf_s_ != RF_OK) return rf_s_; \
    } while (0)

inline unsigned blocks_for(long long n, int threads) { return (unsigned)((n + threads - 1) / threads); }

// A chain of small kernels is launched so that a kernel may start while the one before it in the
// stream still runs (programmatic dependent launch): its launch latency is then hidden. Every kernel
// of such a chain calls chain_wait() first, before it touches memory, so each waits for all before it.
template <class... Params, class... Args>
int launch_chained(void (*kernel)(Params...), unsigned grid, int block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchAttribute overlap = {};
    overlap.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    overlap.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &overlap;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return cuda_status(e);
    }
    return launch_status();
}
__device__ __forceinline__ void chain_wait() {
#if __CUDA_ARCH__ >= 900
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
#endif
}
__host__ __device__ inline bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

// The traces: threads of a block, ghost paths a thread may trace at once (rf_trace_core.cuh), and the
// blocks per SM that a launch should have, below which a block takes fewer paths.
constexpr int kTraceThreads = 128;
constexpr int kMaxTracePaths = 16;
constexpr int kTraceBlocksPerSm = 16;
// The largest number of paths a block takes at once, up to kMaxTracePaths, that leaves blocks_wanted
// blocks (ray_blocks per path): more paths share more legs, too few blocks leave SMs idle at the
// end. Limits of 12 / 16 / 20 blocks per SM: 3.9 M rays 0.371 / 0.334 / 0.337 ms, 7.9 M 0.597 / 0.592 /
// 0.596 ms, 72.4 M no difference. Up to 32 paths: 72.4 M rays (276 paths) 5.40 instead of 5.63 ms, but
// 15.1 M (182 paths) 0.939 instead of 0.800 ms. Blocks of 64 and of 256 threads: 72.4 M 5.86 ms.
inline int paths_per_block(long long path_count, long long ray_blocks, long long blocks_wanted) {
    int k = kMaxTracePaths;
    while (k > 1 && (path_count + k - 1) / k * ray_blocks < blocks_wanted) k /= 2;
    return k;
}
// The first path of block b: the paths are shared out evenly (sixteen to each block and the rest to the last, a few
// paths leave the double trace short of warps once the small blocks are done: 49,152 rays per path, 16
// surfaces, 5 paths 1.29 -> 0.88 ms, 17 paths 4.36 -> 2.38 ms; k_trace no difference).
__host__ __device__ inline int first_path(int b, int path_blocks, int path_count) {
    return (int)(((long long)b * path_count + path_blocks - 1) / path_blocks);
}
// paths_per_block for a batch, from its number of rays, and a frame's work items with k paths each.
inline int batch_trace_paths(long long rays, int rays_per_thread) {
    int k = kMaxTracePaths;
    while (k > 1 && rays / ((long long)k * kTraceThreads * rays_per_thread) < 152 * kTraceBlocksPerSm) k /= 2;
    return k;
}
__host__ __device__ inline long long batch_trace_items(const rf_trace_args& t, int k, int rays_per_thread) {
    const long long pairs = (long long)t.wavelength_count * t.grid_count * t.grid_count;
    const int chunk = kTraceThreads * rays_per_thread;
    return ((long long)t.path_count + k - 1) / k * ((pairs + chunk - 1) / chunk);
}

// ---------------------------------------------------------------- batched frames
// The frame owning work unit `unit` of a stage: the last frame whose first unit of that
// stage (first(frame), non-decreasing over the frames) is <= unit. Frames without units
// share their first unit with the next frame, so the last of equal starts owns it.
template <class First>
__device__ __forceinline__ int find_frame(const rf_frame* __restrict__ frames, int F, long long unit, First first) {
    int lo = 0, hi = F - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if ((long long)first(frames[mid]) <= unit) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Two FP32 values in one 64-bit register pair, for the packed FP32 instructions of sm_100 and later (two
// operations per instruction, each rounded as the scalar one).
using f2 = unsigned long long;
__device__ __forceinline__ f2 pk(float lo, float hi) {
    f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float lo2(f2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi2(f2 v) { return __uint_as_float((unsigned)(v >> 32)); }

// Quotient and remainder of a >= 0 by b > 0, in 32 bits where a allows (a 64-bit division takes several
// times as many instructions).
__device__ __forceinline__ void divide(long long a, int b, long long& q, int& r) {
    if (a >> 32 == 0) {
        q = (unsigned)a / (unsigned)b;
        r = (int)((unsigned)a - (unsigned)q * (unsigned)b);
    } else {
        q = a / b;
        r = (int)(a - q * b);
    }
}

// ---------------------------------------------------------------- integer semantics
// float -> int truncating toward zero, saturating, NaN -> 0 (cvt.rzi.s32.f32 semantics,
// the conversion the reference's convert_int2/convert_int4 compile to on NVIDIA GPUs).
__device__ __forceinline__ int32_t cvt_rz_sat(float x) { return __float2int_rz(x); }
__device__ __forceinline__ int32_t wadd(int32_t a, int32_t b) { return (int32_t)((uint32_t)a + (uint32_t)b); }
__device__ __forceinline__ int32_t wsub(int32_t a, int32_t b) { return (int32_t)((uint32_t)a - (uint32_t)b); }
__device__ __forceinline__ int32_t wmul(int32_t a, int32_t b) { return (int32_t)((uint32_t)a * (uint32_t)b); }

// Correctly rounded square root without the range handling of the general operation, which the
// trace's and the noise's operands do not need (both are bound by instruction issue): the hardware
// approximation and one residual correction with fused multiply-adds (P. Markstein, Computation of
// elementary functions on the IBM RISC System/6000 processor, 1990). Compared with the correctly
// rounded instruction for every float in [1, 4): equal; scaling by 4 scales every step exactly while
// the residual does not underflow. x = 0 or in [2^-100, 2^127] (below, where an ulp can be lost, the
// roots of the trace's squared distances are added to or compared with lens radii: no effect); inf
// gives NaN. rcp_rn (rf_trace_core.cuh) is the reciprocal's like.
__device__ __forceinline__ float sqrt_rn(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(fmaxf(x, 1.17549435e-38f)));
    const float s = __fmul_rn(x, y);
    return __fmaf_rn(__fmaf_rn(-s, s, x), __fmul_rn(0.5f, y), s);
}
__device__ __forceinline__ float clampf(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }
__device__ __forceinline__ float smoothstepf(float e0, float e1, float x) {
    float t = clampf((x - e0) / (e1 - e0), 0.0f, 1.0f);
    return t * t * (3.0f - 2.0f * t);
}

// read_imagef with CLK_FILTER_LINEAR | CLK_NORMALIZED_COORDS_TRUE, computed in FP32 from
// the OpenCL specification's formula on a w x h texture of `ch` floats per texel (channel
// c). edge: CLAMP_TO_EDGE, else CLAMP with border 0. Non-finite coordinates give 0.
__device__ __forceinline__ float sample_linear(const float* __restrict__ tex, int w, int h, int ch, int c,
                                               float s, float t, bool edge) {
    float u = s * (float)w - 0.5f, v = t * (float)h - 0.5f;
    if (!isfinite(u) || !isfinite(v)) return 0.0f;
    float fu = floorf(u), fv = floorf(v);
    float a = u - fu, b = v - fv;
    long long i0 = cvt_rz_sat(fu), j0 = cvt_rz_sat(fv);
    long long is[2] = {i0, i0 + 1}, js[2] = {j0, j0 + 1};
    float T[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        long long i = is[k & 1], j = js[k >> 1];
        if (edge) {
            i = i < 0 ? 0 : (i >= w ? w - 1 : i);
            j = j < 0 ? 0 : (j >= h ? h - 1 : j);
            T[k] = __ldg(tex + ((size_t)j * w + i) * ch + c);
        } else {
            T[k] = (i < 0 || i >= w || j < 0 || j >= h) ? 0.0f : __ldg(tex + ((size_t)j * w + i) * ch + c);
        }
    }
    return (1.0f - a) * (1.0f - b) * T[0] + a * (1.0f - b) * T[1] + (1.0f - a) * b * T[2] + a * b * T[3];
}

// xyz_to_ap1 (realflare/api/tasks/cl/color.cl:3-10): the matrix literals are double in OpenCL C, so
// the products and sums are evaluated in double there. Double precision runs at 1/64 of FP32's
// rate here (15 double operations per pixel were 14 % of a starburst's time), so each output is first
// an unevaluated sum of two floats, by error-free products (fused multiply-add) and sums (D. Knuth's
// two-sum), within 2^-44 of the terms' magnitudes. Where every value within 2^-42 of it rounds to the
// same float, that is what the double form rounds to as well; the others (one in some
// 100,000; sums that cancel; magnitudes whose errors could underflow; infinities and NaN) take the
// double form.
__device__ __forceinline__ bool dot_rounded(float x, float y, float z, double cx, double cy, double cz, float& out) {
    const float c[3] = {(float)cx, (float)cy, (float)cz};
    const float l[3] = {(float)(cx - c[0]), (float)(cy - c[1]), (float)(cz - c[2])};
    const float v[3] = {x, y, z};
    float hi = 0.0f, lo = 0.0f, magnitude = 0.0f;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const float p = __fmul_rn(v[k], c[k]);
        const float e = __fmaf_rn(v[k], l[k], __fmaf_rn(v[k], c[k], -p));
        const float s = __fadd_rn(hi, p), b = __fsub_rn(s, hi);
        lo = __fadd_rn(lo, __fadd_rn(e, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, b)), __fsub_rn(p, b))));
        hi = s;
        magnitude += fabsf(p);
    }
    const float d = magnitude * 0x1p-42f;
    out = __fadd_rn(hi, __fsub_rn(lo, d));
    return out == __fadd_rn(hi, __fadd_rn(lo, d)) && (magnitude >= 0x1p-80f || magnitude == 0.0f);
}
__device__ __forceinline__ float4 xyz_to_ap1(float x, float y, float z) {
    float4 o;
    o.w = 0.0f;
    bool ok = dot_rounded(x, y, z, 1.6410233797, -0.3248032942, -0.2364246952, o.x);
    ok = dot_rounded(x, y, z, -0.6636628587, 1.6153315917, 0.0167563477, o.y) && ok;
    ok = dot_rounded(x, y, z, 0.0117218943, -0.0082844420, 0.9883948585, o.z) && ok;
    if (!ok) {
        const double dx = x, dy = y, dz = z;
        o.x = (float)(1.6410233797 * dx + -0.3248032942 * dy + -0.2364246952 * dz);
        o.y = (float)(-0.6636628587 * dx + 1.6153315917 * dy + 0.0167563477 * dz);
        o.z = (float)(0.0117218943 * dx + -0.0082844420 * dy + 0.9883948585 * dz);
    }
    return o;
}

// The n-rook sample offsets of realflare/api/tasks/rasterizing.py:78-87.
__device__ __constant__ static const unsigned char SUB_OFFSETS[15] = {0, 1, 0, 1, 2, 0, 3, 4, 1, 6, 2, 5, 0, 3, 7};

// ---------------------------------------------------------------- batch workspace
// Scratch of rf_bin_tiles_batch and rf_raster_batch (rf_bin.cu): pair rectangles, their blocks'
// entry counts and scan, the entry sort's buffers, the raster's tile order and its queue head.
struct BatchWorkspace {
    unsigned long long* rects;
    uint32_t *sums, *scan_scratch, *keys_a, *keys_b, *vals_tmp, *radix_scratch;
    uint32_t *order_keys, *order_vals, *order_keys_b, *order_vals_b, *queue;
    size_t bytes;
};
BatchWorkspace batch_layout(char* base, const rf_batch_sizes& sizes, long long entry_capacity);
const uint32_t* batch_tile_order(const BatchWorkspace& w, const rf_batch_sizes& sizes);

// ---------------------------------------------------------------- scans / sorting
// Exclusive prefix sum of n uint32 values (in may equal out). scratch: scan_scratch_words(n)
// uint32 words. Values must not overflow 32 bits.
size_t scan_scratch_words(long long n);
int exclusive_scan_u32(const uint32_t* in, uint32_t* out, long long n, uint32_t* scratch, cudaStream_t s);

// Stable LSD radix sort of (key, value) pairs by the low key_bits bits of key.
// keys/vals hold the input; keys_alt/vals_alt are buffers of the same size. On return
// *result_in_alt tells which pair of buffers holds the sorted output.
size_t radix_scratch_words(long long n);
int radix_sort_pairs(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt, long long n,
                     int key_bits, uint32_t* scratch, bool* result_in_alt, cudaStream_t s);

}  // namespace rf
