// rf_fft.cu — 2-D FFTs for the diffraction stages.
//
// A 2-D transform of a [batch][h][w] complex64 array is a pass over rows and a pass over the
// rows of the transposed result. A block holds a few rows in shared memory, each thread eight
// elements of one row in registers: three radix-2 levels at a time in Stockham's self-sorting
// order, so data stays in natural order and a row of 512 takes three exchanges instead of nine. The
// butterflies are those of the plain radix-2 decimation in time, operation for operation, and the
// passes come in the order of separate 2-D transforms: gradients through the ghost texture can
// amplify its last bits a thousandfold (the light's are small differences of large terms), so these
// stay what they were. What the callers do before and after transforms happens in the passes: a
// pass loads elements through a program, transforms and stores through the program.
//  * the starburst power spectrum (realflare/api/tasks/starburst.py:45-81): load
//    A * exp(i pi (x^2 + y^2) / (lambda d)), store |F|^2 at the fftshift position;
//  * the ghost texture's fractional Fourier transform (realflare/api/tasks/ghost.py:13-36
//    and realflare/utils/frft.py:20-62, Ozaktas et al. 1996 chirp convolution): three 2-D
//    transforms of the aperture and one of a chirp in six passes, or two and one in four
//    (rf_ghost_frft).
// Rows whose length is a power of two from 8 on are transformed directly; any other length from
// 2 to 4096 runs Bluestein's chirp-z form (Bluestein 1970): with w_m = exp(d pi i m^2 / n),
// X_k = w_k sum_j (x_j w_j) conj(w_{k-j}), a linear convolution evaluated by transforms of a
// power-of-two length M >= 2n - 1; the filter's transform is evaluated once per block.
//
// What bounds it: latency on the small textures (a few microseconds per launch), shared memory and
// the transposing stores on batches. 512 x 512, 16 spectra 161 -> 76 us (both passes); a 256 x 256
// ghost texture 74 -> 45 us in 13 -> 6 launches; 702 x 954 (chirp-z) 759 -> 381 us. (Radix-8
// butterflies and merged passes took 34 and 322 us, with other last bits.)
#include <complex>
#include <math.h>

#include <algorithm>

#include "rf_common.cuh"

namespace rf {
namespace {

constexpr int kMaxN = 4096;

// Complex product with one product of each part rounded and the other fused, fixed here so that the
// results' bits do not depend on how a compiler contracts the expression around: of the imaginary
// part a.y b.x is rounded (kFlip: a.x b.y).
template <bool kFlip = false>
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)),
                       kFlip ? __fmaf_rn(a.y, b.x, __fmul_rn(a.x, b.y)) : __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float square_sum(float x, float y) { return __fmaf_rn(x, x, __fmul_rn(y, y)); }
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y)); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y)); }
// ---------------------------------------------------------------- row transforms
// How rows of length n are transformed: M is the power-of-two length, n itself or the convolution's.
struct RowPlan {
    int n, M, log_m, rows_per_block, threads;
    size_t smem;
};

// lengths the row transforms accept: 2 to 4096, any factorisation
bool fft_length_ok(int n) { return n >= 2 && n <= kMaxN; }

__host__ __device__ constexpr int padded(int i) { return i + (i >> 3); }  // conflict-free strides of 8

// Plan for `rows` rows of length n: enough blocks for the SMs first, then more rows per block (longer
// runs in the transposing stores, shared tables), up to 8 and 512 threads.
RowPlan row_plan(int n, long long rows) {
    RowPlan p;
    p.n = n;
    p.M = 8;
    p.log_m = 3;
    const bool direct = n >= 8 && (n & (n - 1)) == 0;
    while (direct ? p.M < n : p.M < 2 * n - 1) p.M <<= 1, p.log_m++;
    const int per_row = p.M / 8;
    p.rows_per_block = per_row < 32 ? 32 / per_row : 1;  // whole warps
    while (p.rows_per_block < 8 && 2 * p.rows_per_block * per_row <= 512 &&
           rows / (2 * p.rows_per_block) >= 128)
        p.rows_per_block *= 2;
    p.threads = p.rows_per_block * per_row;
    // Threads for the filter alone (k_fft_pass) where all blocks fit the SMs at once with them (64 registers a
    // thread: 1024 threads per SM): what counts there is the way through one block. 128 x 300 40 -> 21 us (24 with
    // a launch per step), 128 x 777 43 -> 25, 300 x 500 41 -> 39. In more blocks they cost occupancy:
    // 702 x 954 112 -> 126 us, 2000 x 1500 414 -> 590.
    const int with_filter = p.threads + per_row;
    if (!direct && per_row >= 32 && with_filter <= 1024 &&
        (rows + p.rows_per_block - 1) / p.rows_per_block <= 152LL * (1024 / with_filter))
        p.threads = with_filter;
    const size_t row = sizeof(float2) * padded(p.M);
    p.smem = row * p.rows_per_block + (direct ? 0 : row) + sizeof(float2) * p.M;
    return p;
}

// Transform of one row of length M by its M / 8 threads: thread t brings elements t + r M / 8 in v;
// the result lies in x (padded), natural order. s: the exponent's sign. tw[k] = exp(-2 pi i k / M).
// Every thread of the block takes part (rows share the barriers; rows of at most 32 threads lie
// within a warp).
template <bool kFlip>
__device__ __forceinline__ void fft_row(float2 v[8], float2* x, const float2* tw, int M, int log_m, int t, float s) {
    const int eighth = M >> 3;
    const bool in_warp = eighth <= 32;
    auto sync = [&]() {
        if (in_warp)
            __syncwarp();
        else
            __syncthreads();
    };
    auto twiddle = [&](int k) {
        const float2 w = tw[k];
        return make_float2(w.x, s < 0.0f ? w.y : -w.y);
    };
    auto butterfly = [](float2& a, float2& b, float2 w) {
        const float2 u = a, c = cmul<kFlip>(b, w);
        a = cadd(u, c);
        b = csub(u, c);
    };
    // At ns, blocks of ns elements are transformed; a level combines elements M / 2 apart, at place k of
    // their blocks, with the twiddle exp(s 2 pi i k / (2 ns)) = tw[k M / (2 ns)].
    int log_ns = 0;
    for (int rest = log_m; rest > 0;) {
        if (log_ns > 0) {
#pragma unroll
            for (int r = 0; r < 8; r++) v[r] = x[padded(t + r * eighth)];
        }
        const int ns = 1 << log_ns, sh = log_m - log_ns;
        if (rest >= 3) {
            const int k = t & (ns - 1);
            {
                const float2 w = twiddle(k << (sh - 1));
#pragma unroll
                for (int r = 0; r < 4; r++) butterfly(v[r], v[r + 4], w);
            }
            {
                const float2 w0 = twiddle(k << (sh - 2)), w1 = twiddle((k + ns) << (sh - 2));
                butterfly(v[0], v[2], w0);
                butterfly(v[1], v[3], w0);
                butterfly(v[4], v[6], w1);
                butterfly(v[5], v[7], w1);
            }
            butterfly(v[0], v[1], twiddle(k << (sh - 3)));
            butterfly(v[4], v[5], twiddle((k + ns) << (sh - 3)));
            butterfly(v[2], v[3], twiddle((k + 2 * ns) << (sh - 3)));
            butterfly(v[6], v[7], twiddle((k + 3 * ns) << (sh - 3)));
            const int d = ((t - k) << 3) + k;
            sync();  // everything is read
            const float2 out[8] = {v[0], v[4], v[2], v[6], v[1], v[5], v[3], v[7]};
#pragma unroll
            for (int r = 0; r < 8; r++) x[padded(d + (r << log_ns))] = out[r];
            log_ns += 3;
            rest -= 3;
        } else if (rest == 2) {  // two levels of two groups: elements t + (q + 2 r) M / 8, r = 0 .. 3
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int k = (t + q * eighth) & (ns - 1);
                const float2 w = twiddle(k << (sh - 1));
                butterfly(v[q], v[q + 4], w);
                butterfly(v[q + 2], v[q + 6], w);
                butterfly(v[q], v[q + 2], twiddle(k << (sh - 2)));
                butterfly(v[q + 4], v[q + 6], twiddle((k + ns) << (sh - 2)));
            }
            sync();
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int j = t + q * eighth, k = j & (ns - 1), d = ((j - k) << 2) + k;
                const float2 out[4] = {v[q], v[q + 4], v[q + 2], v[q + 6]};
#pragma unroll
                for (int r = 0; r < 4; r++) x[padded(d + (r << log_ns))] = out[r];
            }
            log_ns += 2;
            rest = 0;
        } else {  // one level of four groups: elements t + (q + 4 r) M / 8, r = 0, 1
#pragma unroll
            for (int q = 0; q < 4; q++)
                butterfly(v[q], v[q + 4], twiddle(((t + q * eighth) & (ns - 1)) << (sh - 1)));
            sync();
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int j = t + q * eighth, k = j & (ns - 1), d = ((j - k) << 1) + k;
                x[padded(d)] = v[q];
                x[padded(d + ns)] = v[q + 4];
            }
            log_ns += 1;
            rest = 0;
        }
        sync();  // everything is written
    }
}

// exp(d pi i m^2 / n), the phase reduced exactly: m^2 mod 2n (m < n <= 4096)
__device__ __forceinline__ float2 bluestein_chirp(int m, int n, float d) {
    const unsigned r = ((unsigned)m * (unsigned)m) % (2u * (unsigned)n);
    float sn, cs;
    sincospif(d * (float)r / (float)n, &sn, &cs);
    return make_float2(cs, sn);
}

// One pass. Program: float2 load(row, i); float sign(row), the transform's direction (+-1); and
// store(row, i, value).
template <class Program>
__global__ void __launch_bounds__(1024) k_fft_pass(const Program p, int rows, int n, int M, int log_m,
                                                   int rows_per_block) {
    extern __shared__ float2 sm[];
    const bool chirp_z = M != n;
    const int eighth = M >> 3, row_size = padded(M);
    const int g = threadIdx.x / eighth, t = threadIdx.x % eighth;  // the thread's row in the block, and place in it
    float2* x = sm + g * row_size;
    float2* filter = sm + rows_per_block * row_size;          // chirp_z: the filter's transform
    float2* tw = filter + (chirp_z ? row_size : 0);
    const int row0 = blockIdx.x * rows_per_block, row = row0 + g;
    const bool valid = row < rows;
    // A pass may start while the one before it runs (launch_pass): its tables need nothing from it. (Only the
    // first half of the twiddles is read; a pass that builds no more is slower on small textures: 256 x
    // 256 46.5 against 44.8 us, 64 x 64 41.2 against 39.3, larger ones the same.)
    // With the filter, which takes a third of the work, it is let in only at the end of its
    // predecessor, whose blocks it would otherwise slow down (82 x 554: 93 against 83 us).
    if (!chirp_z) cudaTriggerProgrammaticLaunchCompletion();
    for (int k = threadIdx.x; k < M; k += blockDim.x) {
        float sn, cs;
        sincospif(-2.0f * (float)k / (float)M, &sn, &cs);
        tw[k] = make_float2(cs, sn);
    }
    float2 v[8];
    const float s = p.sign(row0);  // (programs keep directions equal within a block)
    // chirp_z: the filter's threads are a group of their own behind the rows' where the block has them, and
    // transform it beside the rows' first transform; elsewhere every group does so before.
    const bool filter_group = g == rows_per_block, apart = blockDim.x > (unsigned)(rows_per_block * eighth);
    if (chirp_z && (filter_group || !apart)) {
        // b_m = conj(w_m) for |m| < n, wrapped
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const int i = t + r * eighth, m = i < n ? i : M - i;
            const float2 w = bluestein_chirp(m, n, s);
            v[r] = m < n ? make_float2(w.x, -w.y) : make_float2(0.0f, 0.0f);
        }
    }
    if (chirp_z && !apart) {
        __syncthreads();
        fft_row<false>(v, x, tw, M, log_m, t, -1.0f);
        if (g == 0)
#pragma unroll
            for (int r = 0; r < 8; r++) {
                const int i = padded(t + r * eighth);
                filter[i] = x[i];
            }
    }
    __syncthreads();
    cudaGridDependencySynchronize();  // the passes before are complete
    const float inv_m = 1.0f / (float)M;
    if (!filter_group) {
#pragma unroll
        for (int r = 0; r < 8; r++) {
            const int i = t + r * eighth;
            v[r] = valid && i < n ? p.load(row, i) : make_float2(0.0f, 0.0f);
            if (chirp_z && i < n) v[r] = cmul(v[r], bluestein_chirp(i, n, s));
        }
    }
    if (chirp_z)
        fft_row<false>(v, x, tw, M, log_m, t, -1.0f);
    else
        fft_row<true>(v, x, tw, M, log_m, t, s);
    if (chirp_z) {
        if (apart && eighth <= 32) __syncthreads();  // (else fft_row ends with one)
        if (!filter_group) {
#pragma unroll
            for (int r = 0; r < 8; r++) {
                const int i = padded(t + r * eighth);
                v[r] = cmul<true>(x[i], filter[i]);
            }
        }
        if (eighth <= 32) __syncwarp();
        // (the filter's threads take part in the barriers of the others' last transform, and overwrite the filter
        // behind its first one)
        if (!filter_group || eighth > 32) fft_row<false>(v, x, tw, M, log_m, t, 1.0f);
    }
    if (chirp_z) cudaTriggerProgrammaticLaunchCompletion();
    __syncthreads();  // every row of the block is transformed
    // consecutive threads store one element of the block's consecutive rows: runs in the
    // transposed result
    const int log_rows = __ffs(rows_per_block) - 1;
    for (int e = threadIdx.x; e < n << log_rows; e += blockDim.x) {
        const int q = e & (rows_per_block - 1), i = e >> log_rows;
        if (row0 + q >= rows) continue;
        const float2 c = sm[q * row_size + padded(i)];
        p.store(row0 + q, i, chirp_z ? cmul<true>(bluestein_chirp(i, n, s), make_float2(c.x * inv_m, c.y * inv_m)) : c);
    }
}

template <class Program>
int launch_pass(const Program& program, long long rows, const RowPlan& plan, cudaStream_t s) {
    if (rows > 0x7fffffff - 64) return RF_ERR_NOT_SUPPORTED;
    auto kernel = k_fft_pass<Program>;
    if (plan.smem > 48 * 1024)
        RF_TRY(cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)plan.smem)));
    const long long blocks = (rows + plan.rows_per_block - 1) / plan.rows_per_block;
    // (the launch latency and the tables overlap the pass before)
    return launch_chained(kernel, (unsigned)blocks, plan.threads, plan.smem, s, program, (int)rows, plan.n, plan.M,
                          plan.log_m, plan.rows_per_block);
}

// rows of a [batch][rows][n] array, transformed and stored transposed ([batch][n][rows]), scaled
struct TransposePass {
    const float2* in;
    float2* out;
    int n, rows;
    float s, scale;
    __device__ float sign(int) const { return s; }
    __device__ float2 load(int row, int i) const { return in[(size_t)row * n + i]; }
    __device__ void store(int row, int i, float2 v) const {
        const unsigned b = (unsigned)row / (unsigned)rows, r = (unsigned)row % (unsigned)rows;
        out[((size_t)b * n + i) * rows + r] = make_float2(v.x * scale, v.y * scale);
    }
};

// 2-D transform of data [batch][h][w] in place (scratch of the same size).
int fft2(float2* data, float2* scratch, int batch, int w, int h, int direction, float scale, cudaStream_t s) {
    const float dir = direction < 0 ? -1.0f : 1.0f;
    const long long rows = (long long)batch * h, cols = (long long)batch * w;
    RF_TRY(launch_pass(TransposePass{data, scratch, w, h, dir, 1.0f}, rows, row_plan(w, rows), s));
    return launch_pass(TransposePass{scratch, data, h, w, dir, scale}, cols, row_plan(h, cols), s);
}

// ---------------------------------------------------------------- starburst spectrum
struct StarburstRows {  // aperture * chirp, batch = wavelength
    const float* aperture;
    float2* out;  // [batch][w][h]
    int w, h;
    float phase_scale[256];  // per batch: 1 / (lambda d); the phase is pi * scale * r^2
    __device__ float sign(int) const { return -1.0f; }
    __device__ float2 load(int row, int i) const {
        const int b = (int)((unsigned)row / (unsigned)h), y = (int)((unsigned)row % (unsigned)h);
        const float x0 = w > 1 ? -1.0f + (float)i * (2.0f / (float)(w - 1)) : -1.0f;
        const float y0 = h > 1 ? -1.0f + (float)y * (2.0f / (float)(h - 1)) : -1.0f;
        const float a = __ldg(aperture + (size_t)y * w + i);
        float s, c;
        sincospif(phase_scale[b] * square_sum(x0, y0), &s, &c);
        return make_float2(a * c, a * s);
    }
    __device__ void store(int row, int i, float2 v) const {
        const unsigned b = (unsigned)row / (unsigned)h, y = (unsigned)row % (unsigned)h;
        out[((size_t)b * w + i) * h + y] = v;
    }
};
struct PowerColumns {  // |v|^2 at the fftshift position of the [batch][h][w] image
    const float2* in;  // [batch][w][h]
    float* out;
    int w, h;
    __device__ float sign(int) const { return -1.0f; }
    __device__ float2 load(int row, int i) const { return in[(size_t)row * h + i]; }
    __device__ void store(int row, int i, float2 v) const {
        const unsigned b = (unsigned)row / (unsigned)w;
        const int x = (int)((unsigned)row % (unsigned)w);
        int ys = i + h / 2, xs = x + w / 2;
        ys -= ys >= h ? h : 0, xs -= xs >= w ? w : 0;
        out[((size_t)b * h + ys) * w + xs] = square_sum(v.x, v.y);
    }
};

// ---------------------------------------------------------------- ghost texture
// chirp(shape) of frft.py:8-17: pi * (a^2 / h + b^2 / w), a/b = fftshift(arange(-n/2, n/2))
__device__ __forceinline__ float2 chirp_value(int y, int x, int w, int h, float c) {
    const int a = y < h / 2 ? y : y - h;
    const int b = x < w / 2 ? x : x - w;
    const float r = (float)(a * a) / (float)h + (float)(b * b) / (float)w;
    float sn, cs;
    sincospif(r * c, &sn, &cs);
    return make_float2(cs, sn);
}
struct FrftArgs {
    int w, h;
    float first;  // the transform before the chirp convolution (normalize() of frft.py): +-1, 0 none
    bool flip;
    float c1, c2, ortho;
    float2 scale;
    float norm;
};
// The first two passes carry two arrays, the aperture's (rows below `split`) and chirp 2's, so that a
// launch holds the work of both; `split` is a multiple of the rows per block. numpy's fftshift
// moves element i to (i + n / 2) mod n: output i reads (i + n - n / 2) mod n.
struct FrftRows1 {  // rows y: of the shifted aperture, times chirp 1 without a first transform; of chirp 2
    FrftArgs f;
    const float* aperture;
    float2 *a, *b;  // out [w][h]
    int split;
    __device__ float sign(int row) const { return row < split && f.first != 0.0f ? f.first : -1.0f; }
    __device__ float2 load(int row, int x) const {
        if (row >= split) return chirp_value((int)(row - split), x, f.w, f.h, f.c2);
        if (row >= f.h) return make_float2(0.0f, 0.0f);
        const int sy = f.flip ? f.h - 1 - row : row, sx = f.flip ? f.w - 1 - x : x;
        const float2 v = make_float2(
            __ldg(aperture + (size_t)((sy + f.h - f.h / 2) % f.h) * f.w + (sx + f.w - f.w / 2) % f.w), 0.0f);
        return f.first != 0.0f ? v : cmul(v, chirp_value(row, x, f.w, f.h, f.c1));
    }
    __device__ void store(int row, int x, float2 v) const {
        if (row >= split)
            b[(size_t)x * f.h + (row - split)] = v;
        else if (row < f.h)
            a[(size_t)x * f.h + row] = v;
    }
};
struct FrftColumns2 {  // columns x of the same; a first transform's result times chirp 1
    FrftArgs f;
    const float2* a;  // [w][h]
    float2* b;        // [w][h], in place
    float2* out;      // [h][w]
    int split;
    __device__ float sign(int row) const { return row < split && f.first != 0.0f ? f.first : -1.0f; }
    __device__ float2 load(int row, int y) const {
        if (row >= split) return b[(size_t)(row - split) * f.h + y];
        return row < f.w ? a[(size_t)row * f.h + y] : make_float2(0.0f, 0.0f);
    }
    __device__ void store(int row, int y, float2 v) const {
        v = make_float2(v.x * f.ortho, v.y * f.ortho);
        if (row >= split)
            b[(size_t)(row - split) * f.h + y] = v;
        else if (row < f.w)
            out[(size_t)y * f.w + row] = f.first != 0.0f ? cmul(v, chirp_value(y, row, f.w, f.h, f.c1)) : v;
    }
};
struct FrftRows3 {  // rows y: the product of the two transforms, transformed back
    FrftArgs f;
    const float2 *a, *b;  // [h][w], [w][h]
    float2* out;          // [w][h]
    __device__ float sign(int) const { return 1.0f; }
    __device__ float2 load(int row, int x) const { return cmul<true>(a[(size_t)row * f.w + x], b[(size_t)x * f.h + row]); }
    __device__ void store(int row, int x, float2 v) const { out[(size_t)x * f.h + row] = v; }
};
struct FrftColumns4 {  // columns x of that; |fftshift(scale * chirp 1 * data)| * norm
    FrftArgs f;
    const float2* a;  // [w][h]
    float* out;
    __device__ float sign(int) const { return 1.0f; }
    __device__ float2 load(int row, int y) const { return a[(size_t)row * f.h + y]; }
    __device__ void store(int row, int y, float2 v) const {
        v = make_float2(v.x * f.ortho, v.y * f.ortho);
        const float2 r = cmul(cmul(f.scale, chirp_value(y, (int)row, f.w, f.h, f.c1)), v);
        int ys = y + f.h / 2, xs = (int)row + f.w / 2;
        ys -= ys >= f.h ? f.h : 0, xs -= xs >= f.w ? f.w : 0;
        out[(size_t)ys * f.w + xs] = sqrtf(square_sum(r.x, r.y)) * f.norm;
    }
};

}  // namespace
}  // namespace rf

extern "C" int rf_fft2(float* data, float* scratch, int32_t batch, int32_t width, int32_t height, int32_t direction,
                       float scale, void* stream) {
    using namespace rf;
    if (!data || !scratch || batch < 1) return RF_ERR_INVALID_ARG;
    if (!fft_length_ok(width) || !fft_length_ok(height)) return RF_ERR_NOT_SUPPORTED;
    return fft2((float2*)data, (float2*)scratch, batch, width, height, direction, scale, (cudaStream_t)stream);
}

extern "C" int rf_starburst_spectrum(const float* aperture, int32_t width, int32_t height, const float* lambdas_mm,
                                     int32_t count, float distance_mm, float* scratch, float* spectrum,
                                     void* stream) {
    using namespace rf;
    if (!aperture || !lambdas_mm || !scratch || !spectrum || count < 1 || count > 256) return RF_ERR_INVALID_ARG;
    if (!fft_length_ok(width) || !fft_length_ok(height)) return RF_ERR_NOT_SUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    float2* buf = (float2*)scratch;
    // phase = pi * (x^2 + y^2) / (lambda d): one factor per wavelength, passed by value
    StarburstRows load;
    load.aperture = aperture;
    load.out = buf;
    load.w = width;
    load.h = height;
    for (int b = 0; b < count; b++) load.phase_scale[b] = (float)(1.0 / ((double)lambdas_mm[b] * (double)distance_mm));
    // rows: aperture * chirp -> transposed; columns: -> |F|^2 at the fftshift position
    const long long rows = (long long)count * height, cols = (long long)count * width;
    RF_TRY(launch_pass(load, rows, row_plan(width, rows), s));
    return launch_pass(PowerColumns{buf, spectrum, width, height}, cols, row_plan(height, cols), s);
}

extern "C" int rf_ghost_frft(const float* aperture, int32_t width, int32_t height, float alpha, float* scratch,
                             float* texture, void* stream) {
    using namespace rf;
    if (!aperture || !scratch || !texture) return RF_ERR_INVALID_ARG;
    if (!fft_length_ok(width) || !fft_length_ok(height)) return RF_ERR_NOT_SUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    const long long n = (long long)width * height;
    float2* S0 = (float2*)scratch;
    float2* S1 = S0 + n;
    float2* S2 = S1 + n;
    FrftArgs f;
    f.w = width;
    f.h = height;
    f.ortho = (float)(1.0 / std::sqrt((double)n));
    // normalize() of frft.py:20-40, in double on the host
    double rel = std::fmod((double)alpha, 4.0);
    if (rel < 0) rel += 4.0;
    double a;
    f.flip = false;
    if (rel < 0.5) {
        a = rel + 1;
        f.first = 1.0f;
    } else if (rel < 1.5) {
        a = rel;
        f.first = 0.0f;
    } else if (rel < 2.5) {
        a = rel - 1;
        f.first = -1.0f;
    } else if (rel < 3.5) {
        a = rel - 2;
        f.first = 0.0f;
        f.flip = true;
    } else {
        a = rel - 3;
        f.first = 1.0f;
    }
    const double phi = a * M_PI / 2.0;
    const double cot = 1.0 / std::tan(phi);
    const double sq = std::sqrt(1.0 + cot * cot);
    const std::complex<double> scale = std::sqrt(std::complex<double>(1.0, -cot)) / std::sqrt((double)n);
    f.c1 = (float)(cot - sq);
    f.c2 = (float)sq;
    f.scale = make_float2((float)scale.real(), (float)scale.imag());
    f.norm = (float)std::sqrt((double)n);  // ghost.py:33-35
    // fft2 = fftn(chirp1 * A); fft1 = fftn(chirp2); A = ifftn(fft1 * fft2)
    const RowPlan by_row = row_plan(width, 2LL * height), by_column = row_plan(height, 2LL * width);
    const long long split1 = (height + by_row.rows_per_block - 1) / by_row.rows_per_block * by_row.rows_per_block;
    const long long split2 = (width + by_column.rows_per_block - 1) / by_column.rows_per_block * by_column.rows_per_block;
    RF_TRY(launch_pass(FrftRows1{f, aperture, S0, S1, (int)split1}, split1 + height, by_row, s));
    RF_TRY(launch_pass(FrftColumns2{f, S0, S1, S2, (int)split2}, split2 + width, by_column, s));
    if (f.first != 0.0f) {  // the first transform is done: the forward one
        RF_TRY(launch_pass(TransposePass{S2, S0, width, height, -1.0f, 1.0f}, height, row_plan(width, height), s));
        RF_TRY(launch_pass(TransposePass{S0, S2, height, width, -1.0f, f.ortho}, width, row_plan(height, width), s));
    }
    RF_TRY(launch_pass(FrftRows3{f, S2, S1, S0}, height, row_plan(width, height), s));
    return launch_pass(FrftColumns4{f, S0, texture}, width, row_plan(height, width), s);
}

// ---------------------------------------------------------------- no-allocation variant
//
// Some callers cannot allocate device memory at render time: a plugin inside a host
// application that owns every device allocation through its own pool (and forbids
// cudaMalloc in its render callback), or a real-time loop that must not allocate after
// start-up because an allocation can synchronise the device and stall a frame. For them,
// rf_ghost_frft_static keeps its scratch in this file-scope device array instead of a
// caller buffer. Every GPU that loads the library holds the array (6 MiB) until the
// process exits; all calls share it.
static __device__ __align__(256) float2 g_ghost_frft_scratch[3 * RF_GHOST_FRFT_STATIC_MAX_PIXELS];

namespace rf {
namespace {
// Device address of the static scratch on the current device. The host-side symbol is
// not a device address; the lookup runs on every call (it is cheap), so a pointer is
// never kept across a device reset, after which the module and its array are reloaded.
int static_scratch(float** out) {
    void* p = nullptr;
    RF_TRY(cuda_status(cudaGetSymbolAddress(&p, g_ghost_frft_scratch)));
    *out = (float*)p;
    return RF_OK;
}
}  // namespace
}  // namespace rf

extern "C" int rf_ghost_frft_static(const float* aperture, int32_t width, int32_t height, float alpha,
                                    float* texture, void* stream) {
    using namespace rf;
    if (!aperture || !texture || width < 1 || height < 1) return RF_ERR_INVALID_ARG;
    if ((long long)width * height > RF_GHOST_FRFT_STATIC_MAX_PIXELS) {
        set_error_text("rf_ghost_frft_static: width * height exceeds RF_GHOST_FRFT_STATIC_MAX_PIXELS (512 x 512)");
        return RF_ERR_INVALID_ARG;
    }
    float* scratch = nullptr;
    RF_TRY(static_scratch(&scratch));
    // every scratch plane is fully written before it is read, so the previous call's
    // contents never need clearing
    return rf_ghost_frft(aperture, width, height, alpha, scratch, texture, stream);
}
