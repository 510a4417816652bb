// rf_image.cu — per-pixel image kernels: the starburst compositor, the aperture masks and
// the flare/starburst composite.
//
// k_starburst follows realflare/api/tasks/cl/starburst.cl:1-87 with noise.cl:1-5 and
// geometry.cl:1-48; k_aperture_shape / k_aperture_dust follow aperture.cl:5-47 / 139-174.
#include <math.h>

#include <cmath>

#include "rf_common.cuh"

namespace rf {
namespace {

// Packed FP32 (f2, rf_common.cuh): two terms in one issue slot.
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__device__ __forceinline__ float fract1(float x) { return fminf(x - floorf(x), 0x1.fffffep-1f); }
// The noise hash's sine. Its arguments x reach 10^6, where sinf takes its slow
// reduction path; here x is reduced by pi/2 with the Cody-Waite method (W. J. Cody and
// W. Waite, Software Manual for the Elementary Functions, 1980) using a three-part split of
// pi/2 (C1 = fl(pi/2), C2 = fl(pi/2 - C1), C3 = fl(pi/2 - C1 - C2), which sum to pi/2 within
// 1e-23, computed in 200-bit arithmetic) and fused multiply-adds, then sin or cos of the
// remainder (|r| <= pi/4 + a rounding) by quadrant. Accurate to a few ulps for |x| < 2^22.
// The sine of a reduced argument r = x - k pi / 2.
__device__ __forceinline__ float sine_of(float r, float k) {
    // (beyond 2^22 k loses bits and r grows, to less than 10^5 for every sample index there is: no
    // case for the slow reduction path, which the compiler then leaves out)
    __builtin_assume(fabsf(r) < 1.0e5f);
    float sr, cr;
    sincosf(r, &sr, &cr);
    const unsigned q = (unsigned)(int)k;
    return __uint_as_float(__float_as_uint((q & 1) ? cr : sr) ^ (q & 2) << 30);
}
// noise(x, y, z) of noise.cl:1-5 at z and z + 1, with the terms in x and y given
__device__ __forceinline__ void noise_at(float xy, float z, float& n0, float& n1) {
    auto both = [](float v) { return pk(v, v); };
    const f2 x = fma2(pk(z, z + 1.0f), both(237.212f), both(xy)), t = mul2(x, both(0x1.45f306p-1f));  // x * 2 / pi
    const float k0 = rintf(lo2(t)), k1 = rintf(hi2(t));
    const f2 k = pk(k0, k1);
    f2 r = fma2(k, both(-0x1.921fb6p+0f), x);
    r = fma2(k, both(0x1.777a5cp-25f), r);
    r = fma2(k, both(0x1.ee59dap-50f), r);
    const f2 v = mul2(pk(sine_of(lo2(r), k0), sine_of(hi2(r), k1)), both(43758.5453f));
    n0 = fract1(lo2(v));
    n1 = fract1(hi2(v));
}
__device__ __forceinline__ float noise3(float x, float y, float z) {
    float n0, n1;
    noise_at(x * 112.9898f + y * 179.233f, z, n0, n1);
    return n0;
}
__device__ __forceinline__ void ndc_of(int px, int py, int w, int h, float& nx, float& ny) {
    nx = 2.0f * ((float)px / (float)(w - 1)) - 1.0f;
    ny = 2.0f * ((float)py / (float)(h - 1)) - 1.0f;
}
__device__ __forceinline__ void rot2(float& x, float& y, float angle) {
    float s, c;
    sincosf(angle, &s, &c);
    const float nx = x * c + y * s, ny = y * c - x * s;
    x = nx;
    y = ny;
}

// Per-sample terms of k_starburst that do not depend on the pixel, tabulated per CTA in
// chunks of kStarburstChunk samples: the light's XYZ weight at the sample's spectral position, the
// spectrum plane's number, the texel scale 0.5 * size / (chromatic scale) per axis, and the
// reciprocal of the chromatic scale.
constexpr int kStarburstChunk = 256;
struct alignas(16) StarburstSample {
    float x, y, z;
    int plane;
    float su, sv, inv_scale, pad;
};

// The sum over samples of light x bilinear spectrum lookup. A position p (in [-1, 1]) divided by the
// chromatic scale lies at texel p * (0.5 * size / scale) + (0.5 * size - 0.5): one fused
// multiply-add per axis instead of a division and four roundings. The first texel of the
// footprint is the nearest integer of the texel coordinate less a half, read from the sum with
// 1.5 * 2^23 (floors and conversions would go to the unit that also serves the jitter's
// noise); coordinates too large for that come out as integers outside every texture with sides
// below 2^22. kWide: a spectrum with a longer side or a plane of 2^31 texels or more, by the general lookup.
//
// What bounds it: instruction issue. 1920 x 1080, 100 samples, 16 spectra, no jitter: 733 -> 280 us
// (310 with scalar coordinates, texel rows and sums instead of packed ones, four samples unrolled instead
// of two; before that, lookups with 64-bit indices and divisions); 1000 samples with jitter 16.1 ->
// 9.8 ms (12.3 with the sines' slow path, their quadrant by three selections and a general square root;
// 10.0 with one hash at a time; the two hashes are most of what is left); 512 x 512 with jitter and
// rotation 434 -> 241 us.
template <bool kJitter, bool kRotate, int kPix, bool kWide = false>
__global__ void __launch_bounds__(256, kPix == 2 ? 4 : 7) k_starburst(const float* __restrict__ spectrum,
                                                   const float* __restrict__ light, rf_starburst_args a,
                                                   float4* __restrict__ image) {
    __shared__ StarburstSample tab[kStarburstChunk];
    // kPix pixels of a column per thread, 16 rows apart: they share the table's loads
    const int x = blockIdx.x * 16 + (threadIdx.x & 15), y = blockIdx.y * (16 * kPix) + (threadIdx.x >> 4);
    const bool inside = x < a.width && y < a.height;  // (every thread takes part in the table fills)
    const int w = a.spectrum_width, h = a.spectrum_height;
    // texel coordinates less a half: see above
    const f2 centre = pk(0.5f * (float)w - 1.0f, 0.5f * (float)h - 1.0f);
    float nx, ny[kPix], hash0[kPix];
#pragma unroll
    for (int k = 0; k < kPix; k++) {
        ndc_of(x, y + 16 * k, a.width, a.height, nx, ny[k]);
        ny[k] = (ny[k] - a.offset[1]) / fmaxf(a.scale[1], 1.17549435e-38f);
        hash0[k] = (float)x * 112.9898f + (float)(y + 16 * k) * 179.233f;
    }
    nx = (nx - a.offset[0]) / fmaxf(a.scale[0], 1.17549435e-38f);
    f2 acc[3] = {0, 0, 0};  // of both pixels
    for (int t0 = 0; t0 < a.samples; t0 += kStarburstChunk) {
        const int n = min(kStarburstChunk, a.samples - t0);
        __syncthreads();  // the previous chunk's table is no longer read
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const int t = t0 + i;
            const float step = (float)t / (float)a.samples;
            // no contraction into an FMA: the spectrum index below rounds this value, and a
            // sample can fall exactly halfway between two spectra
            const float wavelength = __fadd_rn(__fmul_rn(step, (float)(RF_LAMBDA_MAX - RF_LAMBDA_MIN)),
                                               (float)RF_LAMBDA_MIN);
            StarburstSample e;
            // chromatic scale 1 - (1 - lambda / 560) = (390 n + 340 t) / (560 n) for sample t of n
            // (LAMBDA_MID is an int in starburst.cl): integers, so its reciprocal rounds once
            const float inv_scale = (float)a.samples / ((float)RF_LAMBDA_MIN * (float)a.samples +
                                                        (float)(RF_LAMBDA_MAX - RF_LAMBDA_MIN) * (float)t);
            int sidx = 0;
            if (a.spectrum_count > 1) {
                const int k = cvt_rz_sat(floorf(__fadd_rn(__fsub_rn(wavelength, a.lambda_first) / a.lambda_step, 0.5f)));
                sidx = k < 0 ? 0 : (k >= a.spectrum_count ? a.spectrum_count - 1 : k);
            }
            e.plane = sidx;
            e.su = (0.5f * (float)RF_LAMBDA_MID * (float)w) * inv_scale;
            e.sv = (0.5f * (float)RF_LAMBDA_MID * (float)h) * inv_scale;
            e.x = sample_linear(light, RF_SPECTRUM_WIDTH, 1, 4, 0, step, 0.0f, false);
            e.y = sample_linear(light, RF_SPECTRUM_WIDTH, 1, 4, 1, step, 0.0f, false);
            e.z = sample_linear(light, RF_SPECTRUM_WIDTH, 1, 4, 2, step, 0.0f, false);
            e.inv_scale = (float)RF_LAMBDA_MID * inv_scale;
            e.pad = 0.0f;
            tab[i] = e;
        }
        __syncthreads();
        if (!inside) continue;
#pragma unroll 4
        for (int i = 0; i < n; i++) {
            const float4 e0 = *reinterpret_cast<const float4*>(&tab[i].x);
            const f2 scale = *reinterpret_cast<const f2*>(&tab[i].su);
            const float seed = (float)((t0 + i) * 4);
            const float* plane = spectrum + (size_t)(unsigned)__float_as_int(e0.w) * (unsigned)h * w;
            float fi[2] = {0.0f, 0.0f};
#pragma unroll
            for (int k = 0; k < kPix; k++) {
                float px = nx, py = ny[k];
                if (kJitter) {
                    float n0, n1, sa, ca;
                    noise_at(hash0[k], seed, n0, n1);
                    const float radius = a.blur * sqrt_rn(n0);
                    sincospif(2.0f * n1, &sa, &ca);
                    px += ca * radius;
                    py += sa * radius;
                }
                if (kRotate) {  // (the chromatic scale is uniform: it can follow the rotation)
                    float n0, r;
                    noise_at(hash0[k], seed + 2.0f, n0, r);
                    const float sign = n0 > 0.5f ? 1.0f : -1.0f;
                    const float angle = sign * a.rotation * (1.0f - (a.rotation_weight == 1.0f ? r : powf(r, a.rotation_weight)));
                    rot2(px, py, angle);
                }
                if (kWide) {
                    const float k_inv = tab[i].inv_scale;
                    fi[k] = sample_linear(plane, w, h, 1, 0, px * k_inv * 0.5f + 0.5f, py * k_inv * 0.5f + 0.5f, false);
                    continue;
                }
                const f2 big = pk(12582912.0f, 12582912.0f);
                const f2 uv = fma2(pk(px, py), scale, centre), near = add2(uv, big);
                const int i0 = __float_as_int(lo2(near)) - 0x4b400000, j0 = __float_as_int(hi2(near)) - 0x4b400000;
                const f2 frac = add2(sub2(uv, sub2(near, big)), pk(0.5f, 0.5f));
                f2 left = 0, right = 0;  // texels (i0, j0), (i0, j0 + 1); (i0 + 1, ...)
                if ((unsigned)i0 < (unsigned)(w - 1) && (unsigned)j0 < (unsigned)(h - 1)) {
                    const float* q = plane + (j0 * w + i0);
                    left = pk(__ldg(q), __ldg(q + w));
                    right = pk(__ldg(q + 1), __ldg(q + w + 1));
                } else {
                    const bool i0_in = (unsigned)i0 < (unsigned)w, i1_in = i0 >= -1 && i0 < w - 1;
                    const bool j0_in = (unsigned)j0 < (unsigned)h, j1_in = j0 >= -1 && j0 < h - 1;
                    if (!((i0_in || i1_in) && (j0_in || j1_in))) continue;  // outside: adds 0
                    const float* q = plane + max(j0, 0) * w;
                    const float* q1 = j0 < 0 ? q : q + w;
                    left = pk(i0_in && j0_in ? __ldg(q + i0) : 0.0f, i0_in && j1_in ? __ldg(q1 + i0) : 0.0f);
                    right = pk(i1_in && j0_in ? __ldg(q + i0 + 1) : 0.0f, i1_in && j1_in ? __ldg(q1 + i0 + 1) : 0.0f);
                }
                const f2 rows = fma2(pk(lo2(frac), lo2(frac)), sub2(right, left), left);
                fi[k] = fmaf(hi2(frac), hi2(rows) - lo2(rows), lo2(rows));
            }
            if (kPix == 1) {
                acc[0] = pk(fmaf(e0.x, fi[0], lo2(acc[0])), 0.0f);
                acc[1] = pk(fmaf(e0.y, fi[0], lo2(acc[1])), 0.0f);
                acc[2] = pk(fmaf(e0.z, fi[0], lo2(acc[2])), 0.0f);
                continue;
            }
            const f2 f = pk(fi[0], fi[1]);
            acc[0] = fma2(pk(e0.x, e0.x), f, acc[0]);
            acc[1] = fma2(pk(e0.y, e0.y), f, acc[1]);
            acc[2] = fma2(pk(e0.z, e0.z), f, acc[2]);
        }
    }
    if (!inside) return;
#pragma unroll
    for (int k = 0; k < kPix; k++) {
        if (y + 16 * k >= a.height) break;
        float v[3];
#pragma unroll
        for (int c = 0; c < 3; c++) v[c] = (k ? hi2(acc[c]) : lo2(acc[c])) / (float)a.samples;
        if (!isnan(a.vignetting[0])) {
            const float sdf = sqrtf(nx * nx + ny[k] * ny[k]) - 0.0f;
            const float f = smoothstepf(a.vignetting[1], a.vignetting[0], sdf);
#pragma unroll
            for (int c = 0; c < 3; c++) v[c] *= f;
        }
#pragma unroll
        for (int c = 0; c < 3; c++) v[c] *= a.intensity;
        image[(size_t)(y + 16 * k) * a.width + x] = xyz_to_ap1(v[0], v[1], v[2]);
    }
}

__global__ void __launch_bounds__(256) k_aperture_shape(float* __restrict__ image, int w, int h, float sx, float sy,
                                                        int blades, float rotation, float roundness, float softness) {
    const int x = blockIdx.x * 16 + (threadIdx.x & 15), y = blockIdx.y * 16 + (threadIdx.x >> 4);
    if (x >= w || y >= h) return;
    float px, py;
    ndc_of(x, y, w, h, px, py);
    px = px / fmaxf(sx, 1.17549435e-38f);
    py = py / fmaxf(sy, 1.17549435e-38f);
    rot2(px, py, rotation);
    float sdf = 0.0f;
    for (int i = 0; i < blades; i++) {
        const float angle = ((float)i / (float)blades + 0.25f) * 2.0f * RF_MPI_F;
        float s, c;
        sincosf(angle, &s, &c);
        sdf = fmaxf(sdf, c * px + s * py);
    }
    const float cg = atan2f(-px, -py) / (2.0f * RF_MPI_F) + 0.5f;
    const float bg = fmodf(cg * (float)blades + 0.5f, 1.0f);
    sdf += sinf(bg * RF_MPI_F) * roundness;
    image[(size_t)y * w + x] = 1.0f - smoothstepf(1.0f - softness, 1.0f + softness, sdf);
}

__global__ void __launch_bounds__(256) k_aperture_dust(float* __restrict__ image, int w, int h, float sx, float sy,
                                                       float strength, int count, float radius, float par_x,
                                                       float par_y, float softness) {
    const int x = blockIdx.x * 16 + (threadIdx.x & 15), y = blockIdx.y * 16 + (threadIdx.x >> 4);
    if (x >= w || y >= h) return;
    float px, py;
    ndc_of(x, y, w, h, px, py);
    px = px / fmaxf(sx, 1.17549435e-38f);
    py = py / fmaxf(sy, 1.17549435e-38f);
    float sdf = 1.0f;
    for (int i = 0; i < count; i++) {
        float cx = noise3((float)i, (float)count, 0.0f) + par_x;
        float cy = noise3((float)i, (float)count, 1.0f) + par_y;
        cx = fmodf(1.0f + fmodf(cx, 1.0f), 1.0f) * 2.0f - 1.0f;
        cy = fmodf(1.0f + fmodf(cy, 1.0f), 1.0f) * 2.0f - 1.0f;
        const float dx = px - cx, dy = py - cy;
        sdf = fminf(sdf, sqrtf(dx * dx + dy * dy) - radius);
    }
    float v = image[(size_t)y * w + x];
    v *= 1.0f - (strength * smoothstepf(softness, -softness, sdf));
    image[(size_t)y * w + x] = v;
}

// numpy's Generator(PCG64(seed)).random(dtype=float32): the permuted congruential generator PCG
// XSL-RR 128/64 (M. E. O'Neill, PCG: A Family of Simple Fast Space-Efficient Statistically Good
// Algorithms for Random Number Generation, 2014), each 64-bit output giving two floats (low half
// first), the top 24 bits of each half over 2^24. Threads jump to their place in the sequence (F.
// B. Brown, Random Number Generation with Arbitrary Strides, 1994): the state after n steps is
// an affine map of the first one, by squaring. 512 x 512: 7.4 us, where the host's generator and
// the copy of its pageable result took about 700.
constexpr int kNoiseOutputs = 4;  // 64-bit outputs per thread
__global__ void __launch_bounds__(256) k_noise_pcg64(unsigned long long state_hi, unsigned long long state_lo,
                                                     unsigned long long inc_hi, unsigned long long inc_lo,
                                                     float* __restrict__ out, long long n) {
    using u128 = unsigned __int128;
    const u128 mult = ((u128)0x2360ed051fc65da4ull << 64) | 0x4385df649fccf645ull;
    const u128 inc = ((u128)inc_hi << 64) | inc_lo;
    const long long first = ((long long)blockIdx.x * blockDim.x + threadIdx.x) * kNoiseOutputs;
    if (2 * first >= n) return;
    u128 a = 1, c = 0, step_a = mult, step_c = inc;  // state -> a state + c: so far, and per power of two
    for (unsigned long long d = (unsigned long long)first; d; d >>= 1) {
        if (d & 1) {
            a *= step_a;
            c = c * step_a + step_c;
        }
        step_c *= step_a + 1;
        step_a *= step_a;
    }
    u128 state = a * (((u128)state_hi << 64) | state_lo) + c;
    float v[2 * kNoiseOutputs];
#pragma unroll
    for (int k = 0; k < kNoiseOutputs; k++) {
        state = state * mult + inc;
        const unsigned long long x = (unsigned long long)(state >> 64) ^ (unsigned long long)state;
        const int r = (int)(state >> 122);
        const unsigned long long o = (x >> r) | (x << ((64 - r) & 63));
        v[2 * k] = (float)((unsigned)o >> 8) * (1.0f / 16777216.0f);
        v[2 * k + 1] = (float)((unsigned)(o >> 32) >> 8) * (1.0f / 16777216.0f);
    }
    if (2 * first + 2 * kNoiseOutputs <= n) {
#pragma unroll
        for (int k = 0; k < kNoiseOutputs / 2; k++)
            reinterpret_cast<float4*>(out + 2 * first)[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    } else {
        for (int k = 0; k < 2 * kNoiseOutputs && 2 * first + k < n; k++) out[2 * first + k] = v[k];
    }
}

// Separable Gaussian over the noise (no reference counterpart): pass 0 blurs rows into
// tmp, pass 1 blurs columns of tmp and multiplies the image by 1 - strength * blur.
struct BlurWeights {
    float w[513];
    int rad;
};

__global__ void __launch_bounds__(256) k_noise_blur(const float* __restrict__ src, float* __restrict__ dst,
                                                    float* __restrict__ image, int w, int h,
                                                    const __grid_constant__ BlurWeights bw, int pass, float strength) {
    const int rad = bw.rad;
    const float* weights = bw.w;
    const int x = blockIdx.x * 16 + (threadIdx.x & 15), y = blockIdx.y * 16 + (threadIdx.x >> 4);
    if (x >= w || y >= h) return;
    float acc = 0.0f;
    for (int k = -rad; k <= rad; k++) {
        int xx = x, yy = y;
        if (pass == 0) xx = min(max(x + k, 0), w - 1);
        else yy = min(max(y + k, 0), h - 1);
        acc += weights[k + rad] * src[(size_t)yy * w + xx];
    }
    if (pass == 0) dst[(size_t)y * w + x] = acc;
    else image[(size_t)y * w + x] = image[(size_t)y * w + x] * (1.0f - strength * acc);
}

// Engine.image_flare's accumulation (realflare/api/engine.py:120-150): per light sample i,
// image += v_i0 * F_i + v_i1 * flip_y(F_i) + v_i2 * flip_yx(F_i) + v_i3 * flip_x(F_i) (per
// channel weights), in sample order, each product and sum rounded as in float32 numpy;
// then image /= count. One thread per output pixel (float4).
__global__ void k_accumulate_mirrored(const float4* __restrict__ frames, const float4* __restrict__ weights, int n,
                                      int w, int h, float divisor, float4* __restrict__ image) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)w * h) return;
    const int x = (int)(i % w), y = (int)(i / w);
    const long long frame = (long long)w * h;
    const long long src[4] = {(long long)y * w + x, (long long)(h - 1 - y) * w + x,
                              (long long)(h - 1 - y) * w + (w - 1 - x), (long long)y * w + (w - 1 - x)};
    float4 acc = image[i];
    for (int k = 0; k < n; k++) {
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const float4 f = frames[k * frame + src[m]];
            const float4 v = weights[4 * k + m];
            acc.x = __fadd_rn(acc.x, __fmul_rn(v.x, f.x));
            acc.y = __fadd_rn(acc.y, __fmul_rn(v.y, f.y));
            acc.z = __fadd_rn(acc.z, __fmul_rn(v.z, f.z));
            acc.w = __fadd_rn(acc.w, __fmul_rn(v.w, f.w));
        }
    }
    if (divisor > 0.0f) {
        acc.x = __fdiv_rn(acc.x, divisor);
        acc.y = __fdiv_rn(acc.y, divisor);
        acc.z = __fdiv_rn(acc.z, divisor);
        acc.w = __fdiv_rn(acc.w, divisor);
    }
    image[i] = acc;
}

__global__ void k_axpby(const float* __restrict__ a, float wa, const float* __restrict__ b, float wb,
                        float* __restrict__ out, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = a[i] * wa + b[i] * wb;
}

}  // namespace
}  // namespace rf

extern "C" int rf_starburst(const float* spectrum, const float* light_spectrum, const rf_starburst_args* args,
                            float* image, void* stream) {
    using namespace rf;
    if (!spectrum || !light_spectrum || !args || !image) return RF_ERR_INVALID_ARG;
    const rf_starburst_args& a = *args;
    if (a.width < 2 || a.height < 2 || a.samples < 1 || a.spectrum_width < 1 || a.spectrum_height < 1 ||
        a.spectrum_count < 1 || !aligned16(image))
        return RF_ERR_INVALID_ARG;
    // With blur 0 the jitter radius is 0 * sqrt(noise) = 0 (noise in [0, 1)), and with
    // rotation 0 and a non-negative weight the angle is +-0 * (1 - noise^weight) = +-0: the
    // jitter and the rotation then leave the position unchanged and their noise is skipped.
    const bool jitter = a.blur != 0.0f, rotate = a.rotation != 0.0f || !(a.rotation_weight >= 0.0f);
    // Lookups by 32-bit offsets and texel coordinates to 2^22 (k_starburst); beyond, one kernel for all
    // settings (the noise then multiplies a radius or an angle of 0).
    const int longest = a.spectrum_width > a.spectrum_height ? a.spectrum_width : a.spectrum_height;
    const bool wide = longest >= (1 << 22) || (long long)a.spectrum_width * a.spectrum_height > 0x7fffffffLL;
    // Plain lookups take two pixels per thread where the image still fills the SMs (scalar form: 2048^2
    // 0.71 -> 0.59 ms, 640 x 480 0.068 -> 0.061, 300^2 0.035 -> 0.039); with noise one is faster (512^2
    // 0.32 against 0.39 ms).
    const bool two = !wide && !jitter && !rotate && (long long)a.width * a.height >= 200000;
    const dim3 grid((a.width + 15) / 16, (a.height + (two ? 31 : 15)) / (two ? 32 : 16));
    const auto kernel = wide ? k_starburst<true, true, 1, true> : two ? k_starburst<false, false, 2>
                            : (jitter ? (rotate ? k_starburst<true, true, 1> : k_starburst<true, false, 1>)
                                      : (rotate ? k_starburst<false, true, 1> : k_starburst<false, false, 1>));
    kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(spectrum, light_spectrum, a, (float4*)image);
    return launch_status();
}

extern "C" int rf_aperture_shape(float* image, int32_t width, int32_t height, float size_x, float size_y,
                                 int32_t blades, float rotation, float roundness, float softness, void* stream) {
    using namespace rf;
    if (!image || width < 2 || height < 2 || blades < 0) return RF_ERR_INVALID_ARG;
    dim3 grid((width + 15) / 16, (height + 15) / 16);
    k_aperture_shape<<<grid, 256, 0, (cudaStream_t)stream>>>(image, width, height, size_x, size_y, blades, rotation,
                                                             roundness, softness);
    return launch_status();
}

extern "C" int rf_aperture_dust(float* image, int32_t width, int32_t height, float size_x, float size_y,
                                float strength, float density, float radius, float parallax_x, float parallax_y,
                                float softness, void* stream) {
    using namespace rf;
    if (!image || width < 2 || height < 2) return RF_ERR_INVALID_ARG;
    // int count = fmin(density, 1) * 1000 (aperture.cl:160)
    const int count = (int)(fminf(density, 1.0f) * 1000.0f);
    dim3 grid((width + 15) / 16, (height + 15) / 16);
    k_aperture_dust<<<grid, 256, 0, (cudaStream_t)stream>>>(image, width, height, size_x, size_y, strength, count,
                                                            radius, parallax_x, parallax_y, softness);
    return launch_status();
}

extern "C" int rf_noise_pcg64(uint64_t state_hi, uint64_t state_lo, uint64_t inc_hi, uint64_t inc_lo, float* out,
                              int64_t count, void* stream) {
    using namespace rf;
    if (!out || count < 0 || !aligned16(out)) return RF_ERR_INVALID_ARG;
    if (count == 0) return RF_OK;
    const long long threads = (count + 2 * kNoiseOutputs - 1) / (2 * kNoiseOutputs);
    if (threads > 0x7fffffffLL) return RF_ERR_NOT_SUPPORTED;
    k_noise_pcg64<<<blocks_for(threads, 256), 256, 0, (cudaStream_t)stream>>>(state_hi, state_lo, inc_hi, inc_lo, out,
                                                                            count);
    return launch_status();
}

extern "C" int rf_aperture_noise_dust(float* image, const float* noise, float* scratch, int32_t width,
                                      int32_t height, float strength, float sigma, void* stream) {
    using namespace rf;
    if (!image || !noise || !scratch || width < 1 || height < 1 || !(sigma >= 0.0f) || sigma > 64.0f)
        return RF_ERR_INVALID_ARG;
    // weights exp(-k^2 / (2 sigma^2)) normalised to 1 in FP32 (the oracle's values),
    // passed by value
    BlurWeights bw;
    bw.rad = (int)std::ceil((double)sigma * 4.0);
    float sum = 0.0f;
    for (int k = -bw.rad; k <= bw.rad; k++) {
        bw.w[k + bw.rad] = sigma > 0.0f ? expf(-(float)(k * k) / (2.0f * sigma * sigma)) : 1.0f;
        sum += bw.w[k + bw.rad];
    }
    for (int k = 0; k <= 2 * bw.rad; k++) bw.w[k] = bw.w[k] / sum;
    cudaStream_t s = (cudaStream_t)stream;
    dim3 grid((width + 15) / 16, (height + 15) / 16);
    k_noise_blur<<<grid, 256, 0, s>>>(noise, scratch, image, width, height, bw, 0, strength);
    RF_TRY(launch_status());
    k_noise_blur<<<grid, 256, 0, s>>>(scratch, nullptr, image, width, height, bw, 1, strength);
    return launch_status();
}

extern "C" int rf_axpby(const float* a, float wa, const float* b, float wb, float* out, int64_t n, void* stream) {
    using namespace rf;
    if (!a || !b || !out || n < 0) return RF_ERR_INVALID_ARG;
    if (n == 0) return RF_OK;
    k_axpby<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(a, wa, b, wb, out, n);
    return launch_status();
}

extern "C" int rf_accumulate_mirrored(const float* frames, const float* weights, int32_t count, int32_t width,
                                      int32_t height, float divisor, float* image, void* stream) {
    using namespace rf;
    if (!frames || !weights || !image || count < 0 || width < 1 || height < 1) return RF_ERR_INVALID_ARG;
    if (!aligned16(frames) || !aligned16(weights) || !aligned16(image)) return RF_ERR_INVALID_ARG;
    const long long n = (long long)width * height;
    k_accumulate_mirrored<<<blocks_for(n, 256), 256, 0, (cudaStream_t)stream>>>(
        (const float4*)frames, (const float4*)weights, count, width, height, divisor, (float4*)image);
    return launch_status();
}
