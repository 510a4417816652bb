// rf_trace.cu — the ghost-path spectral ray trace.
//
// One thread per ray (ghost path, wavelength, grid point), in the reference's ray order
// ((path * W + wavelength) * G^2 + ray). Follows realflare/api/tasks/cl/raytracing.cl:
// init_ray (178-215), the element loop of raytrace (218-359), intersect (123-175), refract
// / reflect (70-102), dispersion (107-120), fresnel (1-16) and fresnel_ar (18-59).
//
// GB300 layout:
//  * the lens elements (radius, center, height, ior, coating) and the refractive index and index
//    ratios of every (wavelength, element) pair are staged in shared memory once per block; the
//    tables replace the per-interaction Sellmeier evaluation and division with lookups of the
//    same FP32 values (dispersion() depends only on the wavelength and the element);
//  * what bounds it is instruction issue (87 % of cycles). Square roots and reciprocals take short
//    correctly rounded forms (sqrt_rn, rcp_rn), rrel is evaluated only where it can be the largest,
//    reflectances go without trigonometric functions: 72.4 M rays through the 24-surface lens
//    18.36 -> 12.42 ms, 7.9 M through the 16-surface lens 1.607 -> 1.052 ms, positions the same
//    bit for bit;
//  * rays of a warp share path and wavelength (G^2 is a multiple of 32 for G >= 32 in
//    practice), so the element loop is warp-uniform up to rays that stop early;
//  * the grid coordinates grid_length * (x / (G - 1) - 0.5), which the reference evaluates
//    in double, are computed once on the host in double and passed as a kernel parameter;
//  * output is six coalesced float planes (pos.xy, pos_apt.xy, rrel, reflectance): the
//    fields the rasteriser reads (pos.z and dir are never read downstream).
#include <math.h>
#include <stdio.h>

#include "rf_trace_core.cuh"

namespace rf {
namespace {

template <bool kAngles>
__global__ void __launch_bounds__(kTraceThreads) k_trace(const rf_lens_element* __restrict__ elements,
                                                         const int2* __restrict__ paths,
                                                         const float* __restrict__ wavelengths,
                                                         const __grid_constant__ TraceParams p, bool table,
                                                         int rays_per_thread, float* __restrict__ rays) {
    __shared__ SmemElement se[kMaxElements];
    extern __shared__ float2 ratio_tab[];  // [rows][E], then the indices
    const int E = p.E;
    // this block's rays_per_thread * kTraceThreads consecutive rays, and the rows (path, wavelength) of
    // R rays they lie in; counted from the first row's start they fit 32 bits
    const long long chunk = (long long)kTraceThreads * rays_per_thread;
    const long long first = (long long)blockIdx.x * chunk;
    const long long last = min(first + chunk, p.n_rays) - 1;
    const long long pw_first = first / p.R;
    const unsigned in_row = (unsigned)(first - pw_first * p.R), R = (unsigned)p.R;
    const int path_first = (int)(pw_first / p.W), wl_first = (int)(pw_first % p.W);
    const int span = min((int)((in_row + (unsigned)(last - first)) / R) + 1, p.W);
    float* ior_tab = (float*)(ratio_tab + span * E);
    // dispersion is on unless coefficient 0 of element 0 is NaN (raytracing.cl:255)
    const bool disperse = !isnan(__ldg(&elements[0].coefficients[0]));
    stage_lens(elements, wavelengths, E, p.W, wl_first, span, table, disperse, se, ratio_tab, ior_tab);
    __syncthreads();

    TraceFrame f;
    f.E = E;
    f.aperture = p.aperture;
    f.W = p.W;
    f.G = p.G;
    f.R = p.R;
    f.cmin = p.cmin;
    f.layer_n0 = p.layer_n0;
    f.layer_n1 = p.layer_n1;
    f.dir[0] = p.dir[0];
    f.dir[1] = p.dir[1];
    f.dir[2] = p.dir[2];
    const long long n = p.n_rays;
#pragma unroll 1
    for (int r = 0; r < rays_per_thread; r++) {
        const unsigned offset = r * kTraceThreads + threadIdx.x;
        const long long idx = first + offset;
        if (idx > last) break;
        const unsigned at = in_row + offset, rows = at / R;
        const int ray_id = (int)(at - rows * R);
        const unsigned wl = wl_first + rows;
        const int path_id = path_first + (int)(wl / (unsigned)p.W), wl_id = (int)(wl % (unsigned)p.W);
        const int row = (int)(rows % (unsigned)p.W);
        // init_ray grid point, raytracing.cl:178-215
        const int gy = (int)truncf((float)ray_id / (float)p.G);
        const int gx = ray_id - gy * p.G;
        float out[6];
        trace_ray<kAngles>(se, table ? ior_tab + row * E : nullptr, table ? ratio_tab + row * E : nullptr, disperse,
                  &elements[0].coefficients[0], __ldg(wavelengths + wl_id), __ldg(paths + path_id), p.grid[gx],
                  p.grid[gy], f, out);
#pragma unroll
        for (int k = 0; k < 6; k++) rays[k * n + idx] = out[k];
    }
}

// Every frame of a batch: block b traces rays_per_thread * 256 consecutive rays of the frame
// whose first trace block is the largest one <= b.
__global__ void __launch_bounds__(kTraceThreads) k_trace_batch(const rf_frame* __restrict__ frames, int F,
                                                               const rf_lens_element* __restrict__ elements_all,
                                                               const int2* __restrict__ paths_all,
                                                               const float* __restrict__ wavelengths_all,
                                                               float* __restrict__ rays_all, int rays_per_thread,
                                                               int table_capacity) {
    __shared__ SmemElement se[kMaxElements];
    extern __shared__ float2 ratio_tab[];  // [rows][E], then the indices
    __shared__ float grid[kMaxGrid];
    __shared__ int frame_index;
    if (threadIdx.x == 0)
        frame_index = find_frame(frames, F, blockIdx.x, [](const rf_frame& fr) { return fr.trace_block; });
    __syncthreads();
    const rf_frame& fr = frames[frame_index];
    TraceFrame f;
    f.E = fr.trace.element_count;
    f.aperture = fr.trace.aperture_index;
    f.W = fr.trace.wavelength_count;
    f.G = fr.trace.grid_count;
    f.R = f.G * f.G;
    f.cmin = fr.trace.coating_min_ior;
    f.layer_n0 = fr.trace.coating_layer_ior[0];
    f.layer_n1 = fr.trace.coating_layer_ior[1];
    f.dir[0] = fr.direction_n[0];
    f.dir[1] = fr.direction_n[1];
    f.dir[2] = fr.direction_n[2];
    const long long n_rays = (long long)fr.trace.path_count * f.W * f.R;
    const rf_lens_element* elements = elements_all + fr.element_offset;
    const float* wavelengths = wavelengths_all + fr.wavelength_offset;
    const int2* paths = paths_all + fr.path_offset;
    float* rays = rays_all + 6 * fr.ray_offset;
    const long long chunk = kTraceThreads * (long long)rays_per_thread;
    const long long first = (blockIdx.x - fr.trace_block) * chunk;
    const long long last = min(first + chunk, n_rays) - 1;
    const long long pw_first = first / f.R, pw_last = last / f.R;
    const long long span_rows = pw_last - pw_first + 1;
    const int span = (int)(span_rows < (long long)f.W ? span_rows : (long long)f.W);
    const bool table = span * f.E <= table_capacity;
    float* ior_tab = (float*)(ratio_tab + span * f.E);
    const bool disperse = !isnan(__ldg(&elements[0].coefficients[0]));
    stage_lens(elements, wavelengths, f.E, f.W, pw_first, span, table, disperse, se, ratio_tab, ior_tab);
    // grid_length * (x / (G - 1) - 0.5), in double as in the reference (and rf_trace's host table)
    for (int i = threadIdx.x; i < f.G; i += kTraceThreads) {
        const float t = (float)i / (float)(f.G - 1);
        grid[i] = (float)((double)fr.trace.grid_length * ((double)t - 0.5));
    }
    __syncthreads();
    const unsigned in_row = (unsigned)(first - pw_first * f.R), R = (unsigned)f.R;
    const int path_first = (int)(pw_first / f.W), wl_first = (int)(pw_first % f.W);
    for (int r = 0; r < rays_per_thread; r++) {
        const unsigned offset = r * kTraceThreads + threadIdx.x;
        const long long idx = first + offset;
        if (idx > last) break;
        const unsigned at = in_row + offset, rows = at / R;
        const int ray_id = (int)(at - rows * R);
        const unsigned wl = wl_first + rows;
        const int path_id = path_first + (int)(wl / (unsigned)f.W), wl_id = (int)(wl % (unsigned)f.W);
        const int row = (int)(rows % (unsigned)f.W);
        const int gy = (int)truncf((float)ray_id / (float)f.G);
        const int gx = ray_id - gy * f.G;
        float out[6];
        trace_ray<false>(se, table ? ior_tab + row * f.E : nullptr, table ? ratio_tab + row * f.E : nullptr, disperse,
                  &elements[0].coefficients[0],
                  __ldg(wavelengths + wl_id), __ldg(paths + path_id), grid[gx], grid[gy], f, out);
#pragma unroll
        for (int k = 0; k < 6; k++) rays[k * n_rays + idx] = out[k];
    }
}

}  // namespace
}  // namespace rf

namespace {
template <bool kAngles>
int trace_entry(const rf_lens_element* elements, const int32_t* paths, const float* wavelengths,
                const rf_trace_args* args, float* rays, void* stream) {
    using namespace rf;
    if (!elements || !paths || !wavelengths || !args || !rays) return RF_ERR_INVALID_ARG;
    const rf_trace_args& a = *args;
    if (a.element_count < 2 || a.element_count > kMaxElements || a.path_count < 0 || a.wavelength_count < 1 ||
        a.grid_count < 2 || a.grid_count > kMaxGrid || a.aperture_index < 0)
        return RF_ERR_INVALID_ARG;
    TraceParams p;
    if (!trace_params(a, p)) return RF_ERR_INVALID_ARG;
    if (p.n_rays == 0) return RF_OK;
    // Several rays per thread share a block's staging of the lens and its index tables, where that
    // leaves many blocks for every SM. 1 / 2 / 4 rays: 72.4 M rays 12.88 / 12.57 / 12.42 ms, 7.9 M
    // 1.086 / 1.052 / 1.052 ms, 3.9 M 0.560 / 0.554 / 0.575 ms (3.9 M are 25 blocks of 4 rays per SM).
    int sms = 0, dev = 0;
    RF_TRY(cuda_status(cudaGetDevice(&dev)));
    RF_TRY(cuda_status(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)));
    int rays_per_thread = 4;
    while (rays_per_thread > 1 && p.n_rays < (long long)rays_per_thread * kTraceThreads * sms * 48) rays_per_thread /= 2;
    const long long chunk = (long long)kTraceThreads * rays_per_thread;
    const size_t table = table_bytes(chunk, p.R, p.W, p.E);
    k_trace<kAngles><<<blocks_for(p.n_rays, (int)chunk), kTraceThreads, table, (cudaStream_t)stream>>>(
        elements, (const int2*)paths, wavelengths, p, table > 0, rays_per_thread, rays);
    return launch_status();
}
}  // namespace

extern "C" int rf_trace(const rf_lens_element* elements, const int32_t* paths, const float* wavelengths,
                        const rf_trace_args* args, float* rays, void* stream) {
    return trace_entry<false>(elements, paths, wavelengths, args, rays, stream);
}

extern "C" int rf_trace_differentiable(const rf_lens_element* elements, const int32_t* paths,
                                       const float* wavelengths, const rf_trace_args* args, float* rays,
                                       void* stream) {
    return trace_entry<true>(elements, paths, wavelengths, args, rays, stream);
}

extern "C" int rf_trace_batch(const rf_frame* frames, const rf_batch_sizes* sizes, const rf_lens_element* elements,
                              const int32_t* paths, const float* wavelengths, float* rays, void* stream) {
    using namespace rf;
    if (!frames || !sizes || !elements || !paths || !wavelengths || !rays) return RF_ERR_INVALID_ARG;
    if (sizes->trace_blocks == 0) return RF_OK;
    if (sizes->trace_blocks > 0x7fffffffLL) return RF_ERR_NOT_SUPPORTED;
    // the frames' sizes are on the device: a table of 16 KB holds every block's rows but those of
    // the smallest grids, which look their indices up one by one
    constexpr int kBatchTable = 16 * 1024;
    k_trace_batch<<<(unsigned)sizes->trace_blocks, kTraceThreads, kBatchTable, (cudaStream_t)stream>>>(
        frames, sizes->frame_count, elements, (const int2*)paths, wavelengths, rays, sizes->rays_per_thread,
        kBatchTable / (int)sizeof(IorEntry));
    return launch_status();
}
