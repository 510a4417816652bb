// rf_trace.cu — the ghost-path spectral ray trace.
//
// A thread traces one grid point and wavelength along up to 16 ghost paths (trace_paths in
// rf_trace_core.cuh); rays are stored in the reference's order ((path * W + wavelength) * G^2 + ray).
// Follows realflare/api/tasks/cl/raytracing.cl: init_ray (178-215), the element loop of
// raytrace (218-359), intersect (123-175), refract / reflect (70-102), dispersion (107-120),
// fresnel (1-16) and fresnel_ar (18-59).
//
// GB300 layout:
//  * legs that ghost paths share are traced once: 72.4 M rays through the 24-surface lens 12.55 ms one
//    path at a time, 5.63 sixteen at a time; 7.9 M through the 16-surface lens 1.055 -> 0.592 ms; 15.1 M
//    of the zoom 1.698 -> 0.800 ms; the results the same bit for bit;
//  * the lens elements (radius, center, height, ior, coating) and the refractive index and index
//    ratios of every (wavelength, element) pair are staged in shared memory once per block; the
//    tables replace the per-interaction Sellmeier evaluation and division with lookups of the
//    same FP32 values (dispersion() depends only on the wavelength and the element);
//  * what bounds it is instruction issue (89 % of active cycles). Square roots and reciprocals take
//    short correctly rounded forms (sqrt_rn, rcp_rn), rrel is evaluated only where it can be the
//    largest, reflectances go without trigonometric functions: 72.4 M rays 18.36 -> 12.42 ms one
//    path at a time;
//  * the rays of a warp walk the same elements together; those that fail wait for the others;
//  * the grid coordinates grid_length * (x / (G - 1) - 0.5), which the reference evaluates
//    in double, are computed once on the host in double and passed as a kernel parameter;
//  * output is six coalesced float planes (pos.xy, pos_apt.xy, rrel, reflectance): the
//    fields the rasteriser reads (pos.z and dir are never read downstream).
#include <math.h>

#include <algorithm>

#include "rf_trace_core.cuh"

namespace rf {
namespace {

template <bool kAngles>
__global__ void __launch_bounds__(kTraceThreads) k_trace(const rf_lens_element* __restrict__ elements,
                                                         const int2* __restrict__ paths,
                                                         const float* __restrict__ wavelengths,
                                                         const __grid_constant__ TraceParams p, bool table,
                                                         int path_blocks, float* __restrict__ rays) {
    __shared__ SmemElement se[kMaxElements];
    __shared__ PathList list;
    extern __shared__ float2 ratio_tab[];  // [rows][E], then the indices
    const int E = p.E;
    // this block's paths, and its kTraceThreads consecutive ones of a path's (wavelength, grid point) pairs and
    // the wavelengths they span; counted from the first one's start the pairs fit 32 bits. The
    // paths with the longest shared legs come last in a list of pairs: their blocks go first
    const int path_block = path_blocks - 1 - (int)(blockIdx.x % path_blocks);
    const int path_first = first_path(path_block, path_blocks, p.P);
    const int path_count = first_path(path_block + 1, path_blocks, p.P) - path_first;
    const long long per_path = (long long)p.W * p.R;
    const long long first = (long long)(blockIdx.x / path_blocks) * kTraceThreads;
    const long long last = min(first + kTraceThreads, per_path) - 1;
    const int wl_first = (int)(first / p.R);
    const unsigned in_row = (unsigned)(first - (long long)wl_first * p.R), R = (unsigned)p.R;
    const int span = (int)((in_row + (unsigned)(last - first)) / R) + 1;
    float* ior_tab = (float*)(ratio_tab + span * E);
    // dispersion is on unless coefficient 0 of element 0 is NaN (raytracing.cl:255)
    const bool disperse = !isnan(__ldg(&elements[0].coefficients[0]));
    if (threadIdx.x < 32) stage_paths(paths, path_first, path_count, E, p.aperture, list);
    stage_lens(elements, wavelengths, E, p.W, wl_first, span, table, disperse, se, ratio_tab, ior_tab);
    __syncthreads();

    FloatRay<kAngles> ray;
    ray.f.E = E;
    ray.f.aperture = p.aperture;
    ray.f.cmin = p.cmin;
    ray.f.layer_n0 = p.layer_n0;
    ray.f.layer_n1 = p.layer_n1;
    ray.f.dir[0] = p.dir[0];
    ray.f.dir[1] = p.dir[1];
    ray.f.dir[2] = p.dir[2];
    ray.mine = first + threadIdx.x <= last;
    const unsigned at = in_row + (ray.mine ? threadIdx.x : 0), row = at / R;
    const int ray_id = (int)(at - row * R);
    ray.se = se;
    ray.ior_row = table ? ior_tab + row * E : nullptr;
    ray.ratio_row = table ? ratio_tab + row * E : nullptr;
    ray.disperse = disperse;
    ray.coef_base = &elements[0].coefficients[0];
    ray.wavelength = __ldg(wavelengths + wl_first + row);
    ray.out = rays + first + threadIdx.x;
    ray.per_path = per_path;
    ray.plane = p.n_rays;
    const int gy = (int)truncf((float)ray_id / (float)p.G);
    const int gx = ray_id - gy * p.G;
    trace_paths(ray, ray.start(p.grid[gx], p.grid[gy]), ray.mine, list, path_count, E, p.aperture);
}

// Every frame of a batch: a work item is paths_each paths and rays_per_thread * kTraceThreads (wavelength,
// grid point) pairs of the frame whose first item is the largest one <= its index. Blocks take
// items gridDim.x apart (about one each; the frames' exact number is known on the device).
__global__ void __launch_bounds__(kTraceThreads) k_trace_batch(const rf_frame* __restrict__ frames, int F,
                                                               const rf_lens_element* __restrict__ elements_all,
                                                               const int2* __restrict__ paths_all,
                                                               const float* __restrict__ wavelengths_all,
                                                               float* __restrict__ rays_all, int paths_each,
                                                               int rays_per_thread, int table_capacity) {
    __shared__ SmemElement se[kMaxElements];
    __shared__ PathList list;
    extern __shared__ float2 ratio_tab[];  // [rows][E], then the indices
    __shared__ int frame_index;
    const long long items = frames[F - 1].trace_item + batch_trace_items(frames[F - 1].trace, paths_each, rays_per_thread);
#pragma unroll 1
    for (long long item = blockIdx.x; item < items; item += gridDim.x) {
        if (threadIdx.x == 0)
            frame_index = find_frame(frames, F, item, [](const rf_frame& fr) { return fr.trace_item; });
        __syncthreads();
        const rf_frame& fr = frames[frame_index];
        FloatRay<false> ray;
        const int E = fr.trace.element_count, aperture = fr.trace.aperture_index, W = fr.trace.wavelength_count;
        const int G = fr.trace.grid_count, R = G * G;
        ray.f.E = E;
        ray.f.aperture = aperture;
        ray.f.cmin = fr.trace.coating_min_ior;
        ray.f.layer_n0 = fr.trace.coating_layer_ior[0];
        ray.f.layer_n1 = fr.trace.coating_layer_ior[1];
        ray.f.dir[0] = fr.direction_n[0];
        ray.f.dir[1] = fr.direction_n[1];
        ray.f.dir[2] = fr.direction_n[2];
        const rf_lens_element* elements = elements_all + fr.element_offset;
        const float* wavelengths = wavelengths_all + fr.wavelength_offset;
        const int path_blocks = (fr.trace.path_count + paths_each - 1) / paths_each;
        const long long block = item - fr.trace_item;
        const int path_block = path_blocks - 1 - (int)(block % path_blocks);
        const int path_first = first_path(path_block, path_blocks, fr.trace.path_count);
        const int path_count = first_path(path_block + 1, path_blocks, fr.trace.path_count) - path_first;
        const long long per_path = (long long)W * R, chunk = kTraceThreads * (long long)rays_per_thread;
        const long long first = block / path_blocks * chunk;
        const long long last = min(first + chunk, per_path) - 1;
        const int wl_first = (int)(first / R);
        const unsigned in_row = (unsigned)(first - (long long)wl_first * R);
        const int span = (int)((in_row + (unsigned)(last - first)) / R) + 1;
        const bool table = span * E <= table_capacity;
        float* ior_tab = (float*)(ratio_tab + span * E);
        const bool disperse = !isnan(__ldg(&elements[0].coefficients[0]));
        if (threadIdx.x < 32) stage_paths(paths_all + fr.path_offset, path_first, path_count, E, aperture, list);
        stage_lens(elements, wavelengths, E, W, wl_first, span, table, disperse, se, ratio_tab, ior_tab);
        __syncthreads();
        ray.se = se;
        ray.disperse = disperse;
        ray.coef_base = &elements[0].coefficients[0];
        ray.per_path = per_path;
        ray.plane = fr.trace.path_count * per_path;
        for (int r = 0; r < rays_per_thread; r++) {
            const unsigned offset = r * kTraceThreads + threadIdx.x;
            ray.mine = first + offset <= last;
            const unsigned at = in_row + (ray.mine ? offset : 0), row = at / (unsigned)R;
            const int ray_id = (int)(at - row * R);
            ray.ior_row = table ? ior_tab + row * E : nullptr;
            ray.ratio_row = table ? ratio_tab + row * E : nullptr;
            ray.wavelength = __ldg(wavelengths + wl_first + row);
            ray.out = rays_all + 6 * fr.ray_offset + first + offset;
            const int gy = (int)truncf((float)ray_id / (float)G);
            const int gx = ray_id - gy * G;
            // grid_length * (x / (G - 1) - 0.5), in double as in the reference (and rf_trace's host table)
            const float tx = (float)gx / (float)(G - 1), ty = (float)gy / (float)(G - 1);
            const double length = fr.trace.grid_length;
            trace_paths(ray, ray.start((float)(length * ((double)tx - 0.5)), (float)(length * ((double)ty - 0.5))),
                        ray.mine, list, path_count, E, aperture);
        }
        __syncthreads();  // before the next item's staging
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
    const long long per_path = (long long)p.W * p.R;
    const long long ray_blocks = (per_path + kTraceThreads - 1) / kTraceThreads;
    int sms = 0, dev = 0;
    RF_TRY(cuda_status(cudaGetDevice(&dev)));
    RF_TRY(cuda_status(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)));
    const int paths_each = paths_per_block(p.P, ray_blocks, (long long)sms * kTraceBlocksPerSm);
    const long long path_blocks = (p.P + paths_each - 1) / paths_each, blocks = ray_blocks * path_blocks;
    if (blocks > 0x7fffffffLL) return RF_ERR_NOT_SUPPORTED;
    const size_t table = table_bytes(kTraceThreads, p.R, p.W, p.E);
    k_trace<kAngles><<<(unsigned)blocks, kTraceThreads, table, (cudaStream_t)stream>>>(
        elements, (const int2*)paths, wavelengths, p, table > 0, (int)path_blocks, rays);
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
    // the frames' sizes are on the device: a table of 8 KB holds every block's rows but those of
    // the smallest grids, which look their indices up one by one
    constexpr int kBatchTable = 8 * 1024;
    const int paths_each = batch_trace_paths(sizes->rays, sizes->rays_per_thread);
    const long long per_item = (long long)paths_each * kTraceThreads * sizes->rays_per_thread;
    const long long blocks = std::min<long long>((sizes->rays + per_item - 1) / per_item + sizes->frame_count, 0x7fffffffLL);
    k_trace_batch<<<(unsigned)blocks, kTraceThreads, kBatchTable, (cudaStream_t)stream>>>(
        frames, sizes->frame_count, elements, (const int2*)paths, wavelengths, rays, paths_each, sizes->rays_per_thread,
        kBatchTable / (int)sizeof(IorEntry));
    return launch_status();
}
