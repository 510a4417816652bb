// rf_bin.cu — binning of ghost quads.
//
// The reference bins primitives into BIN_SIZE-pixel bins with 255-primitive bit masks
// (realflare/api/tasks/cl/rasterizing.cl:388-469) and then lets every pixel scan every
// mask of its bin. Here a primitive's reference bins form a rectangle, computed with the
// reference's exact integer test (convert_int4 truncation, integer res / 2, inclusive
// overlap on both ends), and:
//  * rf_bin_masks materialises the reference's mask layout from those rectangles (parity);
//  * rf_bin_tiles emits one entry per (primitive, wavelength pair, raster tile) where the
//    tile lies in the primitive's reference bins and in the conservative bounds of that
//    wavelength pair's quads, then orders every tile's entries by (primitive, pair) with a
//    stable radix sort keyed by tile. The raster then visits exactly the reference's
//    (pixel, primitive) candidates that can produce coverage, in the reference's order.
#include <algorithm>

#include "rf_common.cuh"

namespace rf {
namespace {

constexpr int kThreads = 256;
// Sample coordinates below this magnitude keep the reference's 32-bit edge functions
// free of overflow (|difference| < 2^15, |product| < 2^30), so a sample outside the
// integer bounds of a quad is never inside it.
constexpr float kSafeSamples = 16383.0f;

struct BinGeometry {
    int width, height, B, T, bdx, bdy, ntx, nty, S, W, G, maxW, wide_bits;
    float st;
    bool safe_screen;  // width * S and height * S fit the overflow-free range
};

__device__ __forceinline__ long long floor_div(long long a, long long b) {
    long long q = a / b;
    if ((a % b != 0) && ((a < 0) != (b < 0))) q--;
    return q;
}

// Reference bins overlapped by a primitive's bounds (mm), rasterizing.cl:449-453.
// Returns false for culled primitives (bounds.x NaN) or empty rectangles.
__device__ __forceinline__ bool ref_bin_rect(float4 b, const BinGeometry& g, int& bx0, int& bx1, int& by0,
                                             int& by1) {
    if (isnan(b.x)) return false;
    int32_t sx0 = wadd(cvt_rz_sat(b.x * g.st), g.width / 2);
    int32_t sy0 = wadd(cvt_rz_sat(b.y * g.st), g.height / 2);
    int32_t sx1 = wadd(cvt_rz_sat(b.z * g.st), g.width / 2);
    int32_t sy1 = wadd(cvt_rz_sat(b.w * g.st), g.height / 2);
    // bin bx covers [bx*B, bx*B + B] inclusive: sx0 <= bx*B + B and sx1 >= bx*B
    long long lx = floor_div((long long)sx0 - 1, g.B), hx = floor_div((long long)sx1, g.B);
    long long ly = floor_div((long long)sy0 - 1, g.B), hy = floor_div((long long)sy1, g.B);
    lx = max(lx, 0LL);
    ly = max(ly, 0LL);
    hx = min(hx, (long long)g.bdx - 1);
    hy = min(hy, (long long)g.bdy - 1);
    if (lx > hx || ly > hy) return false;
    bx0 = (int)lx;
    bx1 = (int)hx;
    by0 = (int)ly;
    by1 = (int)hy;
    return true;
}

__global__ void __launch_bounds__(kThreads) k_bin_masks(const float4* __restrict__ bounds, int prim_count,
                                                        BinGeometry g, int batch_count,
                                                        unsigned long long* __restrict__ masks) {
    const int prim = blockIdx.x * kThreads + threadIdx.x;
    if (prim >= prim_count) return;
    int bx0, bx1, by0, by1;
    if (!ref_bin_rect(bounds[prim], g, bx0, bx1, by0, by1)) return;
    const int batch = prim / RF_BATCH_PRIMITIVE_COUNT;
    const int bit = prim % RF_BATCH_PRIMITIVE_COUNT + 1;
    for (int by = by0; by <= by1; by++)
        for (int bx = bx0; bx <= bx1; bx++) {
            unsigned long long* q = masks + 4 * ((size_t)(by * g.bdx + bx) * batch_count + batch);
            atomicOr(q + (bit >> 6), 1ull << (bit & 63));
            atomicOr(q, 1ull);
        }
}

// Tile rectangle of one (primitive, wavelength pair); false when it contributes nothing.
__device__ __forceinline__ bool pair_tile_rect(const float4* __restrict__ bounds, const float4* __restrict__ vtx,
                                               long long pair, const BinGeometry& g, int& tx0, int& tx1,
                                               int& ty0, int& ty1) {
    int bx0, bx1, by0, by1, w, quad;
    long long prim, path;
    divide(pair, g.maxW, prim, w);
    if (!ref_bin_rect(__ldg(bounds + prim), g, bx0, bx1, by0, by1)) return false;
    const int Q = (g.G - 1) * (g.G - 1), VC = g.G * g.G;
    divide(prim, Q, path, quad);
    const int row = quad / (g.G - 1), col = quad % (g.G - 1);
    const int c0 = row * g.G + col;
    const int corners[4] = {c0, c0 + 1, c0 + 1 + g.G, c0 + g.G};
    float mnx = INFINITY, mny = INFINITY, mxx = -INFINITY, mxy = -INFINITY;
    bool finite = true;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const long long vi = (path * VC + corners[k]) * g.W + w;
#pragma unroll
        for (int e = 0; e < 2; e++) {  // endpoints at pair wavelengths w and w + 1
            const float4 a = __ldg(vtx + 2 * (vi + e));
            const float refl = __ldg(&vtx[2 * (vi + e) + 1].y);
            if (isnan(refl)) return false;  // an invalid endpoint: the pair contributes 0
            finite = finite && isfinite(a.x) && isfinite(a.y);
            mnx = fminf(mnx, a.x);
            mxx = fmaxf(mxx, a.x);
            mny = fminf(mny, a.y);
            mxy = fmaxf(mxy, a.y);
        }
    }
    const int tpb = g.B / g.T;  // tiles per bin edge
    tx0 = bx0 * tpb;
    tx1 = min((bx1 + 1) * tpb - 1, g.ntx - 1);
    ty0 = by0 * tpb;
    ty1 = min((by1 + 1) * tpb - 1, g.nty - 1);
    const float S = (float)g.S;
    const bool safe = g.safe_screen && finite && fabsf(mnx * S) < kSafeSamples && fabsf(mxx * S) < kSafeSamples &&
                      fabsf(mny * S) < kSafeSamples && fabsf(mxy * S) < kSafeSamples;
    if (safe) {
        // pixels with a sample inside the quads lie within [min - 2, max + 2]
        tx0 = max(tx0, (int)floorf((mnx - 2.0f) / (float)g.T));
        tx1 = min(tx1, (int)floorf((mxx + 2.0f) / (float)g.T));
        ty0 = max(ty0, (int)floorf((mny - 2.0f) / (float)g.T));
        ty1 = min(ty1, (int)floorf((mxy + 2.0f) / (float)g.T));
    }
    return tx0 <= tx1 && ty0 <= ty1;
}

// A pair's tile rectangle in 64 bits, so that it is found once, when it is counted, and not again
// when its entries are written: its first tile (31 bits), width - 1 (wide_bits, those of the largest
// there is) and height - 1; all ones: empty.
constexpr unsigned long long kNoTiles = ~0ull;
__device__ __forceinline__ unsigned long long pack_rect(int tx0, int tx1, int ty0, int ty1, const BinGeometry& g) {
    return (unsigned long long)((unsigned)ty0 * (unsigned)g.ntx + (unsigned)tx0) |
           (unsigned long long)(tx1 - tx0) << 31 | (unsigned long long)(ty1 - ty0) << (31 + g.wide_bits);
}

// Rectangle of a thread's pair into *rect, and the block's number of entries.
__device__ __forceinline__ void count_pair(const float4* __restrict__ bounds, const float4* __restrict__ vtx,
                                           long long pair, bool valid, const BinGeometry& g,
                                           unsigned long long* rect, uint32_t* __restrict__ sums,
                                           unsigned long long* __restrict__ total) {
    __shared__ unsigned long long warp_sums[kThreads / 32];
    unsigned long long c = 0;
    if (valid) {
        int tx0, tx1, ty0, ty1;
        unsigned long long packed = kNoTiles;
        if (pair_tile_rect(bounds, vtx, pair, g, tx0, tx1, ty0, ty1)) {
            c = (unsigned long long)(tx1 - tx0 + 1) * (unsigned long long)(ty1 - ty0 + 1);
            packed = pack_rect(tx0, tx1, ty0, ty1, g);
        }
        *rect = packed;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 1; k < kThreads / 32; k++) c += warp_sums[k];
        sums[blockIdx.x] = (uint32_t)c;  // (a total beyond 32 bits is reported or refused by it)
        if (c) atomicAdd(total, c);
    }
}

__global__ void __launch_bounds__(kThreads) k_pair_count(const float4* __restrict__ bounds,
                                                         const float4* __restrict__ vtx, long long n_pairs,
                                                         BinGeometry g, unsigned long long* __restrict__ rects,
                                                         uint32_t* __restrict__ sums,
                                                         unsigned long long* __restrict__ total) {
    const long long j = (long long)blockIdx.x * kThreads + threadIdx.x;
    count_pair(bounds, vtx, j, j < n_pairs, g, rects + j, sums, total);
}

// Writes the entries of a block's pairs (rects[0, n), the first one's number first_pair): the block's place in
// the lists is base, its pairs' places follow from a scan of their counts. Threads take places, not
// pairs (a pair covers one tile or thousands), and find a place's pair by bisection, so the stores
// are coalesced. 92 M entries of 67 M pairs: 0.92 -> 0.48 ms (a thread per pair, its rectangle found
// anew); 62 k of 27 k: 14.8 -> 5.3 us.
__device__ __forceinline__ void emit_pairs(const unsigned long long* rects, int n, uint32_t base, long long capacity,
                                           int ntx, int wide_bits, uint32_t first_tile, uint32_t first_pair,
                                           uint32_t* keys, uint32_t* vals) {
    __shared__ uint32_t start[kThreads], corner[kThreads], width[kThreads], warp_sums[kThreads / 32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const unsigned long long r = t < n ? rects[t] : kNoTiles;
    const uint32_t w = (uint32_t)(r >> 31 & ((1ull << wide_bits) - 1)) + 1, h = (uint32_t)(r >> (31 + wide_bits)) + 1;
    const uint32_t count = r == kNoTiles ? 0 : w * h;
    uint32_t x = count;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (int k = 0; k < kThreads / 32; k++) {
        if (k == warp) before = total;
        total += warp_sums[k];
    }
    start[t] = before + x - count;
    corner[t] = (uint32_t)r & 0x7fffffffu;
    width[t] = w;
    __syncthreads();
    for (uint32_t k = t; k < total; k += kThreads) {
        int i = 0;  // the last pair that starts at or before place k (those without entries start where the next does)
#pragma unroll
        for (int step = kThreads / 2; step > 0; step >>= 1)
            if (start[i + step] <= k) i += step;
        const uint32_t d = k - start[i], dy = d / width[i], pos = base + k;
        if (pos < capacity) {  // an overflowing batch is reported through the entry total
            keys[pos] = first_tile + corner[i] + dy * (uint32_t)ntx + (d - dy * width[i]);
            vals[pos] = first_pair + (uint32_t)i;
        }
    }
}

__global__ void __launch_bounds__(kThreads) k_pair_emit(const unsigned long long* rects, long long n_pairs, int ntx,
                                                        int wide_bits, const uint32_t* offsets, long long capacity,
                                                        uint32_t* keys, uint32_t* vals) {
    chain_wait();
    const long long first = (long long)blockIdx.x * kThreads;
    emit_pairs(rects + first, (int)min((long long)kThreads, n_pairs - first), offsets[blockIdx.x], capacity, ntx, wide_bits,
               0, (uint32_t)first, keys, vals);
}

// tile_offsets[t] = first position of key >= t in the sorted keys. A warp per tile: each step looks at 32
// places of the interval at once, 6 dependent loads in 92 M keys instead of 27 (15.7 -> 8.3 us).
__global__ void __launch_bounds__(kThreads) k_tile_offsets(const uint32_t* keys, long long n, int ntiles,
                                                           uint32_t* tile_offsets) {
    chain_wait();
    const int lane = threadIdx.x & 31;
    const long long t = ((long long)blockIdx.x * kThreads + threadIdx.x) >> 5;
    if (t > ntiles) return;
    long long lo = 0, hi = n;
    while (hi > lo) {  // the answer lies in [lo, hi]
        const long long len = hi - lo, step = (len + 31) / 32;
        const long long at = lo + lane * step;  // the first of this lane's step places
        const bool less = at < hi && keys[at] < (uint32_t)t;
        const int k = __popc(__ballot_sync(0xffffffffu, less));  // lanes whose first place lies before the answer
        if (k == 0) break;
        hi = min(hi, lo + k * step);
        lo += (k - 1) * step + 1;
    }
    if (lane == 0) tile_offsets[t] = (uint32_t)lo;
}

// Raster tiles are 32 x 32 or 16 x 16 pixels (rf_raster.cu); bins must be multiples of the tile.
// Without a tile size in the arguments: 32, or 16 where an image has too few 32-pixel tiles to fill
// the 152 SMs' 4 resident CTAs evenly (a tile's list is walked by one CTA). k_raster, 32- against
// 16-pixel tiles: 512 x 512, 8 wavelengths (256 tiles) 2.83 / 1.21 ms; 800 x 800 (625) 2.67 / 2.38;
// 900 x 900 (841) 2.89 / 2.94; 1024 x 1024 (1024) 3.18 / 3.57. With several samples per pixel the
// per-entry work is small against the fragments' and the line lies higher: four samples 900 x 900
// 4.00 / 3.59 ms, 1024 x 1024 4.51 / 4.32 ms.
__host__ __device__ inline int auto_tile(const rf_raster_args& a) {
    if (a.tile_size > 0) return a.tile_size;
    const long long tiles = (long long)((a.width + 31) / 32) * ((a.height + 31) / 32);
    return a.bin_size % 32 == 0 && tiles <= (a.sub_steps > 1 ? 1216 : 640) ? 16 : 32;
}

__host__ __device__ inline bool make_geometry(const rf_raster_args& a, BinGeometry& g) {
    if (a.width < 1 || a.height < 1 || a.bin_size < 1 || a.grid_count < 2 || a.wavelength_count < 1 ||
        a.path_count < 0)
        return false;
    g.width = a.width;
    g.height = a.height;
    g.B = a.bin_size;
    g.T = auto_tile(a);
    if ((g.T != 32 && g.T != 16) || g.B % g.T) return false;
    g.bdx = (a.width + g.B - 1) / g.B;
    g.bdy = (a.height + g.B - 1) / g.B;
    g.ntx = (a.width + g.T - 1) / g.T;
    g.nty = (a.height + g.T - 1) / g.T;
    g.wide_bits = 0;
    while ((1LL << g.wide_bits) < g.ntx) g.wide_bits++;
    g.S = a.sub_steps;
    g.W = a.wavelength_count;
    g.G = a.grid_count;
    g.maxW = a.wavelength_count - 1 > 1 ? a.wavelength_count - 1 : 1;
    g.st = a.screen_transform;
    g.safe_screen = (float)a.width * a.sub_steps <= 16384.0f && (float)a.height * a.sub_steps <= 16384.0f;
    return true;
}

// ---------------------------------------------------------------- batched frames
// Block b of a stage works for the frame whose first block is the largest one <= b; the
// frame's pairs, bounds and vertices are found through its offsets, and its tiles are
// numbered from tile_offset in the batch's tile numbering.
struct FramePairs {
    BinGeometry g;
    long long n_pairs;  // the frame's pair count; 0 for a geometry that is not valid
    int frame;
};

__device__ __forceinline__ void frame_pairs(const rf_frame* __restrict__ frames, int F, FramePairs* fp) {
    if (threadIdx.x == 0) {
        fp->frame = find_frame(frames, F, blockIdx.x, [](const rf_frame& fr) { return fr.pair_block; });
        const rf_raster_args& a = frames[fp->frame].raster;
        fp->n_pairs = make_geometry(a, fp->g) ? (long long)a.path_count * (fp->g.G - 1) * (fp->g.G - 1) * fp->g.maxW : 0;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kThreads) k_pair_count_batch(const rf_frame* __restrict__ frames, int F,
                                                               const float4* __restrict__ bounds_all,
                                                               const float4* __restrict__ vtx_all,
                                                               unsigned long long* __restrict__ rects,
                                                               uint32_t* __restrict__ sums,
                                                               unsigned long long* __restrict__ total) {
    __shared__ FramePairs fp;
    frame_pairs(frames, F, &fp);
    const rf_frame& fr = frames[fp.frame];
    const long long j = (blockIdx.x - fr.pair_block) * kThreads + threadIdx.x;
    count_pair(bounds_all + fr.prim_offset, vtx_all + 2 * fr.vertex_offset, j, j < fp.n_pairs, fp.g,
               rects + fr.pair_offset + j, sums, total);
}

__global__ void __launch_bounds__(kThreads) k_pair_emit_batch(const rf_frame* frames, int F,
                                                              const unsigned long long* rects, const uint32_t* offsets,
                                                              long long capacity, uint32_t* keys, uint32_t* vals) {
    __shared__ FramePairs fp;
    chain_wait();
    frame_pairs(frames, F, &fp);
    const rf_frame& fr = frames[fp.frame];
    const long long first = (blockIdx.x - fr.pair_block) * kThreads, rest = fp.n_pairs - first;
    emit_pairs(rects + fr.pair_offset + first, (int)(rest < kThreads ? rest : kThreads), offsets[blockIdx.x], capacity,
               fp.g.ntx, fp.g.wide_bits, (uint32_t)fr.tile_offset, (uint32_t)first, keys, vals);
}

// Entries [total, capacity) get the key `pad` (one past the last tile), so the sort over the
// whole capacity leaves them at the end.
__global__ void k_pad_entries(const unsigned long long* total, long long capacity, uint32_t pad, uint32_t* keys,
                              uint32_t* vals) {
    chain_wait();
    for (unsigned long long i = *total + (unsigned long long)blockIdx.x * kThreads + threadIdx.x;
         i < (unsigned long long)capacity; i += (unsigned long long)gridDim.x * kThreads) {
        keys[i] = pad;
        vals[i] = 0;
    }
}

// Sort keys for the raster's tile order: 255 minus the tile's entry count as a tiny float
// (the position of its leading one bit and the three bits after it), so an ascending
// stable sort puts the heaviest tiles first, within 12.5 %, and ties in tile order; empty
// tiles, which still write their pixels, come last.
constexpr int kOrderKeyBits = 8;
__device__ __forceinline__ uint32_t order_key(uint32_t n) {
    if (n == 0) return 255;
    const int lz = __clz((int)n);
    const uint32_t e = 31 - lz, m = (n << lz) << 1 >> 29;  // the 3 bits after the leading one
    return 255 - (e * 8 + m);
}
__global__ void k_tile_order_keys(const uint32_t* tile_offsets, int tiles, uint32_t* keys, uint32_t* vals) {
    chain_wait();
    const int t = blockIdx.x * kThreads + threadIdx.x;
    if (t >= tiles) return;
    keys[t] = order_key(tile_offsets[t + 1] - tile_offsets[t]);
    vals[t] = (uint32_t)t;
}
// The whole order by one block, for up to kOrderBlockTiles tiles: a warp takes consecutive tiles, 32 at a
// time, counts their keys and, once all counts are prefixed in (key, warp) order, places them. 1024
// tiles: 4.2 us instead of the 16 us of four launches (keys, histogram, scan, scatter).
constexpr int kOrderThreads = 1024, kOrderWarps = kOrderThreads / 32;
constexpr int kOrderBlockTiles = 16384;
__global__ void __launch_bounds__(kOrderThreads) k_tile_order(const uint32_t* tile_offsets, int tiles,
                                                              uint32_t* order) {
    __shared__ uint32_t counts[kOrderWarps][257];
    __shared__ uint32_t warp_sums[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < kOrderWarps * 257; i += kOrderThreads) (&counts[0][0])[i] = 0;
    chain_wait();
    __syncthreads();
    const int per_warp = ((tiles + kOrderThreads - 1) / kOrderThreads) * 32, first = warp * per_warp;
    const int end = min(first + per_warp, tiles);
    for (int pass = 0; pass < 2; pass++) {
        for (int base = first; base < end; base += 32) {
            const int t = base + lane;
            const uint32_t key = t < end ? order_key(tile_offsets[t + 1] - tile_offsets[t]) : 256;
            const unsigned peers = __match_any_sync(0xffffffffu, key);
            const int leader = __ffs(peers) - 1;
            uint32_t at = 0;
            if (lane == leader) {
                at = counts[warp][key];
                counts[warp][key] = at + __popc(peers);
            }
            at = __shfl_sync(0xffffffffu, at, leader) + __popc(peers & ((1u << lane) - 1u));
            if (pass == 1 && t < end) order[at] = (uint32_t)t;
            __syncwarp();
        }
        if (pass == 1) break;
        __syncthreads();
        uint32_t total = 0, x = 0;
        if (threadIdx.x < 256) {
            for (int w = 0; w < kOrderWarps; w++) total += counts[w][threadIdx.x];
            x = total;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) warp_sums[warp] = x;
        }
        __syncthreads();
        if (threadIdx.x < 256) {
            uint32_t run = x - total;
            for (int w = 0; w < warp; w++) run += warp_sums[w];
            for (int w = 0; w < kOrderWarps; w++) {
                const uint32_t c = counts[w][threadIdx.x];
                counts[w][threadIdx.x] = run;
                run += c;
            }
        }
        __syncthreads();
    }
}

struct BinWorkspace {
    unsigned long long* rects;
    uint32_t *sums, *scan_scratch, *keys_a, *keys_b, *vals_tmp, *radix_scratch;
    unsigned long long* total;
    size_t bytes;
};

BinWorkspace layout(char* base, long long n_pairs, long long capacity) {
    BinWorkspace w;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = base ? base + off : nullptr;
        off += (bytes + 255) & ~(size_t)255;
        return p;
    };
    w.total = (unsigned long long*)take(sizeof(unsigned long long));
    const long long blocks = (n_pairs + kThreads - 1) / kThreads;
    w.rects = (unsigned long long*)take(sizeof(unsigned long long) * (size_t)n_pairs);
    w.sums = (uint32_t*)take(sizeof(uint32_t) * (size_t)blocks);
    w.scan_scratch = (uint32_t*)take(sizeof(uint32_t) * scan_scratch_words(blocks));
    w.keys_a = (uint32_t*)take(sizeof(uint32_t) * (size_t)capacity);
    w.keys_b = (uint32_t*)take(sizeof(uint32_t) * (size_t)capacity);
    w.vals_tmp = (uint32_t*)take(sizeof(uint32_t) * (size_t)capacity);
    w.radix_scratch = (uint32_t*)take(sizeof(uint32_t) * radix_scratch_words(capacity));
    w.bytes = off;
    return w;
}

}  // namespace

int tile_size_of(const rf_raster_args& a) { return auto_tile(a); }

BatchWorkspace batch_layout(char* base, const rf_batch_sizes& z, long long capacity) {
    BatchWorkspace w;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = base ? base + off : nullptr;
        off += (bytes + 255) & ~(size_t)255;
        return p;
    };
    const long long sort_n = capacity > z.tiles ? capacity : z.tiles;
    w.rects = (unsigned long long*)take(sizeof(unsigned long long) * (size_t)z.pairs);
    w.sums = (uint32_t*)take(sizeof(uint32_t) * (size_t)z.pair_blocks);
    w.scan_scratch = (uint32_t*)take(sizeof(uint32_t) * scan_scratch_words(z.pair_blocks));
    w.keys_a = (uint32_t*)take(sizeof(uint32_t) * (size_t)capacity);
    w.keys_b = (uint32_t*)take(sizeof(uint32_t) * (size_t)capacity);
    w.vals_tmp = (uint32_t*)take(sizeof(uint32_t) * (size_t)capacity);
    w.radix_scratch = (uint32_t*)take(sizeof(uint32_t) * radix_scratch_words(sort_n));
    w.order_keys = (uint32_t*)take(sizeof(uint32_t) * (size_t)z.tiles);
    w.order_vals = (uint32_t*)take(sizeof(uint32_t) * (size_t)z.tiles);
    w.order_keys_b = (uint32_t*)take(sizeof(uint32_t) * (size_t)z.tiles);
    w.order_vals_b = (uint32_t*)take(sizeof(uint32_t) * (size_t)z.tiles);
    w.queue = (uint32_t*)take(sizeof(uint32_t) * 4);
    w.bytes = off;
    return w;
}

// The tile order is sorted by 8-bit keys: one pass when there are two tiles or more, so it
// starts in the _b buffers and ends in order_vals; a single tile is never moved.
const uint32_t* batch_tile_order(const BatchWorkspace& w, const rf_batch_sizes& z) {
    return z.tiles > 1 ? w.order_vals : w.order_vals_b;
}

}  // namespace rf

extern "C" int rf_bin_masks(const float* bounds, int32_t prim_count, float screen_transform, int32_t width,
                            int32_t height, int32_t bin_size, uint64_t* masks, void* stream) {
    using namespace rf;
    if (!bounds || !masks || prim_count < 0 || width < 1 || height < 1 || bin_size < 1) return RF_ERR_INVALID_ARG;
    if (!aligned16(bounds)) return RF_ERR_INVALID_ARG;
    BinGeometry g = {};
    g.width = width;
    g.height = height;
    g.B = bin_size;
    g.bdx = (width + bin_size - 1) / bin_size;
    g.bdy = (height + bin_size - 1) / bin_size;
    g.st = screen_transform;
    const int batches = (prim_count + RF_BATCH_PRIMITIVE_COUNT - 1) / RF_BATCH_PRIMITIVE_COUNT;
    cudaStream_t s = (cudaStream_t)stream;
    RF_TRY(cuda_status(cudaMemsetAsync(masks, 0, sizeof(uint64_t) * 4 * (size_t)g.bdx * g.bdy * batches, s)));
    if (prim_count == 0) return RF_OK;
    k_bin_masks<<<blocks_for(prim_count, kThreads), kThreads, 0, s>>>((const float4*)bounds, prim_count, g, batches,
                                                                      (unsigned long long*)masks);
    return launch_status();
}

extern "C" int rf_raster_tiles(const rf_raster_args* args, int32_t* tile_size, int32_t* tile_count) {
    using namespace rf;
    if (!args) return RF_ERR_INVALID_ARG;
    BinGeometry g;
    if (!make_geometry(*args, g)) return RF_ERR_INVALID_ARG;
    if (tile_size) *tile_size = g.T;
    if (tile_count) *tile_count = g.ntx * g.nty;
    return RF_OK;
}

extern "C" int rf_bin_workspace_size(const rf_raster_args* args, int64_t entry_capacity, size_t* bytes) {
    using namespace rf;
    if (!args || !bytes || entry_capacity < 0) return RF_ERR_INVALID_ARG;
    BinGeometry g;
    if (!make_geometry(*args, g)) return RF_ERR_INVALID_ARG;
    const long long n_pairs = (long long)args->path_count * (g.G - 1) * (g.G - 1) * g.maxW;
    *bytes = layout(nullptr, n_pairs, entry_capacity).bytes;
    return RF_OK;
}

extern "C" int rf_bin_tiles(const float* bounds, const float* vertexes, const rf_raster_args* args, void* workspace,
                            size_t workspace_bytes, uint32_t* tile_offsets, uint32_t* tile_entries,
                            int64_t entry_capacity, int64_t* entry_count, void* stream) {
    using namespace rf;
    if (!bounds || !vertexes || !args || !workspace || !tile_offsets || !entry_count || entry_capacity < 0)
        return RF_ERR_INVALID_ARG;
    if (!aligned16(bounds) || !aligned16(vertexes) || !aligned16(workspace)) return RF_ERR_INVALID_ARG;
    BinGeometry g;
    if (!make_geometry(*args, g)) return RF_ERR_INVALID_ARG;
    const long long n_pairs = (long long)args->path_count * (g.G - 1) * (g.G - 1) * g.maxW;
    BinWorkspace w = layout((char*)workspace, n_pairs, entry_capacity);
    if (w.bytes > workspace_bytes) return RF_ERR_INVALID_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    const int ntiles = g.ntx * g.nty;
    *entry_count = 0;
    RF_TRY(cuda_status(cudaMemsetAsync(w.total, 0, sizeof(unsigned long long), s)));
    const unsigned pair_blocks = blocks_for(n_pairs, kThreads);
    if (n_pairs > 0) {
        k_pair_count<<<pair_blocks, kThreads, 0, s>>>((const float4*)bounds, (const float4*)vertexes, n_pairs, g,
                                                      w.rects, w.sums, w.total);
        RF_TRY(launch_status());
        RF_TRY(exclusive_scan_u32(w.sums, w.sums, pair_blocks, w.scan_scratch, s));
    }
    unsigned long long total = 0;
    RF_TRY(cuda_status(cudaMemcpyAsync(&total, w.total, sizeof(total), cudaMemcpyDeviceToHost, s)));
    RF_TRY(cuda_status(cudaStreamSynchronize(s)));
    *entry_count = (int64_t)total;
    if (total > 0xfffffff0ull) return RF_ERR_NOT_SUPPORTED;
    if ((long long)total > entry_capacity || (total > 0 && !tile_entries)) return RF_ERR_WORKSPACE;
    if (total == 0) return cuda_status(cudaMemsetAsync(tile_offsets, 0, sizeof(uint32_t) * (ntiles + 1), s));
    int bits = 0;
    while ((1LL << bits) < ntiles) bits++;
    const int passes = total > 1 ? (bits + 7) / 8 : 0;  // (the sort moves nothing where there is one entry)
    // arrange the ping-pong buffers so that the sorted values land in tile_entries
    uint32_t* vals_first = (passes % 2 == 0) ? tile_entries : w.vals_tmp;
    uint32_t* vals_alt = (passes % 2 == 0) ? w.vals_tmp : tile_entries;
    RF_TRY(launch_chained(k_pair_emit, pair_blocks, kThreads, 0, s, w.rects, n_pairs, g.ntx, g.wide_bits, w.sums,
                          entry_capacity, w.keys_a, vals_first));
    bool in_alt = false;
    RF_TRY(radix_sort_pairs(w.keys_a, vals_first, w.keys_b, vals_alt, (long long)total, bits, w.radix_scratch,
                            &in_alt, s));
    const uint32_t* sorted_keys = in_alt ? w.keys_b : w.keys_a;
    return launch_chained(k_tile_offsets, blocks_for(32 * (long long)(ntiles + 1), kThreads), kThreads, 0, s, sorted_keys,
                          (long long)total, ntiles, tile_offsets);
}

namespace rf {
namespace {
struct OrderWorkspace {
    uint32_t *keys, *keys_b, *vals_b, *radix_scratch;
    size_t bytes;
};
OrderWorkspace order_layout(char* base, int tiles) {
    OrderWorkspace w;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* p = base ? base + off : nullptr;
        off += (bytes + 255) & ~(size_t)255;
        return p;
    };
    w.keys = (uint32_t*)take(sizeof(uint32_t) * (size_t)tiles);
    w.keys_b = (uint32_t*)take(sizeof(uint32_t) * (size_t)tiles);
    w.vals_b = (uint32_t*)take(sizeof(uint32_t) * (size_t)tiles);
    w.radix_scratch = (uint32_t*)take(sizeof(uint32_t) * radix_scratch_words(tiles));
    w.bytes = off;
    return w;
}
}  // namespace
}  // namespace rf

extern "C" int rf_tile_order_workspace_size(int32_t tile_count, size_t* bytes) {
    if (!bytes || tile_count < 1) return RF_ERR_INVALID_ARG;
    *bytes = rf::order_layout(nullptr, tile_count).bytes;
    return RF_OK;
}

extern "C" int rf_tile_order(const uint32_t* tile_offsets, int32_t tile_count, void* workspace,
                             size_t workspace_bytes, uint32_t* tile_order, void* stream) {
    using namespace rf;
    if (!tile_offsets || !workspace || !tile_order || tile_count < 1) return RF_ERR_INVALID_ARG;
    if (!aligned16(workspace)) return RF_ERR_INVALID_ARG;
    OrderWorkspace w = order_layout((char*)workspace, tile_count);
    if (w.bytes > workspace_bytes) return RF_ERR_INVALID_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    if (tile_count <= kOrderBlockTiles)
        return launch_chained(k_tile_order, 1, kOrderThreads, 0, s, tile_offsets, tile_count, tile_order);
    RF_TRY(launch_chained(k_tile_order_keys, blocks_for(tile_count, kThreads), kThreads, 0, s, tile_offsets, tile_count,
                          w.keys_b, w.vals_b));
    // two or more tiles and 8 key bits: exactly one pass, so the sorted pairs land in the
    // alternate buffers (keys, tile_order)
    bool in_alt = false;
    return radix_sort_pairs(w.keys_b, w.vals_b, w.keys, tile_order, tile_count, kOrderKeyBits, w.radix_scratch,
                            &in_alt, s);
}

extern "C" int rf_batch_workspace_size(const rf_batch_sizes* sizes, int64_t entry_capacity, size_t* bytes) {
    using namespace rf;
    if (!sizes || !bytes || entry_capacity < 0) return RF_ERR_INVALID_ARG;
    *bytes = batch_layout(nullptr, *sizes, entry_capacity).bytes;
    return RF_OK;
}

extern "C" int rf_bin_tiles_batch(const rf_frame* frames, const rf_batch_sizes* sizes, const float* bounds,
                                  const float* vertexes, void* workspace, size_t workspace_bytes,
                                  uint32_t* tile_offsets, uint32_t* tile_entries, int64_t entry_capacity,
                                  uint64_t* entry_total, void* stream) {
    using namespace rf;
    if (!frames || !sizes || !bounds || !vertexes || !workspace || !tile_offsets || !entry_total ||
        entry_capacity < 1 || !tile_entries)
        return RF_ERR_INVALID_ARG;
    if (!aligned16(bounds) || !aligned16(vertexes) || !aligned16(workspace)) return RF_ERR_INVALID_ARG;
    const rf_batch_sizes& z = *sizes;
    if (entry_capacity > 0xfffffff0LL || z.tiles < 1 || z.tiles > (1 << 30) || z.pair_blocks > 0x7fffffffLL)
        return RF_ERR_NOT_SUPPORTED;
    BatchWorkspace w = batch_layout((char*)workspace, z, entry_capacity);
    if (w.bytes > workspace_bytes) return RF_ERR_INVALID_ARG;
    cudaStream_t s = (cudaStream_t)stream;
    RF_TRY(cuda_status(cudaMemsetAsync(entry_total, 0, sizeof(uint64_t), s)));
    if (z.pair_blocks > 0) {
        k_pair_count_batch<<<(unsigned)z.pair_blocks, kThreads, 0, s>>>(
            frames, z.frame_count, (const float4*)bounds, (const float4*)vertexes, w.rects, w.sums,
            (unsigned long long*)entry_total);
        RF_TRY(launch_status());
        RF_TRY(exclusive_scan_u32(w.sums, w.sums, z.pair_blocks, w.scan_scratch, s));
    }
    int bits = 0;
    while ((1LL << bits) <= z.tiles) bits++;  // keys 0 .. tiles (tiles = padding)
    const int passes = (entry_capacity > 1) ? (bits + 7) / 8 : 0;
    uint32_t* vals_first = (passes % 2 == 0) ? tile_entries : w.vals_tmp;
    uint32_t* vals_alt = (passes % 2 == 0) ? w.vals_tmp : tile_entries;
    if (z.pair_blocks > 0) {
        RF_TRY(launch_chained(k_pair_emit_batch, (unsigned)z.pair_blocks, kThreads, 0, s, frames, z.frame_count, w.rects,
                              w.sums, entry_capacity, w.keys_a, vals_first));
    }
    RF_TRY(launch_chained(k_pad_entries, std::min(blocks_for(entry_capacity, kThreads), 2048u), kThreads, 0, s,
                          (const unsigned long long*)entry_total, entry_capacity, (uint32_t)z.tiles, w.keys_a,
                          vals_first));
    bool in_alt = false;
    RF_TRY(radix_sort_pairs(w.keys_a, vals_first, w.keys_b, vals_alt, entry_capacity, bits, w.radix_scratch,
                            &in_alt, s));
    const uint32_t* sorted_keys = in_alt ? w.keys_b : w.keys_a;
    RF_TRY(launch_chained(k_tile_offsets, blocks_for(32 * (long long)(z.tiles + 1), kThreads), kThreads, 0, s, sorted_keys,
                          entry_capacity, z.tiles, tile_offsets));
    // the raster's work queue: tiles by decreasing entry count
    if (z.tiles <= kOrderBlockTiles)
        return launch_chained(k_tile_order, 1, kOrderThreads, 0, s, tile_offsets, z.tiles,
                              (uint32_t*)batch_tile_order(w, z));
    RF_TRY(launch_chained(k_tile_order_keys, blocks_for(z.tiles, kThreads), kThreads, 0, s, tile_offsets, z.tiles,
                          w.order_keys_b, w.order_vals_b));
    RF_TRY(radix_sort_pairs(w.order_keys_b, w.order_vals_b, w.order_keys, w.order_vals, z.tiles, kOrderKeyBits,
                            w.radix_scratch, &in_alt, s));
    return RF_OK;
}
