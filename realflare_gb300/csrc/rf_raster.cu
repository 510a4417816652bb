// rf_raster.cu — the ghost rasteriser.
//
// Per pixel the result is the reference's (realflare/api/tasks/cl/rasterizing.cl:524-663):
// the sum over visible primitives (in primitive order), wavelength pairs and sub-wavelength
// steps of XYZ(lambda) * fragment, where a fragment is the n-rook sample coverage of the
// integer quad (intersect_quad 55-93) times the mean-value interpolated ghost texture,
// housing falloff, area intensity and coating reflectance (compute_barycentric_quad
// 95-148, fragment_shader 471-506, mix_vertex 509-522), scaled and converted to AP1
// (color.cl:3-10) and written y-flipped.
//
// GB300 organisation (k_raster): one CTA per T x T tile; warps take the tile's blocks of pixels.
// The tile's list from rf_bin_tiles holds (primitive, wavelength pair) entries in increasing
// order. Entries are expanded in batches into shared-memory records (one per sub-wavelength
// step): the mixed corners, the five edge functions as exact FP32 plane coefficients relative to
// the tile, the integer bounds and the mixed attributes, set up once. Every pixel then walks the
// records in order, so its sum runs in the reference's order; a pixel whose samples lie
// outside a record's integer bounds skips it (exact: with vertex and sample coordinates
// below 2^14 the edge functions cannot wrap, and the quad test then never accepts a
// sample outside the bounds; records beyond that range are tested at every pixel, in wrapping
// int32, WildEdges).
//
// k_raster_masks is the literal per-pixel loop over the reference's bin masks, used for
// parity checks of the binner and the rasteriser.
#include <stddef.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <type_traits>
#include <vector>

#include "rf_common.cuh"

namespace rf {
int tile_size_of(const rf_raster_args& a);

namespace {

// Tuning knobs (compile-time): records per shared-memory batch, resident blocks per SM
// requested from the register allocator.
#ifndef RF_RASTER_BATCH
#define RF_RASTER_BATCH 64
#endif
#ifndef RF_RASTER_MIN_BLOCKS
#define RF_RASTER_MIN_BLOCKS 4
#endif
#ifndef RF_RASTER_MIN_BLOCKS_S1  // the one-sample kernel needs fewer registers
#define RF_RASTER_MIN_BLOCKS_S1 4
#endif
constexpr int kBatchRecords = RF_RASTER_BATCH;
// Pixels of a column a lane of the one-sample kernels shades: two where a tile has enough blocks
// of 8 x 8 pixels for the CTA's 8 warps (32-pixel tiles: 16; production frame 102.0 ms with one
// pixel, 90.4 with two), one in 16-pixel tiles.
#ifndef RF_RASTER_PIX32
#define RF_RASTER_PIX32 2
#endif
#ifndef RF_RASTER_PIX16
#define RF_RASTER_PIX16 1
#endif

#ifdef RF_RASTER_STATS
// Work counters of the statistics build (never compiled into the product library):
// record iterations per block, those of whole-block records, fragments, fragments of
// whole-block records, block visits, fragments whose smoothstep factor is 0 (rrel >= 1),
// record iterations where that holds for every shaded pixel of the block (those two with
// more than one sample per pixel), warp steps of the one-sample shading loop.
constexpr int kRasterStats = 8;
__device__ unsigned long long g_raster_stats[kRasterStats];
#define RF_STAT(stmt) stmt
#else
#define RF_STAT(stmt)
#endif

// Packed FP32 (f2, rf_common.cuh) with denormals flushed as in the rest of this unit: shading is bound by
// instruction issue, and a packed instruction does two corners' work in one issue slot.
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 d;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    f2 d;
    asm("sub.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Every group the shading loop reads starts on a 16-byte boundary and is read with
// 16-byte shared-memory loads that yield two register pairs. Values of the four corners are
// stored even corners first (0, 2, 1, 3), so that one packed operation serves corners 0 and 2
// (or edges 0 and 2) and the next one corners 1 and 3, without register moves. Records are
// 240 bytes apart (15 x 16): where the lanes of a warp read 32 different records at one offset
// (the block selection), each group of 8 lanes then reads 8 different 16-byte bank groups
// instead of one.
struct alignas(16) Rec {
    int bb[4];       // xmin, xmax, ymin, ymax
    float col[4];    // the record's XYZ weight (1, 1, 1 with one wavelength); [3]: 0 when the housing
                     // falloff is 1 and no clamp acts on any covered pixel (inside_housing), else 1
    float xy[12];    // corner positions relative to the tile, exact floats: x0 x2, x1 x3, y0 y2, y1 y3,
                     // x2 x0, y2 y0
    float uv[8];     // ghost texel coordinates: u0 u2, u1 u3, v0 v2, v1 v3, see store_corner
    float rs[4];     // (rrel - 1) / (0.95 - 1): smoothstep(1, 0.95, rrel)'s ramp before clamping
    float inten[4], refl[4];
    // biased edge functions A y + B x + C in samples relative to the tile (exact, see finish_record):
    // A of edges 01 12, B 01 12, C 01 12, A 23 30, B 23 30, C 23 30, then A B C of edge 20
    float ef[15];
    int flags;       // 1: bounds rejection and ef are exact; 2: adds nothing (collinear, or zero_record)
    float ext[4];    // edges 01 12 23 30: half the edge function's range over a block
    // in ef's place: the mixed vertex positions, sample space (x0, y0, ..., x3, y3), while the record is
    // built, and, where ef is not exact (flags & 1 clear), the same coefficients as integers
    __device__ __forceinline__ int* q() { return reinterpret_cast<int*>(ef); }
    __device__ __forceinline__ const int* q() const { return reinterpret_cast<const int*>(ef); }
};
static_assert(sizeof(Rec) == 240 && offsetof(Rec, bb) == 0 && offsetof(Rec, col) % 16 == 0 &&
                  offsetof(Rec, xy) % 16 == 0 && offsetof(Rec, uv) % 16 == 0 && offsetof(Rec, rs) % 16 == 0 &&
                  offsetof(Rec, inten) % 16 == 0 && offsetof(Rec, refl) % 16 == 0 &&
                  offsetof(Rec, ef) % 16 == 0 && offsetof(Rec, flags) == offsetof(Rec, ef) + 15 * sizeof(int) &&
                  offsetof(Rec, ext) % 16 == 0,
              "records are read with 16-byte loads");
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ int4 ld4i(const int* p) { return *reinterpret_cast<const int4*>(p); }
__device__ __forceinline__ void ld2(const float* p, f2& a, f2& b) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    a = v.x, b = v.y;
}
// where corner k's values sit among the four (0, 2, 1, 3)
__device__ __forceinline__ int corner_slot(int k) { return ((k & 1) << 1) | (k >> 1); }

struct RasterParams {
    int width, height, T, ntx, S, W, WS, G, maxW;
    float intensity, ghost_scale;
    int ghost_w, ghost_h;
    bool safe_screen;
    bool ghost_large;  // the ghost texture has a side of 2^22 texels or more, or 2^31 texels (ghost_sample)
    unsigned long long ghost_tex;  // texture object over the ghost texture (the kTex kernels)
};

__device__ __forceinline__ bool top_left(int ax, int ay, int bx, int by) {
    int ex = wsub(bx, ax), ey = wsub(by, ay);
    return (ey == 0 && ex > 0) || ey > 0;
}

__device__ __forceinline__ int32_t edge_i(int ax, int ay, int bx, int by, int cx, int cy) {
    return wsub(wmul(wsub(ax, bx), wsub(cy, ay)), wmul(wsub(ay, by), wsub(cx, ax)));
}

__device__ __forceinline__ void edge_coeffs(int ax, int ay, int bx, int by, int* e) {
    // (a.x - b.x) * (p.y - a.y) - (a.y - b.y) * (p.x - a.x) + bias, as A*p.y + B*p.x + C
    const int A = wsub(ax, bx);
    const int dy = wsub(ay, by);
    e[0] = A;
    e[1] = wsub(0, dy);
    e[2] = wadd(wsub(wmul(dy, ax), wmul(A, ay)), top_left(ax, ay, bx, by) ? 0 : -1);
}

// intersect_quad (rasterizing.cl:55-93) of the sample (px, py), in the reference's wrapping int32
__device__ __forceinline__ bool inside_exact(const int* q, int px, int py) {
    bool w[5];
#pragma unroll
    for (int i = 0; i < 5; i++) {
        const int a = i < 4 ? i : 2, b = i < 4 ? (i + 1) & 3 : 0;
        int e[3];
        edge_coeffs(q[2 * a], q[2 * a + 1], q[2 * b], q[2 * b + 1], e);
        w[i] = wadd(wadd(wmul(e[0], py), wmul(e[1], px)), e[2]) >= 0;
    }
    const bool front = (w[4] && w[0] && w[1] && (w[2] || w[3])) || (!w[4] && w[2] && w[3] && (w[0] || w[1]));
    const bool back = (!w[4] && !w[0] && !w[1] && (!w[2] || !w[3])) || (w[4] && !w[2] && !w[3] && (!w[0] || !w[1]));
    return front || back;
}

// The same decision from the signs of the five edge values (sign bit set: the value is negative),
// in bit 31 of the result, set where the sample is outside: with w20 the front and back
// conditions say that (w01 and w12) equals (w23 or w30), without it that (w23 and w30) equals
// (w01 or w12).
__device__ __forceinline__ unsigned outside_sign(unsigned n01, unsigned n12, unsigned n23, unsigned n30,
                                                 unsigned n20) {
    const unsigned x1 = (n01 | n12) ^ (n23 & n30), x0 = (n23 | n30) ^ (n01 & n12);
    return (~n20 & x1) | (n20 & x0);
}

// The integer edge functions of a record with flags & 1 clear, and whether the sample (px, py) is inside by them, in
// wrapping int32. (Formed anew from the corners at every sample, they took half of the rasters at 8 samples, whose
// coordinates often pass the exact range: 1920 x 1080, 24 surfaces, 60 paths, 136 -> 57 ms; 16 surfaces,
// 40 paths, 4.71 -> 3.13 ms.)
struct WildEdges {
    int4 v0, v1, v2, v3;  // in ef's order: A of edges 01 12, B 01 12, C 01 12, A 23 30, ...
    __device__ __forceinline__ explicit WildEdges(const Rec& r)
        : v0(ld4i(r.q())), v1(ld4i(r.q() + 4)), v2(ld4i(r.q() + 8)), v3(ld4i(r.q() + 12)) {}
    __device__ __forceinline__ bool inside(int px, int py) const {
        auto value = [&](int a, int b, int c) { return (unsigned)wadd(wadd(wmul(a, py), wmul(b, px)), c); };
        return (int)outside_sign(value(v0.x, v0.z, v1.x), value(v0.y, v0.w, v1.y), value(v1.z, v2.x, v2.z),
                                 value(v1.w, v2.y, v2.w), value(v3.x, v3.y, v3.z)) >= 0;
    }
};

// A record's edge functions in registers.
struct Edges {
    f2 a0, b0, c0, a1, b1, c1;  // edges (01, 12) and (23, 30)
    float a20, b20, c20;
    int flags;
};
__device__ __forceinline__ void load_edges(const Rec& r, Edges& e) {
    ld2(r.ef, e.a0, e.b0);
    ld2(r.ef + 4, e.c0, e.a1);
    ld2(r.ef + 8, e.b1, e.c1);
    const float4 d = ld4(r.ef + 12);
    e.a20 = d.x, e.b20 = d.y, e.c20 = d.z, e.flags = __float_as_int(d.w);
}
// The sample at tile-relative coordinates x = (x, x), y = (y, y), for records with flags & 1: the
// edge values are exact integers (an exact zero is +0), so their signs are the reference's.
__device__ __forceinline__ bool inside_at(f2 e0, f2 e1, float e2) {
    return (int)outside_sign((unsigned)e0, (unsigned)(e0 >> 32), (unsigned)e1, (unsigned)(e1 >> 32),
                             __float_as_uint(e2)) >= 0;
}
__device__ __forceinline__ bool inside(const Edges& e, f2 x, f2 y) {
    return inside_at(fma2(e.a0, y, fma2(e.b0, x, e.c0)), fma2(e.a1, y, fma2(e.b1, x, e.c1)),
                     fmaf(e.a20, lo2(y), fmaf(e.b20, lo2(x), e.c20)));
}

// Coverage of a block's samples (centre (xc, yc) as pairs, tile-relative, half extents
// hx, hy) by a record with flags & 1: each edge value is linear in the sample, so its sign is
// constant over the block when its extremes there (centre value -+ ext) agree, and then
// inside() is constant too. Returns 0 (no sample inside), 2 (every sample inside) or 1 (mixed
// or undecided). Where a centre value is not exact (|C| near its clamp) it is far from 0.
__device__ __forceinline__ int rect_coverage(const Rec& r, f2 xc, f2 yc, float hx, float hy) {
    Edges e;
    load_edges(r, e);
    f2 x0, x1;
    ld2(r.ext, x0, x1);
    const f2 e0 = fma2(e.a0, yc, fma2(e.b0, xc, e.c0)), e1 = fma2(e.a1, yc, fma2(e.b1, xc, e.c1));
    const float e2 = fmaf(e.a20, lo2(yc), fmaf(e.b20, lo2(xc), e.c20));
    const float x2 = fmaf(fabsf(e.a20), hy, fabsf(e.b20) * hx);
    const f2 l0 = sub2(e0, x0), l1 = sub2(e1, x1), h0 = add2(e0, x0), h1 = add2(e1, x1);
    const unsigned l2 = __float_as_uint(e2 - x2), h2 = __float_as_uint(e2 + x2);
    // mixed: the lowest value negative, the highest not
    const unsigned mixed = ((unsigned)l0 & ~(unsigned)h0) | ((unsigned)(l0 >> 32) & ~(unsigned)(h0 >> 32)) |
                           ((unsigned)l1 & ~(unsigned)h1) | ((unsigned)(l1 >> 32) & ~(unsigned)(h1 >> 32)) |
                           (l2 & ~h2);
    const unsigned out = outside_sign((unsigned)l0, (unsigned)(l0 >> 32), (unsigned)l1, (unsigned)(l1 >> 32), l2);
    return (int)mixed < 0 ? 1 : ((int)out < 0 ? 0 : 2);
}

// Mean-value weights (compute_barycentric_quad, rasterizing.cl:95-148) at the integer
// sample point (px, py), relative to the tile. The coordinates s_i = q_i - p are exact floats; the
// products a_i, d_i, |s_i|^2 are exact integers wherever |s| < 4096, so fused multiply-adds give
// the reference's values there. Where a_i is 0 the reference divides the rounding residue
// of r_i r_j - d_i by 1e-3: that tangent is evaluated with the reference's exact FP32
// operations (correctly rounded square roots, product, difference, quotient). Elsewhere
// the tangents and the divisions by r_i and by the weight sum use reciprocal and
// reciprocal-square-root instructions (a few ulps).
//
// px is (x, x), py the (y, y) of kN pixels in one column, whose chains run side by side and share
// the terms in x. Corners 0 and 2 and corners 1 and 3 go through packed operations; the cross
// products' second terms are formed from negated odd corners (p - q instead of q - p), because a
// packed fused multiply-add cannot negate an operand. Returns the weights of corners (0, 2) in we
// and (1, 3) in wo for the pixels marked in `need`, and sets `general` where they may have mixed
// signs inside a convex quad (the special cases).
//
// y_last: which of the two products of d_i and |s_i|^2 is fused, and so what they round to where |s| >=
// 4096: that in y with one sample per pixel (the pixels of a column share those in x; the other order
// takes 95.4 instead of 89.4 ms on the production frame), that in x with several, where such
// distances are less rare (the scalar form's roundings). It depends on the samples alone, so that a
// frame's image is the same in tiles of either size and in a batch.
struct CornerTerms {  // in x, shared by the pixels of a column
    f2 xe, xs, nxo, xe_nxo, xs_nxo, xe_xe, xo_xo, qye, qyo, qys;
    __device__ __forceinline__ CornerTerms(const Rec& rec, f2 px) {
        f2 qxe, qxo, qxs;
        ld2(rec.xy, qxe, qxo);
        ld2(rec.xy + 4, qye, qyo);
        ld2(rec.xy + 8, qxs, qys);
        xe = sub2(qxe, px), xs = sub2(qxs, px), nxo = sub2(px, qxo);
        xe_nxo = mul2(xe, nxo), xs_nxo = mul2(xs, nxo), xe_xe = mul2(xe, xe), xo_xo = mul2(nxo, nxo);
    }
};
struct PixelTerms {
    f2 a02, na13, nd02, nd13, r2e, r2o, ire, iro, t02, nt13;  // a0 a2, -a1 -a3, -d0 -d2, -d1 -d3, ...
    __device__ __forceinline__ PixelTerms(const CornerTerms& c, f2 py, bool y_last) {
        const f2 ye = sub2(c.qye, py), ys = sub2(c.qys, py), yo = sub2(c.qyo, py), nyo = sub2(py, c.qyo);
        a02 = fma2(c.xe, yo, mul2(c.nxo, ye));
        na13 = fma2(c.xs, yo, mul2(c.nxo, ys));
        if (y_last) {  // the products in x are shared
            nd02 = fma2(ye, nyo, c.xe_nxo), nd13 = fma2(ys, nyo, c.xs_nxo);
            r2e = fma2(ye, ye, c.xe_xe), r2o = fma2(yo, yo, c.xo_xo);
        } else {
            nd02 = fma2(c.xe, c.nxo, mul2(ye, nyo)), nd13 = fma2(c.xs, c.nxo, mul2(ys, nyo));
            r2e = fma2(c.xe, c.xe, mul2(ye, ye)), r2o = fma2(c.nxo, c.nxo, mul2(yo, yo));
        }
        ire = pk(rsqrtf(lo2(r2e)), rsqrtf(hi2(r2e))), iro = pk(rsqrtf(lo2(r2o)), rsqrtf(hi2(r2o)));
        const f2 re = mul2(r2e, ire), ro = mul2(r2o, iro);
        const f2 n02 = fma2(re, ro, nd02);
        const f2 n13 = pk(fmaf(lo2(ro), hi2(re), lo2(nd13)), fmaf(hi2(ro), lo2(re), hi2(nd13)));
        t02 = mul2(n02, pk(rcp_approx(lo2(a02)), rcp_approx(hi2(a02))));
        nt13 = mul2(n13, pk(rcp_approx(lo2(na13)), rcp_approx(hi2(na13))));
    }
};

// The weights where the common form failed: a vertex on the sample point, an edge's line through
// it (that tangent in the reference's exact operations), or a weight sum of 0, infinity or NaN
// (normalised weights would be infinite or NaN, their intensity and reflectance NaN or 0 and so
// the clamped products 0).
__device__ __forceinline__ void special_weights(const Rec& rec, f2 px, f2 py, bool y_last, f2& we, f2& wo) {
    // (evaluated anew, not kept live from the common form: the empty asm hides that they are the same)
    asm("" : "+l"(px), "+l"(py));
    const PixelTerms p(CornerTerms(rec, px), py, y_last);
    const float r2[4] = {lo2(p.r2e), lo2(p.r2o), hi2(p.r2e), hi2(p.r2o)};
    if (r2[0] == 0.0f || r2[1] == 0.0f || r2[2] == 0.0f || r2[3] == 0.0f) {  // one-hot on the first such vertex
        const int k = r2[0] == 0.0f ? 0 : (r2[1] == 0.0f ? 1 : (r2[2] == 0.0f ? 2 : 3));
        we = pk(k == 0 ? 1.0f : 0.0f, k == 2 ? 1.0f : 0.0f);
        wo = pk(k == 1 ? 1.0f : 0.0f, k == 3 ? 1.0f : 0.0f);
        return;
    }
    const float a[4] = {lo2(p.a02), lo2(p.na13), hi2(p.a02), hi2(p.na13)};
    const float nd[4] = {lo2(p.nd02), lo2(p.nd13), hi2(p.nd02), hi2(p.nd13)};
    float t[4] = {lo2(p.t02), -lo2(p.nt13), hi2(p.t02), -hi2(p.nt13)};
#pragma unroll
    for (int i = 0; i < 4; i++)
        if (a[i] == 0.0f)
            t[i] = __fdiv_rn(__fadd_rn(__fmul_rn(__fsqrt_rn(r2[i]), __fsqrt_rn(r2[(i + 1) & 3])), nd[i]), 1e-3f);
    we = mul2(pk(t[3] + t[0], t[1] + t[2]), p.ire);
    wo = mul2(pk(t[0] + t[1], t[2] + t[3]), p.iro);
    const float sum = (lo2(we) + hi2(we)) + (lo2(wo) + hi2(wo)), inv = rcp_approx(sum);
    const bool ok = sum * inv > 0.5f;
    const f2 inv2 = pk(inv, inv);
    we = ok ? mul2(we, inv2) : 0;
    wo = ok ? mul2(wo, inv2) : 0;
}

template <int kN>
__device__ __forceinline__ void mean_value_weights(const Rec& rec, f2 px, const f2 (&py)[kN], const bool (&need)[kN],
                                                   bool y_last, f2 (&we)[kN], f2 (&wo)[kN], float& general) {
    const CornerTerms c(rec, px);
    // The common case first. a_i are integers (differences of products of integers): when
    // none is 0 each |a_i| >= 1 and every term below is finite, so the weight sum is finite.
    // An a_i of 0 makes t_i infinite or NaN, and a vertex on the sample point (r2_i = 0)
    // makes r_i NaN; either way sum * (1 / sum) is not near 1, and only then are the weights
    // redone with the reference's special cases.
    bool bad = false, ok[kN];
#pragma unroll
    for (int i = 0; i < kN; i++) {
        const PixelTerms p(c, py[i], y_last);
        wo[i] = mul2(sub2(p.t02, p.nt13), p.iro);                                                   // w1, w3
        we[i] = mul2(pk(lo2(p.t02) - hi2(p.nt13), hi2(p.t02) - lo2(p.nt13)), p.ire);                // w0, w2
        const f2 s2 = add2(we[i], wo[i]);
        const float sum = lo2(s2) + hi2(s2), inv = rcp_approx(sum);
        ok[i] = !need[i] || sum * inv > 0.5f;
        bad = bad || !ok[i];
        const f2 inv2 = pk(inv, inv);
        we[i] = mul2(we[i], inv2);
        wo[i] = mul2(wo[i], inv2);
    }
    if (bad) {
        general = 1.0f;
#pragma unroll
        for (int i = 0; i < kN; i++)
            if (!ok[i]) special_weights(rec, px, py[i], y_last, we[i], wo[i]);
    }
}
__device__ __forceinline__ void mean_value_weights(const Rec& rec, f2 px, f2 py, bool y_last, f2& we, f2& wo,
                                                   float& general) {
    const f2 p1[1] = {py};
    const bool need[1] = {true};
    f2 e1[1], o1[1];
    mean_value_weights<1>(rec, px, p1, need, y_last, e1, o1, general);
    we = e1[0];
    wo = o1[0];
}
// sum of weight x value over the corners, values even corners first
__device__ __forceinline__ float blend4(f2 we, f2 wo, const float* v) {
    f2 e, o;
    ld2(v, e, o);
    const f2 s = fma2(wo, o, mul2(we, e));
    return lo2(s) + hi2(s);
}

// Bilinear ghost sample (read_imagef LINEAR, CLAMP -> border 0, rasterizing.cl:483-485) at texel
// coordinates t = uv * size - 0.5, given less half a texel: (u, v) = t - 0.5. The nearest integers
// of those are the footprint's first texel (where t is an integer the footprint before it may
// be taken, with a fraction of 1: the same value), found by adding and subtracting 1.5 * 2^23,
// in packed operations (a floor would go to the same unit as the reciprocals). Returns the
// footprint's centre (i0 + 1, j0 + 1) and the fractions (a, b). Coordinates beyond 2^22 do not
// round to integers, but their texels are all outside a texture with sides below 2^22.
__device__ __forceinline__ void ghost_footprint(f2 uv, f2& centre, f2& frac) {
    const f2 big = pk(12582912.0f, 12582912.0f), big1 = pk(12582911.0f, 12582911.0f), half3 = pk(1.5f, 1.5f);
    centre = sub2(add2(uv, big), big1);
    frac = add2(sub2(uv, centre), half3);
}
// The specification's (1-a)(1-b) t00 + a(1-b) t10 + (1-a) b t01 + a b t11, as three interpolations
// (the same value up to rounding).
__device__ __forceinline__ float ghost_blend(float t00, float t10, float t01, float t11, f2 frac) {
    const float a = lo2(frac), b = hi2(frac);
    const float top = fmaf(a, t10 - t00, t00), bottom = fmaf(a, t11 - t01, t01);
    return fmaf(b, bottom - top, top);
}
// The footprint's texels, the first one (i0, j0), by loads; large: past 32-bit offsets.
__device__ __forceinline__ void ghost_texels(const float* __restrict__ tex, int w, int h, bool large, int i0, int j0,
                                             float& t00, float& t10, float& t01, float& t11) {
    const int i1 = wadd(i0, 1), j1 = wadd(j0, 1);
    if (!large && (unsigned)i0 < (unsigned)(w - 1) && (unsigned)j0 < (unsigned)(h - 1)) {
        // all four texels inside (the common case)
        const float* q = tex + (j0 * w + i0);
        t00 = __ldg(q);
        t10 = __ldg(q + 1);
        t01 = __ldg(q + w);
        t11 = __ldg(q + w + 1);
    } else {
        const bool i0_in = (unsigned)i0 < (unsigned)w, i1_in = (unsigned)i1 < (unsigned)w;
        const bool j0_in = (unsigned)j0 < (unsigned)h, j1_in = (unsigned)j1 < (unsigned)h;
        // load from clamped (always valid) addresses, then zero the texels outside the image
        const int ia = min(max(i0, 0), w - 1), ib = min(max(i1, 0), w - 1);
        const float* row0 = tex + (size_t)min(max(j0, 0), h - 1) * w;
        const float* row1 = tex + (size_t)min(max(j1, 0), h - 1) * w;
        t00 = (i0_in && j0_in) ? __ldg(row0 + ia) : 0.0f;
        t10 = (i1_in && j0_in) ? __ldg(row0 + ib) : 0.0f;
        t01 = (i0_in && j1_in) ? __ldg(row1 + ia) : 0.0f;
        t11 = (i1_in && j1_in) ? __ldg(row1 + ib) : 0.0f;
    }
}
// How a kernel looks the ghost texture up: by loads; by gathers from a texture object; by loads from a texture of any
// size (RasterParams.ghost_large; the test per fragment costs 1.5 % of the kernel).
constexpr int kLoads = 0, kGather = 1, kAnyLoads = 2;
// The same texels through a texture object over them (float, pitch-linear, border address
// mode): tex2Dgather at the footprint's centre, exactly half a texel from every footprint
// boundary, returns texels (i0, j0 + 1), (i0 + 1, j0 + 1), (i0 + 1, j0), (i0, j0) in x, y, z, w, and
// 0 for texels outside the image; one texture instruction instead of the bounds test, the
// address arithmetic and four loads. The values, and so the interpolation, are the loads'. u and v
// are finite: the weights are, and records with a texel coordinate that is not are left out
// (zero_record).
template <int kTex>
__device__ __forceinline__ float ghost_sample(const float* __restrict__ tex, const RasterParams& p, f2 uv) {
    f2 centre, frac;
    ghost_footprint(uv, centre, frac);
    float t00, t10, t01, t11;
    if (kTex == kGather) {
        const float4 g = tex2Dgather<float4>((cudaTextureObject_t)p.ghost_tex, lo2(centre), hi2(centre), 0);
        t00 = g.w, t10 = g.z, t01 = g.x, t11 = g.y;
    } else {
        int i0 = wsub(cvt_rz_sat(lo2(centre)), 1), j0 = wsub(cvt_rz_sat(hi2(centre)), 1);
        const bool large = kTex == kAnyLoads && p.ghost_large;
        if (large) {  // sides past ghost_footprint's range (texture objects have no such sides)
            const float u = lo2(uv) + 0.5f, v = hi2(uv) + 0.5f, fu = floorf(u), fv = floorf(v);
            i0 = cvt_rz_sat(fu), j0 = cvt_rz_sat(fv);
            frac = pk(u - fu, v - fv);
        }
        ghost_texels(tex, p.ghost_w, p.ghost_h, large, i0, j0, t00, t10, t01, t11);
    }
    return ghost_blend(t00, t10, t01, t11, frac);
}

// fragment_shader (rasterizing.cl:471-506) times the hit count. The texture coordinate
// ((uv / scale + 1) / 2) * size - 0.5, less the half texel of ghost_footprint, is evaluated as
// uv * tex_scale + tex_offset.
struct FragmentConsts {
    float tsx, tox, tsy, toy;  // texel coordinate scale and offset per axis
};
template <int kTex, int kN>
__device__ __forceinline__ void fragment_fast(const Rec& r, const f2 (&we)[kN], const f2 (&wo)[kN],
                                              const float* __restrict__ ghost, const RasterParams& p, float general,
                                              float (&f)[kN]) {
    float gi[kN], ai[kN], ci[kN];
#pragma unroll
    for (int i = 0; i < kN; i++) {
        const float u = blend4(we[i], wo[i], r.uv), v = blend4(we[i], wo[i], r.uv + 4);
        gi[i] = ghost_sample<kTex>(ghost, p, pk(u, v));
        ai[i] = blend4(we[i], wo[i], r.inten);
        ci[i] = blend4(we[i], wo[i], r.refl);
    }
    if (general != 0.0f) {
#pragma unroll
        for (int i = 0; i < kN; i++) {
            // smoothstep(1, 0.95, rrel): the ramp (rrel - 1) / (0.95 - 1) is linear in rrel, so the
            // corners' ramps interpolate to the fragment's (the weights sum to one)
            const float st = __saturatef(blend4(we[i], wo[i], r.rs));
            gi[i] *= st * st * (3.0f - 2.0f * st);
            ai[i] = fmaxf(ai[i], 0.0f);
            ci[i] = fmaxf(ci[i], 0.0f);
        }
    }
#pragma unroll
    for (int i = 0; i < kN; i++) f[i] = gi[i] * ai[i] * ci[i];
}
template <int kTex = kAnyLoads>
__device__ __forceinline__ float fragment_fast(const Rec& r, f2 we, f2 wo, const float* __restrict__ ghost,
                                               const RasterParams& p, float general) {
    const f2 e1[1] = {we}, o1[1] = {wo};
    float f[1];
    fragment_fast<kTex, 1>(r, e1, o1, ghost, p, general, f);
    return f[0];
}

__host__ __device__ inline FragmentConsts fragment_consts(const RasterParams& p, double shift = 1.0) {
    FragmentConsts fc;
    const double sx = 0.5 / p.ghost_scale * p.ghost_w, sy = 0.5 / p.ghost_scale * p.ghost_h;
    fc.tsx = (float)sx;
    fc.tsy = (float)sy;
    fc.tox = (float)(0.5 * p.ghost_w - shift);
    fc.toy = (float)(0.5 * p.ghost_h - shift);
    return fc;
}

// 1 / (0.95 - 1), the smoothstep ramp's slope (fragment_shader, rasterizing.cl:487-488)
constexpr float kRampScale = 1.0f / (0.95f - 1.0f);

// Corner k of entry `entry` at the pair's two wavelengths: vertex words a0, a1 (first
// wavelength) and b0, b1 (second).
struct CornerLoad {
    float4 a0, a1, b0, b1;
};
__device__ __forceinline__ void load_corner(const float4* __restrict__ vtx, uint32_t entry, int k,
                                            const RasterParams& p, CornerLoad& c) {
    const long long prim = entry / p.maxW;
    const int w = (int)(entry % p.maxW);
    const int Q = (p.G - 1) * (p.G - 1), VC = p.G * p.G;
    const long long path = prim / Q;
    const int quad = (int)(prim % Q);
    const int c0 = (quad / (p.G - 1)) * p.G + quad % (p.G - 1);
    const int corner = k == 0 ? c0 : (k == 1 ? c0 + 1 : (k == 2 ? c0 + 1 + p.G : c0 + p.G));
    const long long vi = (path * VC + corner) * p.W + w;
    c.a0 = __ldg(vtx + 2 * vi);
    c.a1 = __ldg(vtx + 2 * vi + 1);
    c.b0 = __ldg(vtx + 2 * vi + 2);
    c.b1 = __ldg(vtx + 2 * vi + 3);
}
// mix_vertex (rasterizing.cl:509-522) of one corner into record r. The texture coordinate
// is stored in texels, uv * tex_scale + tex_offset (fragment_fast): the weights sum to one,
// so interpolating texel coordinates is the fragment's ((uv / scale + 1) / 2) * size - 0.5.
__device__ __forceinline__ void store_corner(const CornerLoad& c, int k, float t, int S, const FragmentConsts& fc,
                                             float ox, float oy, Rec& r) {
    const float px = c.a0.x + (c.b0.x - c.a0.x) * t, py = c.a0.y + (c.b0.y - c.a0.y) * t;
    const int s = corner_slot(k);
    r.uv[s] = (c.a0.z + (c.b0.z - c.a0.z) * t) * fc.tsx + fc.tox;
    r.uv[4 + s] = (c.a0.w + (c.b0.w - c.a0.w) * t) * fc.tsy + fc.toy;
    r.rs[s] = ((c.a1.x + (c.b1.x - c.a1.x) * t) - 1.0f) * kRampScale;
    r.refl[s] = c.a1.y + (c.b1.y - c.a1.y) * t;
    r.inten[s] = c.a1.z + (c.b1.z - c.a1.z) * t;
    const int qx = cvt_rz_sat(px * (float)S), qy = cvt_rz_sat(py * (float)S);
    r.q()[2 * k] = qx;
    r.q()[2 * k + 1] = qy;
    const float x = (float)qx - ox, y = (float)qy - oy;
    r.xy[s] = x;
    r.xy[4 + s] = y;
    if (!(k & 1)) {  // the even corners again, swapped
        r.xy[8 + (s ^ 1)] = x;
        r.xy[10 + (s ^ 1)] = y;
    }
}
// Whether every fragment of a record is zero, so that shading it adds nothing:
//  - a corner's reflectance is NaN (a ray that failed, at either wavelength of the pair):
//    the coating term max(NaN, 0) is 0 (rasterizing.cl:495-497) and every other factor is
//    finite, so each fragment is exactly 0;
//  - one sample per pixel, every corner's rrel >= 1 (the ray left the lens housing) and the
//    quad strictly convex and counter-clockwise in sample space, with coordinates that keep
//    the edge functions exact and an extent below 4096: a covered pixel is then inside the
//    quad or on one of its edges or corners, where every cross product a_i is >= 0 (an
//    exact integer) and the tangents share its sign, so the mean-value weights are
//    non-negative up to rounding and their rrel is >= 1; smoothstep(1, 0.95, rrel) is 0
//    there, and at most a few units in the last place of 1 below it (a factor below 1e-9).
// Clockwise quads are left in: on an edge the reference divides by +1e-3 whatever the
// orientation, so the weights there mix signs.
//  - a corner's texel coordinate is not finite (a stop of height 0): so is every fragment's that
//    the corner takes part in, and lookups there are 0.
__device__ __forceinline__ bool zero_record(const RasterParams& p, const Rec& r, bool ccw) {
    const float4 rf = ld4(r.refl);
    if (isnan(rf.x) || isnan(rf.y) || isnan(rf.z) || isnan(rf.w)) return true;
    const float4 u = ld4(r.uv), v = ld4(r.uv + 4);
    if (!(fabsf(u.x) + fabsf(u.y) + fabsf(u.z) + fabsf(u.w) + fabsf(v.x) + fabsf(v.y) + fabsf(v.z) + fabsf(v.w) <=
          3.40282347e38f))
        return true;
    if (!ccw) return false;
    const float4 rl = ld4(r.rs);  // rrel >= 1 exactly when the ramp is <= 0
    return rl.x <= 0.0f && rl.y <= 0.0f && rl.z <= 0.0f && rl.w <= 0.0f;
}
// Whether the housing falloff is 1 and no clamp acts at any covered pixel of a record with one
// sample per pixel: every corner's rrel <= 0.95 (ramp >= 1), intensity and reflectance >= 0, all of
// them finite, and the quad strictly convex. Inside it, off its edges, the cross products a_i share one sign, so
// the normalised weights are positive up to rounding and the ramp stays >= 1 up to a rounding,
// where the smoothstep is 1 to second order. On an edge (a_i = 0: the rare path of the weights)
// a clockwise quad's weights mix signs, and mean_value_weights asks for the general form. A corner
// that is NaN (infinite at both wavelengths: an element of height 0) makes every fragment of the
// general form 0, by its clamps.
__device__ __forceinline__ bool inside_housing(const Rec& r) {
    // As unsigned bits non-negative finite floats come first, in order; then infinity, NaN, the negative ones.
    auto bits = [](const float* p) { return *reinterpret_cast<const uint4*>(p); };
    auto most = [](uint4 v) { return max(max(v.x, v.y), max(v.z, v.w)); };
    const uint4 ramp = bits(r.rs);
    return min(min(ramp.x, ramp.y), min(ramp.z, ramp.w)) >= 0x3f800000u /* 1 */ &&
           max(most(ramp), max(most(bits(r.inten)), most(bits(r.refl)))) <= 0x7f7fffffu /* the largest float */;
}

// edges, bounds and flags of a record whose corners are stored; (ox, oy): the tile's first sample;
// kRows: the pixel rows of a block
template <int kRows>
__device__ __forceinline__ void finish_record(const RasterParams& p, int w, int i, int ox, int oy, const float* xyz,
                                              Rec& r) {
    const int4 q01 = ld4i(r.q()), q23 = ld4i(r.q() + 4);
    const int q[8] = {q01.x, q01.y, q01.z, q01.w, q23.x, q23.y, q23.z, q23.w};
    const int4 bb = make_int4(min(min(q[0], q[2]), min(q[4], q[6])), max(max(q[0], q[2]), max(q[4], q[6])),
                              min(min(q[1], q[3]), min(q[5], q[7])), max(max(q[1], q[3]), max(q[5], q[7])));
    *reinterpret_cast<int4*>(r.bb) = bb;
    // bounds rejection is exact while every coordinate stays below 2^14 - 1 in magnitude: the
    // edge values are then exact in int32. Relative to the tile (its samples x, y < 32 S) they
    // are exact in FP32 too: |A|, |B| <= 32764 (16383 with 8 samples, else the record counts as
    // unsafe), so |A y + B x| < 2^23, and C, the value at the tile's first sample, is clamped
    // to +-2^23: every exact value has magnitude below 2^24, and a clamped one its sign.
    const int lim = 16382;
    const bool safe = p.safe_screen && bb.x >= -lim && bb.y <= lim && bb.z >= -lim && bb.w <= lim &&
                      (p.S < 8 || (bb.y - bb.x < 16384 && bb.w - bb.z < 16384));
    const float hx = 4.0f * (float)p.S - 0.5f, hy = 0.5f * kRows * (float)p.S - 0.5f;
    // (beyond, the integer coefficients' bits, for samples relative to the image: WildEdges)
    float ea[5], eb[5], ecl[5];
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const int a = k < 4 ? k : 2, b = k < 4 ? (k + 1) & 3 : 0;
        int e[3];
        edge_coeffs(q[2 * a], q[2 * a + 1], q[2 * b], q[2 * b + 1], e);
        const int c = wadd(e[2], wadd(wmul(e[0], oy), wmul(e[1], ox)));
        ea[k] = safe ? (float)e[0] : __int_as_float(e[0]);
        eb[k] = safe ? (float)e[1] : __int_as_float(e[1]);
        ecl[k] = safe ? (float)min(max(c, -8388608), 8388608) : __int_as_float(e[2]);
    }
    int flags = safe ? 1 : 0;
    const bool collinear = edge_i(q[0], q[1], q[2], q[3], q[4], q[5]) == 0 &&
                           edge_i(q[0], q[1], q[4], q[5], q[6], q[7]) == 0;
    bool ccw = false, cw = false;  // strictly convex quads of one sample per pixel
    if (p.S == 1 && safe && bb.y - bb.x < 4096 && bb.w - bb.z < 4096) {
        // |differences| < 4096: the turns are exact in 32 bits
        ccw = cw = true;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int j = (k + 1) & 3, l = (k + 2) & 3;
            const int turn = (q[2 * j] - q[2 * k]) * (q[2 * l + 1] - q[2 * j + 1]) -
                             (q[2 * j + 1] - q[2 * k + 1]) * (q[2 * l] - q[2 * j]);
            ccw = ccw && turn > 0;
            cw = cw && turn < 0;
        }
    }
    if (collinear || zero_record(p, r, ccw)) flags |= 2;
    float4 col = make_float4(1.0f, 1.0f, 1.0f, (ccw || cw) && inside_housing(r) ? 0.0f : 1.0f);
    if (p.W > 1) {  // with one wavelength rgb += frag (rasterizing.cl:648-650): a weight of exactly 1
        const float* c = xyz + 3 * (w * p.WS + i);
        col.x = c[0], col.y = c[1], col.z = c[2];
    }
    *reinterpret_cast<float4*>(r.col) = col;
    float4* ef = reinterpret_cast<float4*>(r.ef);
    ef[0] = make_float4(ea[0], ea[1], eb[0], eb[1]);
    ef[1] = make_float4(ecl[0], ecl[1], ea[2], ea[3]);
    ef[2] = make_float4(eb[2], eb[3], ecl[2], ecl[3]);
    ef[3] = make_float4(ea[4], eb[4], ecl[4], __int_as_float(flags));
    // (half ranges over a block, of the exact form only)
    *reinterpret_cast<float4*>(r.ext) =
        make_float4(fabsf(ea[0]) * hy + fabsf(eb[0]) * hx, fabsf(ea[1]) * hy + fabsf(eb[1]) * hx,
                    fabsf(ea[2]) * hy + fabsf(eb[2]) * hx, fabsf(ea[3]) * hy + fabsf(eb[3]) * hx);
}

// How many of the S n-rook samples of this lane's pixel a record covers. (rx0, ry0): the block's first
// sample relative to the tile, (sx0, sy0): the pixel's; wild: the record needs the exact test.
template <int T, int kS = 0>
__device__ __forceinline__ int sample_hits(const Rec& r, int S, bool wild, float rx0, float ry0, int sx0, int sy0,
                                           int lane) {
    int hits = 0;
    if (wild) {
        const WildEdges we(r);
        for (int s = 0; s < S; s++) hits += we.inside(sx0 + s, sy0 + SUB_OFFSETS[S - 1 + s]) ? 1 : 0;
        return hits;
    }
    Edges e;
    load_edges(r, e);
    const float x = rx0 + (float)((lane & 7) * S), y = ry0 + (float)((lane >> 3) * S);
    if constexpr (kS == 2 || kS == 4) {
        // From the first sample on the edge values change by b + (the offsets' difference) a per sample:
        // offsets 1, 0 (two samples) and 1, 2, 0, 3 (four, SUB_OFFSETS). All are integers below 2^24,
        // exact as in inside(). Zoom lens, 4 samples: raster 19.0 -> 18.3 ms.
        const f2 x2 = pk(x, x), y2 = pk(y + 1.0f, y + 1.0f);
        f2 e0 = fma2(e.a0, y2, fma2(e.b0, x2, e.c0)), e1 = fma2(e.a1, y2, fma2(e.b1, x2, e.c1));
        float e2 = fmaf(e.a20, lo2(y2), fmaf(e.b20, x, e.c20));
        hits += inside_at(e0, e1, e2) ? 1 : 0;
        auto next = [&](float offset) {
            const f2 o = pk(offset, offset);
            e0 = add2(e0, fma2(o, e.a0, e.b0));
            e1 = add2(e1, fma2(o, e.a1, e.b1));
            e2 += fmaf(offset, e.a20, e.b20);
            hits += inside_at(e0, e1, e2) ? 1 : 0;
        };
        if constexpr (kS == 2) {
            next(-1.0f);
        } else {
            next(1.0f);
            next(-2.0f);
            next(3.0f);
        }
        return hits;
    }
    for (int s = 0; s < S; s++) {
        const float xs = x + (float)s, ys = y + (float)SUB_OFFSETS[S - 1 + s];
        hits += inside(e, pk(xs, xs), pk(ys, ys)) ? 1 : 0;
    }
    return hits;
}

// A CTA of 8 warps shades one T x T tile (T = 32 or 16): the tile's blocks of 8 x 4 pixels (8 x 8
// with two pixels per lane; block b at column b % (T / 8), row b / (T / 8)) go to warps one at a time,
// so a record outside a block's sample bounds is skipped by the whole warp at once.
constexpr int kThreads = 256;

template <int T>
constexpr size_t raster_smem_bytes(int maxW, int WS) {
    return sizeof(Rec) * 2 * kBatchRecords + sizeof(float) * (3 * maxW * WS + ((WS + 3) & ~3)) +
           sizeof(float) * 96 * (T * T / 32);
}

// Tile (tx, ty), whose entries are tile_entries[begin, end). smem4 holds the dynamic shared
// memory (raster_smem_bytes), next_block four shared counters. kS: the anti-aliasing sample
// count, or 0 for p.S (large ghost textures). kTex: how the ghost texture is looked
// up (kLoads, kGather through p.ghost_tex, kAnyLoads).
template <int T, int kS, int kTex, int kPix>
__device__ __forceinline__ void raster_tile(const float4* __restrict__ vtx, uint32_t begin, uint32_t end,
                                            const uint32_t* __restrict__ tile_entries,
                                            const float* __restrict__ ghost, const float* __restrict__ spectrum,
                                            const RasterParams& p, const FragmentConsts& fcs,
                                            float4* __restrict__ image, int tx, int ty, float4* smem4,
                                            int* next_block) {
    constexpr int kRows = 4 * kPix;                // pixel rows of a block
    constexpr int kBlocks = T * T / (32 * kPix);   // blocks of 8 x kRows pixels per tile
    constexpr int kCols = T / 8;                   // blocks per tile row
    Rec* recbuf = (Rec*)smem4;     // two batches of records
    float* xyz = (float*)(recbuf + 2 * kBatchRecords);  // [maxW * WS][3]
    float* blend = xyz + 3 * p.maxW * p.WS;       // [WS]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        const float sub_step = 1.0f / (float)p.WS;
        float b = 0.0f;
        for (int i = 0; i < p.WS; i++) {
            blend[i] = b;
            b += sub_step;
        }
    }
    if (p.W > 1) {
        const float sub_step = 1.0f / (float)p.WS;
        const float wl_step = sub_step / (float)p.W;
        for (int w = threadIdx.x; w < p.maxW; w += kThreads) {
            float pos = ((float)w + 0.5f) / (float)p.W;
            for (int i = 0; i < p.WS; i++) {
                for (int c = 0; c < 3; c++)
                    xyz[3 * (w * p.WS + i) + c] = sample_linear(spectrum, RF_SPECTRUM_WIDTH, 1, 4, c, pos, 0.0f, true);
                pos += wl_step;
            }
        }
    }

    const int S = kS ? kS : p.S;
    const FragmentConsts fc = fcs;
    RF_STAT(unsigned long long st_iter = 0; unsigned long long st_whole = 0; unsigned long long st_frag = 0;
            unsigned long long st_frag_whole = 0; unsigned long long st_blocks = 0; unsigned long long st_zero = 0;
            unsigned long long st_zero_iter = 0; unsigned long long st_steps = 0;)
    // accumulators of the pixel blocks, [(block * 3 + channel) * kPix + row][lane]
    float* acc = blend + ((p.WS + 3) & ~3);
#pragma unroll
    for (int i = threadIdx.x; i < kBlocks * 96 * kPix; i += kThreads) acc[i] = 0.0f;

    const int per_batch = kBatchRecords / p.WS;  // entries per batch (WS <= kBatchRecords)
    // Batches of records are double-buffered: while warps shade batch t from one buffer,
    // warps that are done build batch t + 1 in the other, one barrier per batch. Thread j
    // loads corner j % 4 of entry j / 4 (the four corners of an entry sit in one warp). The
    // vertices are not fetched ahead: a batch is shaded for tens of microseconds, and 18
    // registers held through the shading loop cost more than the loads' latency.
    const int my_corner = lane & 3;
    // Warps take the batch's entries 8 at a time as they run out of blocks to shade: a warp held
    // up by a heavy block does not also hold the batch up with its share of the building.
    auto build = [&](Rec* dst, uint32_t first, int* next_entry) {
        const int count = (int)min((uint32_t)per_batch, end - first);
        for (;;) {
            int e0 = 0;
            if (lane == 0) e0 = atomicAdd(next_entry, 8);
            e0 = __shfl_sync(0xffffffffu, e0, 0);
            if (e0 >= count) break;
            const int e = e0 + (lane >> 2);
            uint32_t entry = 0;
            if (e < count) {
                entry = tile_entries[first + e];
                CornerLoad c;
                load_corner(vtx, entry, my_corner, p, c);
                for (int i = 0; i < p.WS; i++) store_corner(c, my_corner, blend[i], S, fc, (float)(tx * T * S), (float)(ty * T * S),
                                                                      dst[e * p.WS + i]);
            }
            __syncwarp();  // the four corners of each record are stored
            if (e < count)
                for (int i = my_corner; i < p.WS; i += 4)
                    finish_record<kRows>(p, (int)(entry % p.maxW), i, tx * T * S, ty * T * S, xyz, dst[e * p.WS + i]);
        }
    };
    // next_block[0, 1]: the next block of each buffer's batch, [2, 3]: its next entry to build
    if (threadIdx.x < 4) next_block[threadIdx.x] = 0;
    __syncthreads();  // blend weights and colours are set
    if (begin < end) build(recbuf, begin, next_block + 2);
    __syncthreads();
    int cur = 0;
    for (uint32_t base = begin; base < end; base += per_batch, cur ^= 1) {
        const int n_rec = (int)min((uint32_t)per_batch, end - base) * p.WS;
        const Rec* recs = recbuf + cur * kBatchRecords;
        // Warps take the tile's blocks one at a time (blocks differ widely in work);
        // a block is shaded by one warp per batch, batches in order, so every pixel still
        // adds its records in increasing order.
#pragma unroll 1
        for (;;) {
            int blk = 0;
            if (lane == 0) blk = atomicAdd(&next_block[cur], 1);
            blk = __shfl_sync(0xffffffffu, blk, 0);
            if (blk >= kBlocks) break;
            RF_STAT(st_blocks += lane == 0;)
            const int x0 = tx * T + (blk % kCols) * 8, y0 = ty * T + (blk / kCols) * kRows;
            const int px = x0 + (lane & 7), py = y0 + (lane >> 3) * kPix;  // the lane's first pixel
            const int bx0 = x0 * S, by0 = y0 * S, bx1 = bx0 + 8 * S - 1, by1 = by0 + kRows * S - 1;
            const bool in_image = px < p.width && py < p.height;
            const int sx0 = px * S, sy0 = py * S;
            // which records can touch this block, which cover all of it, and which need the
            // exact test at every sample: lanes test 32 records at a time
            const float rx0 = (float)((blk % kCols) * 8 * S), ry0 = (float)((blk / kCols) * kRows * S);
            const float hx = 4.0f * (float)S - 0.5f, hy = 0.5f * kRows * (float)S - 0.5f;
            const f2 bxc = pk(rx0 + hx, rx0 + hx), byc = pk(ry0 + hy, ry0 + hy);
            unsigned sel[kBatchRecords / 32], whole[kBatchRecords / 32], wild[kBatchRecords / 32];
#pragma unroll
            for (int m = 0; m < kBatchRecords / 32; m++) {
                const int j = m * 32 + lane;
                bool take = false, all = false, far = false;
                if (j < n_rec) {
                    const Rec& r = recs[j];
                    const int flags = __float_as_int(ld4(r.ef + 12).w);  // with ef[12..14], which rect_coverage reads
                    if (!(flags & 2)) {  // collinear (intersect_quad rejects all) or all-zero
                        const int4 bb = *reinterpret_cast<const int4*>(r.bb);
                        far = !(flags & 1);
                        take = far || !(bx1 < bb.x || bx0 > bb.y || by1 < bb.z || by0 > bb.w);
                        if (take && !far) {
                            const int cov = rect_coverage(r, bxc, byc, hx, hy);
                            take = cov != 0;
                            all = cov == 2;
                        }
                    }
                }
                sel[m] = __ballot_sync(0xffffffffu, take);
                whole[m] = __ballot_sync(0xffffffffu, all);
                wild[m] = __ballot_sync(0xffffffffu, far);
            }
            float rgb[3][kPix];
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int i = 0; i < kPix; i++) rgb[c][i] = acc[((3 * blk + c) * kPix + i) * 32 + lane];
            // (no warp-wide operation below: lanes outside the image skip the records)
            if constexpr (kS == 1) {
                // One sample per pixel: every lane first marks the selected records that cover
                // its pixels (whole-block records cover every pixel; the others are tested, in a
                // loop that is the same for all lanes), then shades its own covered records in
                // increasing order. A lane is not held up by records that miss its pixels, so a
                // warp takes about as many shading steps as its busiest lane has records.
                // Masks are kept bit-reversed (record j at bit 31 - j), so the next record is a
                // plain count of leading zeros.
                static_assert(kBatchRecords == 64, "two coverage masks per lane and pixel");
                const float lx = rx0 + (float)(lane & 7);
                const f2 lx2 = pk(lx, lx);
                unsigned cov[2][kPix];
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    unsigned c[kPix], part = __brev(sel[m] & ~whole[m] & ~wild[m]);
#pragma unroll
                    for (int i = 0; i < kPix; i++) c[i] = __brev(whole[m]);
                    while (part) {
                        const int b = __clz(part);
                        const unsigned bit = 0x80000000u >> b;
                        part ^= bit;
                        Edges e;
                        load_edges(recs[m * 32 + b], e);
#pragma unroll
                        for (int i = 0; i < kPix; i++) {
                            const float ly = ry0 + (float)((lane >> 3) * kPix + i);
                            if (inside(e, lx2, pk(ly, ly))) c[i] |= bit;
                        }
                    }
                    for (part = __brev(wild[m]); part;) {
                        const int b = __clz(part);
                        const unsigned bit = 0x80000000u >> b;
                        part ^= bit;
                        const WildEdges we(recs[m * 32 + b]);
#pragma unroll
                        for (int i = 0; i < kPix; i++)
                            if (we.inside(sx0, sy0 + i)) c[i] |= bit;
                    }
#pragma unroll
                    for (int i = 0; i < kPix; i++) cov[m][i] = px < p.width && py + i < p.height ? c[i] : 0;
                    RF_STAT(if (lane == 0) { st_iter += __popc(sel[m]); st_whole += __popc(whole[m]); })
                }
                f2 fy2[kPix];
                unsigned todo[2] = {0, 0};
#pragma unroll
                for (int i = 0; i < kPix; i++) {
                    const float ly = ry0 + (float)((lane >> 3) * kPix + i);
                    fy2[i] = pk(ly, ly);
                    todo[0] |= cov[0][i];
                    todo[1] |= cov[1][i];
                }
                const Rec* half = recs;
                for (;;) {
                    if (todo[0] == 0) {
                        todo[0] = todo[1];
                        todo[1] = 0;
                        half += 32;
#pragma unroll
                        for (int i = 0; i < kPix; i++) cov[0][i] = cov[1][i];
                        if (todo[0] == 0) break;
                    }
                    const int j = __clz(todo[0]);
                    const unsigned bit = 0x80000000u >> j;
                    todo[0] ^= bit;
                    const Rec& r = half[j];
                    bool need[kPix];
#pragma unroll
                    for (int i = 0; i < kPix; i++) need[i] = kPix == 1 || (cov[0][i] & bit) != 0;
                    RF_STAT(const int jj = (int)(&r - recs);
                            for (int i = 0; i < kPix; i++) {
                                st_frag += need[i];
                                st_frag_whole += need[i] && ((whole[jj >> 5] >> (jj & 31)) & 1u);
                            }
                            if (lane == __ffs(__activemask()) - 1) st_steps++;)
                    f2 we[kPix], wo[kPix];
                    float4 col = ld4(r.col);
                    mean_value_weights<kPix>(r, lx2, fy2, need, true, we, wo, col.w);
                    float f[kPix];
                    fragment_fast<kTex, kPix>(r, we, wo, ghost, p, col.w, f);
#pragma unroll
                    for (int i = 0; i < kPix; i++) {
                        const float fi = need[i] ? f[i] : 0.0f;
                        rgb[0][i] += col.x * fi;
                        rgb[1][i] += col.y * fi;
                        rgb[2][i] += col.z * fi;
                    }
                }
            }
            if constexpr (kS != 1) {
                // Several samples per pixel: the same two steps, with each pixel's number of covered samples
                // less one in bit planes. Zoom lens, 1920 x 1080, 4 samples: 21.3 -> 19.0 ms (lanes that
                // missed a record waited for the others: 71 % shaded); 601 x 403, 2 samples 0.296 -> 0.240.
                const float cx = rx0 + (float)((lane & 7) * S + S / 2), cy = ry0 + (float)((lane >> 3) * S + S / 2);
                const f2 cx2 = pk(cx, cx), cy2 = pk(cy, cy);
                unsigned cov[2], h0[2], h1[2], h2[2];
#pragma unroll
                for (int m = 0; m < 2; m++) {
                    const Rec* half = recs + 32 * m;
                    const unsigned far = __brev(wild[m]), all = __brev(whole[m]);
                    unsigned c = all, a0 = all, a1 = all, a2 = all;
#pragma unroll 1
                    for (unsigned part = __brev(sel[m] & ~whole[m]); part;) {
                        const int b = __clz(part);
                        const unsigned bit = 0x80000000u >> b;
                        part ^= bit;
                        const int hits = sample_hits<T, kS>(half[b], S, (far & bit) != 0, rx0, ry0, sx0, sy0, lane);
                        if (hits > 0) {
                            c |= bit;
                            if ((hits - 1) & 1) a0 |= bit;
                            if (kS != 2 && ((hits - 1) & 2)) a1 |= bit;
                            if (kS != 2 && kS != 4 && ((hits - 1) & 4)) a2 |= bit;
                        }
                    }
                    cov[m] = in_image ? c : 0;
                    h0[m] = a0, h1[m] = a1, h2[m] = a2;
                    RF_STAT(if (lane == 0) { st_iter += __popc(sel[m]); st_whole += __popc(whole[m]); })
                }
                const int full = S - 1;  // a plane beyond it is not the record's
                const Rec* half = recs;
                for (;;) {  // in increasing record order: the reference's summation order
                    if (cov[0] == 0) {
                        cov[0] = cov[1], h0[0] = h0[1], h1[0] = h1[1], h2[0] = h2[1];
                        cov[1] = 0;
                        half += 32;
                        if (cov[0] == 0) break;
                    }
                    const int j = __clz(cov[0]);
                    const unsigned bit = 0x80000000u >> j;
                    cov[0] ^= bit;
                    const Rec& r = half[j];
                    const int hits = 1 + (((h0[0] & bit ? 1 : 0) + (kS != 2 && (h1[0] & bit) ? 2 : 0) +
                                          (kS != 2 && kS != 4 && (h2[0] & bit) ? 4 : 0)) & full);
                    RF_STAT(st_frag++; const int jj = (int)(&r - recs); st_frag_whole += (whole[jj >> 5] >> (jj & 31)) & 1u;
                            if (lane == __ffs(__activemask()) - 1) st_steps++;)
                    f2 we, wo;
                    float general = 1.0f;
                    mean_value_weights(r, cx2, cy2, kS == 0 && S == 1, we, wo, general);
                    RF_STAT({
                        const bool z = blend4(we, wo, r.rs) <= 0.0f;
                        st_zero += z;
                        const unsigned am = __activemask();
                        if (__all_sync(am, z) && lane == __ffs(am) - 1) st_zero_iter++;
                    })
                    const float4 col = ld4(r.col);
                    const float f = fragment_fast<kTex>(r, we, wo, ghost, p, 1.0f) * (float)hits;
                    rgb[0][0] += col.x * f;
                    rgb[1][0] += col.y * f;
                    rgb[2][0] += col.z * f;
                }
            }
#pragma unroll
            for (int c = 0; c < 3; c++)
#pragma unroll
                for (int i = 0; i < kPix; i++) acc[((3 * blk + c) * kPix + i) * 32 + lane] = rgb[c][i];
        }
        if (base + per_batch < end) build(recbuf + (cur ^ 1) * kBatchRecords, base + per_batch, next_block + 2 + (cur ^ 1));
        // the other buffer's block counter and this one's entry counter were last used for the
        // batch before and for building this one, behind the last barrier
        if (threadIdx.x == 0) next_block[cur ^ 1] = next_block[2 + cur] = 0;
        __syncthreads();
    }

    RF_STAT(atomicAdd(&g_raster_stats[0], st_iter); atomicAdd(&g_raster_stats[1], st_whole);
            atomicAdd(&g_raster_stats[2], st_frag); atomicAdd(&g_raster_stats[3], st_frag_whole);
            atomicAdd(&g_raster_stats[4], st_blocks); atomicAdd(&g_raster_stats[5], st_zero);
            atomicAdd(&g_raster_stats[6], st_zero_iter); atomicAdd(&g_raster_stats[7], st_steps);)
    __syncthreads();  // every block's last batch is shaded
    const float scale = p.intensity / (float)(p.W * p.S * p.WS);
    for (int blk = warp; blk < kBlocks; blk += 8) {
#pragma unroll
        for (int i = 0; i < kPix; i++) {
            const int px = tx * T + (blk % kCols) * 8 + (lane & 7);
            const int py = ty * T + (blk / kCols) * kRows + (lane >> 3) * kPix + i;
            if (px >= p.width || py >= p.height) continue;
            const float* a = acc + (3 * blk * kPix + i) * 32 + lane;
            const float c0 = a[0], c1 = a[32 * kPix], c2 = a[64 * kPix];
            float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c0 > 0.0f || c1 > 0.0f || c2 > 0.0f) out = xyz_to_ap1(c0 * scale, c1 * scale, c2 * scale);
            image[(size_t)(p.height - (py + 1)) * p.width + px] = out;
        }
    }
}

template <int T, int kS>
constexpr int kPixels = kS != 1 ? 1 : (T == 32 ? RF_RASTER_PIX32 : RF_RASTER_PIX16);

// What bounds it: instruction issue, the FP32 pipe and the reciprocals together (69 % issue-active,
// FP32 pipe 60 %, reciprocals 48 % on the 16-surface frame). Production frame (2048^2, 91.5 M
// entries) / 16-surface frame / four samples x eight sub-steps at 1920 x 1080:
//  118.7 / 4.12 / 29.6 ms  scalar corners, int32 edge functions, one pixel per lane
//  102.1 / 3.57 / 22.3 ms  corners in packed pairs, edge functions as exact packed FP32, records
//                          wholly inside the housing without falloff and clamps
//   90.2 / 3.22 / 21.5 ms  two pixels of a column per lane (one sample per pixel): a record's
//                          loads, loop and x terms serve both, and their chains overlap; next
//                          batch's vertices not held in registers
//   89.6 / 3.19 / 21.4 ms  texel origins without floors
// (Cross products from the edge functions and r_i r_j - d_i from the edge lengths would be 88.6 /
// 3.15 / 21.0 ms and lose fewer digits, but move single pixels of large quads by up to 2e-3 away
// from the form below.)
// One CTA per tile of a frame: CTA k shades tile order[k], or tile k without an order.
// CTAs start in index order as slots free up, so an order by decreasing work starts the
// heaviest tiles first and ends the launch with light ones.
template <int T, int kS, int kTex>
__global__ void __launch_bounds__(kThreads, kS == 1 ? RF_RASTER_MIN_BLOCKS_S1 : RF_RASTER_MIN_BLOCKS)
    k_raster(const float4* __restrict__ vtx, const uint32_t* __restrict__ tile_offsets,
             const uint32_t* __restrict__ tile_entries, const uint32_t* __restrict__ order,
             const float* __restrict__ ghost, const float* __restrict__ spectrum, RasterParams p, FragmentConsts fcs,
             float4* __restrict__ image) {
    extern __shared__ float4 smem4[];
    __shared__ int next_block[4];  // per buffer: blocks handed out, entries handed out to build
    const int tile = order ? (int)order[blockIdx.x] : (int)blockIdx.x;
    raster_tile<T, kS, kTex, kPixels<T, kS>>(vtx, tile_offsets[tile], tile_offsets[tile + 1], tile_entries, ghost, spectrum, p, fcs,
                             image, tile % p.ntx, tile / p.ntx, smem4, next_block);
}

__host__ __device__ inline bool make_params(const rf_raster_args& a, RasterParams& p);

// Every frame of a batch in one persistent launch: each CTA takes the next tile from the
// queue (tiles ordered by decreasing entry count) until none are left. kTex kGather: every frame's
// ghost lookups go through its rf_frame.ghost_texture.
template <int T, int kS, int kTex>
__global__ void __launch_bounds__(kThreads, kS == 1 ? RF_RASTER_MIN_BLOCKS_S1 : RF_RASTER_MIN_BLOCKS)
    k_raster_batch(const rf_frame* __restrict__ frames, int F, int tiles, const uint32_t* __restrict__ order,
                   unsigned* __restrict__ queue, const unsigned long long* __restrict__ entry_total,
                   long long capacity, const float4* __restrict__ vtx_all, const uint32_t* __restrict__ tile_offsets,
                   const uint32_t* __restrict__ tile_entries, const float* __restrict__ ghosts,
                   const float* __restrict__ spectrum, float4* __restrict__ images) {
    extern __shared__ float4 smem4[];
    __shared__ int next_block[4];
    // the current tile's frame settings, held in shared memory rather than registers
    __shared__ RasterParams sp;
    __shared__ FragmentConsts sfc;
    __shared__ int item, s_tile, s_gt;
    __shared__ long long s_vtx, s_ghost, s_image;
    if (*entry_total > (unsigned long long)capacity) return;  // incomplete lists: nothing is drawn
    for (;;) {
        if (threadIdx.x == 0) {
            item = (int)atomicAdd(queue, 1u);
            if (item < tiles) {
                const int gt = (int)order[item];
                const int f = find_frame(frames, F, gt, [](const rf_frame& fr) { return fr.tile_offset; });
                const rf_frame& fr = frames[f];
                RasterParams q;
                make_params(fr.raster, q);
                if (kTex == kGather) q.ghost_tex = fr.ghost_texture;
                q.T = T;
                q.ntx = (q.width + T - 1) / T;
                sp = q;
                sfc = fragment_consts(q);
                s_gt = gt;
                s_tile = gt - fr.tile_offset;
                s_vtx = fr.vertex_offset;
                s_ghost = fr.ghost_offset;
                s_image = fr.image_offset;
            }
        }
        __syncthreads();
        if (item >= tiles) break;
        const int gt = s_gt, tile = s_tile;
        // (the tile's code for the frame's sample count: with a count known at run time only, 12 frames of 1024 x
        // 1024 take 18.5 instead of 16.4 ms at 2 samples, 19.7 / 17.3 at 4, 22.6 / 20.5 at 8)
        auto shade = [&](auto samples) {
            constexpr int kTile = decltype(samples)::value;
            raster_tile<T, kTile, kTex, kPixels<T, kTile>>(vtx_all + 2 * s_vtx, tile_offsets[gt], tile_offsets[gt + 1],
                                                           tile_entries, ghosts + s_ghost, spectrum, sp, sfc,
                                                           images + s_image, tile % sp.ntx, tile / sp.ntx, smem4,
                                                           next_block);
        };
        if (kS == 1 || sp.S == 1)
            shade(std::integral_constant<int, 1>());
        else if (sp.S == 2)
            shade(std::integral_constant<int, 2>());
        else if (sp.S == 4)
            shade(std::integral_constant<int, 4>());
        else
            shade(std::integral_constant<int, 8>());
        __syncthreads();  // the tile's accumulators and `item` are free again
    }
}

// ---------------------------------------------------------------- adjoint
// The adjoint's fragment keeps one scalar operation per term in the corners' order (weights,
// interpolations, floors): where gradients of opposite sign cancel (the light's above all), the
// last bits of the terms show in the sums, and this form's are what its gradients have been
// checked with.
__device__ __forceinline__ void scalar_weights(const Rec& rec, float px, float py, float w[4]) {
    float sx[4], sy[4], a[4], d[4], r2[4], ir[4], r[4], t[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int k = corner_slot(i);
        sx[i] = rec.xy[k] - px;
        sy[i] = rec.xy[4 + k] - py;
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int j = (i + 1) & 3;
        a[i] = sx[i] * sy[j] - sx[j] * sy[i];
        d[i] = sx[i] * sx[j] + sy[i] * sy[j];
        r2[i] = sx[i] * sx[i] + sy[i] * sy[i];
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        ir[i] = rsqrtf(r2[i]);
        r[i] = r2[i] * ir[i];
    }
#pragma unroll
    for (int i = 0; i < 4; i++) t[i] = (r[i] * r[(i + 1) & 3] - d[i]) * __fdividef(1.0f, a[i]);
#pragma unroll
    for (int i = 0; i < 4; i++) w[i] = (t[(i + 3) & 3] + t[i]) * ir[i];
    float sum = w[0] + w[1] + w[2] + w[3];
    if (!(fabsf(sum) <= 3.40282347e38f)) {  // the special cases (special_weights)
        bool zero = false;
#pragma unroll
        for (int i = 0; i < 4; i++) zero = zero || r2[i] == 0.0f;
        if (zero) {
            int k = 0;
#pragma unroll
            for (int i = 3; i >= 0; i--)
                if (sx[i] == 0.0f && sy[i] == 0.0f) k = i;
#pragma unroll
            for (int i = 0; i < 4; i++) w[i] = i == k ? 1.0f : 0.0f;
            return;
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int j = (i + 1) & 3;
            if (a[i] == 0.0f)
                t[i] = __fdiv_rn(__fsub_rn(__fmul_rn(__fsqrt_rn(r2[i]), __fsqrt_rn(r2[j])), d[i]), 1e-3f);
            else
                t[i] = (r[i] * r[j] - d[i]) * __fdividef(1.0f, a[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; i++) w[i] = (t[(i + 3) & 3] + t[i]) * ir[i];
        sum = w[0] + w[1] + w[2] + w[3];
    }
    const float inv = __fdividef(1.0f, sum);
#pragma unroll
    for (int i = 0; i < 4; i++) w[i] *= inv;
}
__device__ __forceinline__ float scalar_blend(const float w[4], const float* v) {  // v: even corners first
    const float4 q = ld4(v);
    return w[0] * q.x + w[1] * q.z + w[2] * q.y + w[3] * q.w;
}

// ghost_sample with its derivatives with respect to the texel coordinates (u, v) = uv * size - 0.5.
template <bool kTex>
__device__ __forceinline__ float ghost_sample_grad(const float* __restrict__ tex, const RasterParams& p, float u,
                                                   float v, float& du, float& dv) {
    du = dv = 0.0f;
    if (!(fabsf(u) < 1e9f) || !(fabsf(v) < 1e9f)) return 0.0f;
    const float fu = floorf(u), fv = floorf(v);
    const float a = u - fu, b = v - fv;
    float t00, t10, t01, t11;
    if (kTex) {
        const float4 g = tex2Dgather<float4>((cudaTextureObject_t)p.ghost_tex, fu + 1.0f, fv + 1.0f, 0);
        t00 = g.w, t10 = g.z, t01 = g.x, t11 = g.y;
    } else {
        ghost_texels(tex, p.ghost_w, p.ghost_h, p.ghost_large, cvt_rz_sat(fu), cvt_rz_sat(fv), t00, t10, t01, t11);
    }
    du = (1.0f - b) * (t10 - t00) + b * (t11 - t01);
    dv = (1.0f - a) * (t01 - t00) + a * (t11 - t10);
    return (1.0f - a) * (1.0f - b) * t00 + a * (1.0f - b) * t10 + (1.0f - a) * b * t01 + a * b * t11;
}

constexpr int kGradAttrs = 5;  // per corner: u, v, rrel, reflectance, intensity
// row stride of the backward's per-warp transpose buffers (floats)
constexpr int kRedStride = 36;
// rows of a warp's transpose buffer: the 5 attribute gradients and the 4 corner weights
constexpr int kRedRows = kGradAttrs + 4;
// adds scale * g to a vertex's attributes: floats 2 to 6 of (pos.xy, uv.xy, rrel, reflectance,
// intensity, pad). vectors: the vertexes start on 16-byte boundaries, as the vector additions
// need (two instead of five; a buffer that starts elsewhere gets scalar ones).
__device__ __forceinline__ void add_gradients(float* vertex, const float g[kGradAttrs], float scale, bool vectors) {
    if (!vectors) {
#pragma unroll
        for (int a = 0; a < kGradAttrs; a++) atomicAdd(vertex + 2 + a, g[a] * scale);
        return;
    }
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" ::"l"(vertex + 2), "f"(g[0] * scale), "f"(g[1] * scale)
                 : "memory");
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(vertex + 4), "f"(g[2] * scale),
                 "f"(g[3] * scale), "f"(g[4] * scale), "f"(0.0f)
                 : "memory");
}

// Backward of k_raster (32 x 32 or 16 x 16 tiles): the same tiles, entry lists, records, coverage
// and mean-value weights as the forward (held fixed: they are piecewise constant in the
// vertex positions), differentiating each fragment with respect to the attributes its
// corners interpolate. Per record the warp sums its pixels' contributions through a
// shared-memory transpose; the CTA sums warps in shared memory and adds each record's totals to the two vertices
// (wavelength pair endpoints) of each corner once per tile. kTex: the ghost lookups gather
// from the texture object p.ghost_tex.
template <int T, int kS, bool kTex>
__global__ void __launch_bounds__(kThreads, kS == 1 ? 3 : 2)
    k_raster_backward(const float4* __restrict__ vtx, const uint32_t* __restrict__ tile_offsets,
                      const uint32_t* __restrict__ tile_entries, const float* __restrict__ ghost,
                      const float* __restrict__ spectrum, RasterParams p, FragmentConsts fc,
                      const float4* __restrict__ image, const float4* __restrict__ grad_image,
                      float* __restrict__ grad_vtx) {
    constexpr int kBlocks = T * T / 32, kCols = T / 8;
    extern __shared__ float4 smem4[];
    Rec* recbuf = (Rec*)smem4;  // two batches of records
    // Where each record's gradients go: the vertex index of corner 0 at the pair's first
    // wavelength and the sub-step's blend weight, set when the record is built and read by the
    // batch's flush. Three batches' worth: the build of batch t + 2 may run while slower warps
    // still flush batch t, and the build of t + 3 comes after the barrier of t + 1.
    long long* vbase_buf = (long long*)(recbuf + 2 * kBatchRecords);  // [3][kBatchRecords]
    float* tbuf = (float*)(vbase_buf + 3 * kBatchRecords);            // [3][kBatchRecords]
    // per-warp transpose buffers of each lane's 5 attribute gradients and 4 corner weights:
    // [row][lane], rows kRedStride floats apart (16-byte aligned, and the rows that lanes read
    // side by side fall in different bank groups)
    float* red = (tbuf + 3 * kBatchRecords) + (threadIdx.x >> 5) * (kRedRows * kRedStride);
    float* xyz = (tbuf + 3 * kBatchRecords) + 8 * kRedRows * kRedStride;
    float* blend = xyz + 3 * p.maxW * p.WS;
    float* grgb = blend + ((p.WS + 3) & ~3);          // [block * 3 + channel][lane]: dL / d(linear XYZ sum)
    float* rgrad_buf = grgb + 96 * kBlocks;            // two batches of [record][corner * 5 + attribute]
    __shared__ int next_block[2];
    const int tile = blockIdx.x;
    const int tx = tile % p.ntx, ty = tile / p.ntx;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // this CTA's part of the tile's batches; without one nothing is set up (1004 x 1434 without entries: 84 ->
    // 23 us; 26 with one CTA a tile)
    const int per_batch = kBatchRecords / p.WS;
    uint32_t begin = tile_offsets[tile], end = tile_offsets[tile + 1];
    {
        const unsigned batches = (end - begin + per_batch - 1) / per_batch;
        const unsigned b0 = batches * blockIdx.y / gridDim.y, b1 = batches * (blockIdx.y + 1) / gridDim.y;
        end = min(end, begin + b1 * per_batch);
        begin += b0 * per_batch;
        if (begin >= end) return;
    }
    if (threadIdx.x == 0) {
        const float sub_step = 1.0f / (float)p.WS;
        float b = 0.0f;
        for (int i = 0; i < p.WS; i++) {
            blend[i] = b;
            b += sub_step;
        }
    }
    if (p.W > 1) {
        const float sub_step = 1.0f / (float)p.WS;
        const float wl_step = sub_step / (float)p.W;
        for (int w = threadIdx.x; w < p.maxW; w += kThreads) {
            float pos = ((float)w + 0.5f) / (float)p.W;
            for (int i = 0; i < p.WS; i++) {
                for (int c = 0; c < 3; c++)
                    xyz[3 * (w * p.WS + i) + c] = sample_linear(spectrum, RF_SPECTRUM_WIDTH, 1, 4, c, pos, 0.0f, true);
                pos += wl_step;
            }
        }
    }
    // out = AP1(rgb * scale) where any channel of rgb is positive, else 0
    const float scale = p.intensity / (float)(p.W * p.S * p.WS);
    const float4 m0 = xyz_to_ap1(1.0f, 0.0f, 0.0f), m1 = xyz_to_ap1(0.0f, 1.0f, 0.0f),
                 m2 = xyz_to_ap1(0.0f, 0.0f, 1.0f);
#pragma unroll
    for (int k = 0; k < kBlocks / 8; k++) {
        const int blk = warp + 8 * k;
        const int px = tx * T + (blk % kCols) * 8 + (lane & 7), py = ty * T + (blk / kCols) * 4 + (lane >> 3);
        float g0 = 0.0f, g1 = 0.0f, g2 = 0.0f;
        if (px < p.width && py < p.height) {
            const size_t o = (size_t)(p.height - (py + 1)) * p.width + px;
            const float4 out = image[o], g = grad_image[o];
            if (out.x != 0.0f || out.y != 0.0f || out.z != 0.0f) {
                g0 = scale * (m0.x * g.x + m0.y * g.y + m0.z * g.z);
                g1 = scale * (m1.x * g.x + m1.y * g.y + m1.z * g.z);
                g2 = scale * (m2.x * g.x + m2.y * g.y + m2.z * g.z);
            }
        }
        grgb[(3 * blk) * 32 + lane] = g0;
        grgb[(3 * blk + 1) * 32 + lane] = g1;
        grgb[(3 * blk + 2) * 32 + lane] = g2;
    }
    for (int i = threadIdx.x; i < 2 * kBatchRecords * 4 * kGradAttrs; i += kThreads) rgrad_buf[i] = 0.0f;

    const int S = kS ? kS : p.S;
    const int my_entry = threadIdx.x >> 2, my_corner = threadIdx.x & 3;
    const int Q = (p.G - 1) * (p.G - 1), VC = p.G * p.G;
    // Records of the batch at `first` into buffer `dst`, as k_raster builds them: thread j
    // loads and mixes corner j % 4 of entry j / 4 (the four corners of an entry sit in one
    // warp), then one thread per record finishes it. Batches are double-buffered: warps that
    // are done shading batch t build batch t + 1 while the others shade, one barrier per
    // batch, and each batch sums its records' gradients in its own buffer.
    auto build = [&](Rec* dst, uint32_t first, int slot) {
        for (int h = 0; h < (kBatchRecords + 63) / 64; h++) {
            const int e = my_entry + 64 * h;
            if (e < per_batch && first + e < end) {
                const uint32_t entry = tile_entries[first + e];
                CornerLoad c;
                load_corner(vtx, entry, my_corner, p, c);
                for (int i = 0; i < p.WS; i++)
                    store_corner(c, my_corner, blend[i], S, fc, (float)(tx * T * S), (float)(ty * T * S), dst[e * p.WS + i]);
                if (my_corner == 0) {  // where the record's gradients go (the batch's flush)
                    const long long prim = entry / p.maxW;
                    const int w = (int)(entry % p.maxW);
                    const int quad = (int)(prim % Q);
                    const long long v0 = ((prim / Q) * VC + (quad / (p.G - 1)) * p.G + quad % (p.G - 1)) * p.W + w;
                    for (int i = 0; i < p.WS; i++) {
                        vbase_buf[slot * kBatchRecords + e * p.WS + i] = v0;
                        tbuf[slot * kBatchRecords + e * p.WS + i] = blend[i];
                    }
                }
            }
        }
        __syncwarp();  // the four corners of each record are stored
        for (int h = 0; h < (kBatchRecords + 63) / 64; h++) {
            const int e = my_entry + 64 * h;
            if (e < per_batch && first + e < end) {
                const uint32_t entry = tile_entries[first + e];
                for (int i = my_corner; i < p.WS; i += 4)
                    finish_record<4>(p, (int)(entry % p.maxW), i, tx * T * S, ty * T * S, xyz, dst[e * p.WS + i]);
            }
        }
    };
    if (threadIdx.x == 0) {
        next_block[0] = 0;
        next_block[1] = 0;
    }
    __syncthreads();  // blend weights, colours and pixel gradients are set
    if (begin < end) build(recbuf, begin, 0);
    __syncthreads();
    int cur = 0, slot = 0;  // record buffer (batch parity) and flush slot (batch index mod 3)
    for (uint32_t base = begin; base < end; base += per_batch, cur ^= 1, slot = slot == 2 ? 0 : slot + 1) {
        const int n_rec = (int)min((uint32_t)per_batch, end - base) * p.WS;
        const Rec* recs = recbuf + cur * kBatchRecords;
        float* rgrad = rgrad_buf + cur * (kBatchRecords * 4 * kGradAttrs);
#pragma unroll 1
        for (;;) {
            int blk = 0;
            if (lane == 0) blk = atomicAdd(&next_block[cur], 1);
            blk = __shfl_sync(0xffffffffu, blk, 0);
            if (blk >= kBlocks) break;
            const int x0 = tx * T + (blk % kCols) * 8, y0 = ty * T + (blk / kCols) * 4;
            const int px = x0 + (lane & 7), py = y0 + (lane >> 3);
            const int bx0 = x0 * S, by0 = y0 * S, bx1 = bx0 + 8 * S - 1, by1 = by0 + 4 * S - 1;
            const bool in_image = px < p.width && py < p.height;
            const int sx0 = px * S, sy0 = py * S;
            const float g0 = grgb[(3 * blk) * 32 + lane], g1 = grgb[(3 * blk + 1) * 32 + lane],
                        g2 = grgb[(3 * blk + 2) * 32 + lane];
            const bool any_grad = __any_sync(0xffffffffu, g0 != 0.0f || g1 != 0.0f || g2 != 0.0f);
            if (!any_grad) continue;
            // which records can touch this 8 x 4 block, which cover all of it, and which need the
            // exact test at every sample: lanes test 32 records at a time
            const float rx0 = (float)((blk % kCols) * 8 * S), ry0 = (float)((blk / kCols) * 4 * S);
            const float hx = 4.0f * (float)S - 0.5f, hy = 2.0f * (float)S - 0.5f;
            const f2 bxc = pk(rx0 + hx, rx0 + hx), byc = pk(ry0 + hy, ry0 + hy);
            unsigned sel[kBatchRecords / 32], whole[kBatchRecords / 32], wild[kBatchRecords / 32];
#pragma unroll
            for (int m = 0; m < kBatchRecords / 32; m++) {
                const int j = m * 32 + lane;
                bool take = false, all = false, far = false;
                if (j < n_rec) {
                    const Rec& r = recs[j];
                    const int flags = __float_as_int(ld4(r.ef + 12).w);  // with ef[12..14], which rect_coverage reads
                    if (!(flags & 2)) {  // collinear (intersect_quad rejects all) or all-zero
                        const int4 bb = *reinterpret_cast<const int4*>(r.bb);
                        far = !(flags & 1);
                        take = far || !(bx1 < bb.x || bx0 > bb.y || by1 < bb.z || by0 > bb.w);
                        if (take && !far) {
                            const int cov = rect_coverage(r, bxc, byc, hx, hy);
                            take = cov != 0;
                            all = cov == 2;
                        }
                    }
                }
                sel[m] = __ballot_sync(0xffffffffu, take);
                whole[m] = __ballot_sync(0xffffffffu, all);
                wild[m] = __ballot_sync(0xffffffffu, far);
            }
#pragma unroll
            for (int m = 0; m < kBatchRecords / 32; m++) {
                unsigned bits = sel[m];
                while (bits) {
                    const int b = __ffs(bits) - 1;
                    const int j = m * 32 + b;
                    bits &= bits - 1;
                    const Rec& r = recs[j];
                    int hits = 0;
                    if (in_image)
                        hits = (whole[m] >> b) & 1u ? S
                                                    : sample_hits<T>(r, S, (wild[m] >> b) & 1u, rx0, ry0, sx0, sy0, lane);
                    if (!__any_sync(0xffffffffu, hits > 0)) continue;
                    float gw[kGradAttrs] = {0.f, 0.f, 0.f, 0.f, 0.f};
                    float wt[4] = {0.f, 0.f, 0.f, 0.f};
                    if (hits > 0) {
                        scalar_weights(r, rx0 + (float)((lane & 7) * S + S / 2), ry0 + (float)((lane >> 3) * S + S / 2), wt);
                        const float4 col = ld4(r.col);
                        const float dLdf = g0 * col.x + g1 * col.y + g2 * col.z;
                        const float u = scalar_blend(wt, r.uv), v = scalar_blend(wt, r.uv + 4);
                        float dgu, dgv;
                        const float gi = ghost_sample_grad<kTex>(ghost, p, u, v, dgu, dgv);
                        const float st = __saturatef(scalar_blend(wt, r.rs));
                        const float ri = st * st * (3.0f - 2.0f * st);
                        const float dri = (st > 0.0f && st < 1.0f) ? 6.0f * st * (1.0f - st) * (1.0f / (0.95f - 1.0f))
                                                                  : 0.0f;
                        const float ai_raw = scalar_blend(wt, r.inten), ci_raw = scalar_blend(wt, r.refl);
                        const float ai = fmaxf(ai_raw, 0.0f), ci = fmaxf(ci_raw, 0.0f);
                        const float H = (float)hits;
                        const float d = dLdf * H;
                        gw[0] = d * ri * ai * ci * dgu * fc.tsx;
                        gw[1] = d * ri * ai * ci * dgv * fc.tsy;
                        gw[2] = d * gi * ai * ci * dri;
                        gw[3] = ci_raw > 0.0f ? d * gi * ri * ai : 0.0f;
                        gw[4] = ai_raw > 0.0f ? d * gi * ri * ci : 0.0f;
                    }
                    // the warp's sum of each corner attribute's gradient, sum over lanes of
                    // gw[a] * wt[c]: every lane writes its 5 attribute gradients and 4 weights
                    // (rows 0-4 and 5-8), lane k < 20 forms column (a, c) = (k % 5, k / 5)
#pragma unroll
                    for (int a = 0; a < kGradAttrs; a++) red[a * kRedStride + lane] = gw[a];
#pragma unroll
                    for (int c = 0; c < 4; c++) red[(kGradAttrs + c) * kRedStride + lane] = wt[c];
                    __syncwarp();
                    if (lane < 4 * kGradAttrs) {
                        const int a = lane % kGradAttrs, c = lane / kGradAttrs;
                        const float* ga = red + a * kRedStride;
                        const float* wc = red + (kGradAttrs + c) * kRedStride;
                        f2 s01 = 0, s23 = 0;
#pragma unroll
                        for (int q = 0; q < 8; q++) {
                            f2 g01, g23, v01, v23;
                            ld2(ga + 4 * q, g01, g23);
                            ld2(wc + 4 * q, v01, v23);
                            s01 = fma2(g01, v01, s01);
                            s23 = fma2(g23, v23, s23);
                        }
                        const float sum = (lo2(s01) + hi2(s01)) + (lo2(s23) + hi2(s23));
                        if (sum != 0.0f) atomicAdd(&rgrad[j * 4 * kGradAttrs + lane], sum);
                    }
                    __syncwarp();
                }
            }
        }
        if (base + per_batch < end) build(recbuf + (cur ^ 1) * kBatchRecords, base + per_batch, slot == 2 ? 0 : slot + 1);
        // the other counter was last used by the previous batch, behind the last barrier
        if (threadIdx.x == 0) next_block[cur ^ 1] = 0;
        __syncthreads();  // every block of this batch is shaded and the next batch is built
        // each record's gradients to the two vertices of each corner (mix_vertex weights);
        // the buffer is cleared here and written again two batches later, behind the next
        // barrier
        // (thread: one corner of one record; a vertex's attributes in two vector additions)
        for (int idx = threadIdx.x; idx < n_rec * 4; idx += kThreads) {
            const int j = idx >> 2, corner = idx & 3;
            float* src = rgrad + (j * 4 + corner) * kGradAttrs;
            float g[kGradAttrs];
            bool any = false;
#pragma unroll
            for (int a = 0; a < kGradAttrs; a++) {
                g[a] = src[a];
                any = any || g[a] != 0.0f;
            }
            if (!any) continue;
#pragma unroll
            for (int a = 0; a < kGradAttrs; a++) src[a] = 0.0f;
            const float t = tbuf[slot * kBatchRecords + j];
            const int offset = corner == 0 ? 0 : (corner == 1 ? 1 : (corner == 2 ? 1 + p.G : p.G));
            float* v = grad_vtx + 8 * (vbase_buf[slot * kBatchRecords + j] + (long long)offset * p.W);
            const bool vectors = aligned16(grad_vtx);
            add_gradients(v, g, 1.0f - t, vectors);
            if (t != 0.0f) add_gradients(v + 8, g, t, vectors);
        }
    }
}

// The reference's own loop: every pixel scans every mask of its bin (rasterizing.cl:573-654).
__global__ void __launch_bounds__(256) k_raster_masks(const float4* __restrict__ vtx,
                                                      const unsigned long long* __restrict__ masks, int batch_count,
                                                      int B, long long prim_total, const float* __restrict__ ghost,
                                                      const float* __restrict__ spectrum, RasterParams p,
                                                      FragmentConsts fc, float4* __restrict__ image) {
    const int x = blockIdx.x * 16 + (threadIdx.x & 15), y = blockIdx.y * 16 + (threadIdx.x >> 4);
    if (x >= p.width || y >= p.height) return;
    const int bdx = (p.width + B - 1) / B;
    const int bin = (y / B) * bdx + (x / B);
    const int S = p.S;
    const int sx0 = x * S, sy0 = y * S;
    const float sub_step = 1.0f / (float)p.WS;
    const float wl_step = sub_step / (float)p.W;
    const int Q = (p.G - 1) * (p.G - 1), VC = p.G * p.G;
    float rgb[3] = {0.f, 0.f, 0.f};
    Rec r;
    for (int batch = 0; batch < batch_count; batch++) {
        const unsigned long long* q = masks + 4 * ((size_t)bin * batch_count + batch);
        if ((q[0] & 1ull) == 0) continue;
        for (int k = 0; k < RF_BATCH_PRIMITIVE_COUNT; k++) {
            const long long prim = (long long)batch * RF_BATCH_PRIMITIVE_COUNT + k;
            if (prim >= prim_total) continue;
            const int bit = k + 1;
            if (!((q[bit >> 6] >> (bit & 63)) & 1ull)) continue;
            const long long path = prim / Q;
            const int quad = (int)(prim % Q);
            const int row = quad / (p.G - 1), col = quad % (p.G - 1);
            const int c0 = row * p.G + col;
            const int corners[4] = {c0, c0 + 1, c0 + 1 + p.G, c0 + p.G};
            for (int w = 0; w < p.maxW; w++) {
                float sub_pos = 0.0f;
                float wl_pos = ((float)w + 0.5f) / (float)p.W;
                for (int i = 0; i < p.WS; i++) {
                    // the full record, no skipping of invalid endpoints
                    for (int c = 0; c < 4; c++) {
                        const long long vi = (path * VC + corners[c]) * p.W + w;
                        const CornerLoad cl = {vtx[2 * vi], vtx[2 * vi + 1], vtx[2 * vi + 2], vtx[2 * vi + 3]};
                        store_corner(cl, c, sub_pos, S, fc, 0.0f, 0.0f, r);
                    }
                    const int* qq = r.q();
                    const bool never = (edge_i(qq[0], qq[1], qq[2], qq[3], qq[4], qq[5]) == 0 &&
                                       edge_i(qq[0], qq[1], qq[4], qq[5], qq[6], qq[7]) == 0) ||
                                       zero_record(p, r, false);
                    int hits = 0;
                    if (!never)
                        for (int s = 0; s < S; s++)
                            hits += inside_exact(qq, sx0 + s, sy0 + SUB_OFFSETS[S - 1 + s]) ? 1 : 0;
                    float f = 0.0f;
                    if (hits > 0) {
                        f2 we, wo;
                        const float cx = (float)(sx0 + S / 2), cy = (float)(sy0 + S / 2);
                        float general = 1.0f;
                        mean_value_weights(r, pk(cx, cx), pk(cy, cy), S == 1, we, wo, general);
                        f += fragment_fast(r, we, wo, ghost, p, 1.0f) * (float)hits;
                    }
                    if (p.W > 1) {
                        for (int c = 0; c < 3; c++)
                            rgb[c] += sample_linear(spectrum, RF_SPECTRUM_WIDTH, 1, 4, c, wl_pos, 0.0f, true) * f;
                    } else {
                        rgb[0] += f;
                        rgb[1] += f;
                        rgb[2] += f;
                    }
                    sub_pos += sub_step;
                    wl_pos += wl_step;
                }
            }
        }
    }
    float4 out = make_float4(0.f, 0.f, 0.f, 0.f);
    if (rgb[0] > 0.0f || rgb[1] > 0.0f || rgb[2] > 0.0f) {
        const float scale = p.intensity / (float)(p.W * p.S * p.WS);
        out = xyz_to_ap1(rgb[0] * scale, rgb[1] * scale, rgb[2] * scale);
    }
    image[(size_t)(p.height - (y + 1)) * p.width + x] = out;
}

__host__ __device__ inline bool make_params(const rf_raster_args& a, RasterParams& p) {
    if (a.width < 1 || a.height < 1 || a.grid_count < 2 || a.wavelength_count < 1 || a.wavelength_sub_count < 1 ||
        a.path_count < 0 || a.ghost_width < 1 || a.ghost_height < 1)
        return false;
    if (a.sub_steps != 1 && a.sub_steps != 2 && a.sub_steps != 4 && a.sub_steps != 8) return false;
    p.width = a.width;
    p.height = a.height;
    p.S = a.sub_steps;
    p.W = a.wavelength_count;
    p.WS = a.wavelength_sub_count;
    p.G = a.grid_count;
    p.maxW = a.wavelength_count - 1 > 1 ? a.wavelength_count - 1 : 1;
    p.intensity = a.intensity;
    p.ghost_scale = a.ghost_scale;
    p.ghost_w = a.ghost_width;
    p.ghost_h = a.ghost_height;
    p.safe_screen = (float)a.width * a.sub_steps <= 16384.0f && (float)a.height * a.sub_steps <= 16384.0f;
    p.ghost_large = a.ghost_width >= 1 << 22 || a.ghost_height >= 1 << 22 ||
                    (long long)a.ghost_width * a.ghost_height > 0x7fffffffLL;
    p.ghost_tex = 0;  // the texels are loaded unless a launcher sets a texture object
    return true;
}

// Raise a kernel's dynamic shared-memory limit once per device and size, so that later
// launches of it can be captured into a CUDA graph without further attribute calls.
constexpr int kMaxDevices = 64;
template <class K>
int allow_smem(K kernel, size_t bytes, std::atomic<size_t>* allowed) {
    if (bytes <= 48 * 1024) return RF_OK;
    int dev = 0;
    RF_TRY(cuda_status(cudaGetDevice(&dev)));
    if (dev < 0 || dev >= kMaxDevices) return RF_ERR_NOT_SUPPORTED;
    if (bytes <= allowed[dev].load()) return RF_OK;
    RF_TRY(cuda_status(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes)));
    allowed[dev].store(bytes);
    return RF_OK;
}

// A texture object over a caller's ghost texture (float texels, pitch w * 4 bytes, border
// address mode, point filtering, unnormalised coordinates) for ghost_sample_tex, created once
// per device, address and size and kept (at most kMaxGhostTextures; rf_ghost_textures_forget
// drops a device's objects after a device reset). 0 when the address or the row pitch is not
// aligned as textures require, or past the cap; the raster then loads texels.
constexpr size_t kMaxGhostTextures = 4096;
struct GhostTextureEntry {
    int dev;
    const float* ptr;
    int w, h;
    cudaTextureObject_t obj;
};
std::mutex ghost_texture_mutex;
std::vector<GhostTextureEntry> ghost_texture_cache;

unsigned long long ghost_texture_object(const float* ghost, int w, int h) {
    using Entry = GhostTextureEntry;
    std::mutex& mutex = ghost_texture_mutex;
    std::vector<Entry>& cache = ghost_texture_cache;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> lock(mutex);
    for (const Entry& e : cache)
        if (e.dev == dev && e.ptr == ghost && e.w == w && e.h == h) return e.obj;
    // the row pitch must be a multiple of the texture pitch alignment, the base address a
    // multiple of the texture alignment
    int pitch_align = 0, base_align = 0;
    if (cudaDeviceGetAttribute(&pitch_align, cudaDevAttrTexturePitchAlignment, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&base_align, cudaDevAttrTextureAlignment, dev) != cudaSuccess || pitch_align <= 0 ||
        base_align <= 0)
        return 0;
    if (((size_t)w * sizeof(float)) % (size_t)pitch_align != 0 || (uintptr_t)ghost % (uintptr_t)base_align != 0)
        return 0;
    // Objects are kept for the life of the process (one per device, address and size; a
    // kernel in flight may still use any of them, and no synchronisation is allowed here:
    // a caller may be capturing a graph). Past the cap the raster loads the texels.
    if (cache.size() >= kMaxGhostTextures) return 0;
    cudaResourceDesc rd = {};
    rd.resType = cudaResourceTypePitch2D;
    rd.res.pitch2D.devPtr = const_cast<float*>(ghost);
    rd.res.pitch2D.desc = cudaCreateChannelDesc<float>();
    rd.res.pitch2D.width = (size_t)w;
    rd.res.pitch2D.height = (size_t)h;
    rd.res.pitch2D.pitchInBytes = (size_t)w * sizeof(float);
    cudaTextureDesc td = {};
    td.addressMode[0] = td.addressMode[1] = cudaAddressModeBorder;
    td.filterMode = cudaFilterModePoint;
    td.readMode = cudaReadModeElementType;
    td.normalizedCoords = 0;
    cudaTextureObject_t obj = 0;
    if (cudaCreateTextureObject(&obj, &rd, &td, nullptr) != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    cache.push_back({dev, ghost, w, h, obj});
    return obj;
}

template <int T, int kS, int kTex>
int launch_raster_k(const float* vertexes, const uint32_t* offsets, const uint32_t* entries, const uint32_t* order,
                    const float* ghost, const float* spectrum, const RasterParams& p, float* image, cudaStream_t s) {
    static std::atomic<size_t> allowed[kMaxDevices];
    const size_t smem = raster_smem_bytes<T>(p.maxW, p.WS);
    RF_TRY(allow_smem(k_raster<T, kS, kTex>, smem, allowed));
    k_raster<T, kS, kTex><<<p.ntx * ((p.height + T - 1) / T), kThreads, smem, s>>>(
        (const float4*)vertexes, offsets, entries, order, ghost, spectrum, p, fragment_consts(p), (float4*)image);
    return launch_status();
}

template <int T, int kS>
int launch_raster_s(const float* vertexes, const uint32_t* offsets, const uint32_t* entries, const uint32_t* order,
                    const float* ghost, const float* spectrum, RasterParams p, float* image, cudaStream_t s) {
    p.T = T;
    p.ntx = (p.width + T - 1) / T;
    p.ghost_tex = ghost_texture_object(ghost, p.ghost_w, p.ghost_h);
    if (p.ghost_tex)
        return launch_raster_k<T, kS, kGather>(vertexes, offsets, entries, order, ghost, spectrum, p, image, s);
    if (p.ghost_large)  // one kernel for all sample counts
        return launch_raster_k<T, 0, kAnyLoads>(vertexes, offsets, entries, order, ghost, spectrum, p, image, s);
    return launch_raster_k<T, kS, kLoads>(vertexes, offsets, entries, order, ghost, spectrum, p, image, s);
}

template <int T>
int launch_raster(const float* vertexes, const uint32_t* offsets, const uint32_t* entries, const uint32_t* order,
                  const float* ghost, const float* spectrum, RasterParams p, float* image, cudaStream_t s) {
    if (p.S == 1) return launch_raster_s<T, 1>(vertexes, offsets, entries, order, ghost, spectrum, p, image, s);
    // (the sample count known: its tests unroll. Zoom lens, 4 samples: 21.7 ms with a runtime count)
    if (p.S == 2) return launch_raster_s<T, 2>(vertexes, offsets, entries, order, ghost, spectrum, p, image, s);
    if (p.S == 4) return launch_raster_s<T, 4>(vertexes, offsets, entries, order, ghost, spectrum, p, image, s);
    return launch_raster_s<T, 8>(vertexes, offsets, entries, order, ghost, spectrum, p, image, s);
}

template <int T, int kS, int kTex>
int launch_raster_batch(const rf_frame* frames, const rf_batch_sizes& z, const float* vertexes,
                        const uint32_t* tile_offsets, const uint32_t* tile_entries, const float* ghosts,
                        const float* spectrum, const BatchWorkspace& w, long long capacity,
                        const uint64_t* entry_total, float* images, cudaStream_t s) {
    static std::atomic<size_t> allowed[kMaxDevices];
    static std::atomic<int> ctas_per_sm[kMaxDevices];
    // the largest frame layout: 3 * max(W-1,1) * WS colours, WS blend weights (rounded to 4)
    const size_t smem = sizeof(Rec) * 2 * kBatchRecords + sizeof(float) * (3 * z.max_colors + ((z.max_sub + 3) & ~3)) +
                        sizeof(float) * 96 * (T * T / 32);
    RF_TRY(allow_smem(k_raster_batch<T, kS, kTex>, smem, allowed));
    int dev = 0, sms = 0;
    RF_TRY(cuda_status(cudaGetDevice(&dev)));
    RF_TRY(cuda_status(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)));
    int per_sm = ctas_per_sm[dev].load();
    if (per_sm == 0) {
        RF_TRY(cuda_status(
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_raster_batch<T, kS, kTex>, kThreads, smem)));
        per_sm = per_sm > 0 ? per_sm : 1;
        ctas_per_sm[dev].store(per_sm);
    }
    const long long ctas = std::min<long long>((long long)sms * per_sm, z.tiles);
    RF_TRY(cuda_status(cudaMemsetAsync(w.queue, 0, sizeof(uint32_t), s)));
    k_raster_batch<T, kS, kTex><<<(unsigned)ctas, kThreads, smem, s>>>(
        frames, z.frame_count, z.tiles, batch_tile_order(w, z), w.queue, (const unsigned long long*)entry_total,
        capacity, (const float4*)vertexes, tile_offsets, tile_entries, ghosts, spectrum, (float4*)images);
    return launch_status();
}

}  // namespace
}  // namespace rf

extern "C" int rf_raster_batch(const rf_frame* frames, const rf_batch_sizes* sizes, const float* vertexes,
                               const uint32_t* tile_offsets, const uint32_t* tile_entries, const float* ghosts,
                               const float* spectrum, void* workspace, size_t workspace_bytes,
                               int64_t entry_capacity, const uint64_t* entry_total, float* images, void* stream) {
    using namespace rf;
    if (!frames || !sizes || !vertexes || !tile_offsets || !tile_entries || !ghosts || !spectrum || !workspace ||
        !entry_total || !images || entry_capacity < 1)
        return RF_ERR_INVALID_ARG;
    if (!aligned16(vertexes) || !aligned16(images) || !aligned16(workspace)) return RF_ERR_INVALID_ARG;
    const rf_batch_sizes& z = *sizes;
    if (z.tiles < 1) return RF_OK;
    if (z.max_sub < 1 || z.max_sub > kBatchRecords || z.max_colors > 4096) return RF_ERR_INVALID_ARG;
    BatchWorkspace w = batch_layout((char*)workspace, z, entry_capacity);
    if (w.bytes > workspace_bytes) return RF_ERR_INVALID_ARG;
    const bool one = z.max_sub_steps <= 1;  // every frame takes one sample per pixel
    cudaStream_t s = (cudaStream_t)stream;
#define RF_BATCH_LAUNCH(T, S, X)                                                                              \
    launch_raster_batch<T, S, X>(frames, z, vertexes, tile_offsets, tile_entries, ghosts, spectrum, w, entry_capacity, \
                                 entry_total, images, s)
    const bool tex = z.ghost_textures != 0;
    switch (z.tile_size) {
        case 32:
            return one ? (tex ? RF_BATCH_LAUNCH(32, 1, kGather) : RF_BATCH_LAUNCH(32, 1, kAnyLoads))
                       : (tex ? RF_BATCH_LAUNCH(32, 0, kGather) : RF_BATCH_LAUNCH(32, 0, kAnyLoads));
        case 16:
            return one ? (tex ? RF_BATCH_LAUNCH(16, 1, kGather) : RF_BATCH_LAUNCH(16, 1, kAnyLoads))
                       : (tex ? RF_BATCH_LAUNCH(16, 0, kGather) : RF_BATCH_LAUNCH(16, 0, kAnyLoads));
#undef RF_BATCH_LAUNCH
        default:
            return RF_ERR_NOT_SUPPORTED;
    }
}

extern "C" int rf_ghost_textures_forget(void) {
    using namespace rf;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        (void)cudaGetLastError();
        return RF_ERR_CUDA;
    }
    std::lock_guard<std::mutex> lock(ghost_texture_mutex);
    auto& c = ghost_texture_cache;
    c.erase(std::remove_if(c.begin(), c.end(), [dev](const GhostTextureEntry& e) { return e.dev == dev; }), c.end());
    return RF_OK;
}

extern "C" int rf_ghost_texture_object(const float* ghost, int32_t width, int32_t height, uint64_t* texture) {
    using namespace rf;
    if (!ghost || !texture || width < 1 || height < 1) return RF_ERR_INVALID_ARG;
    *texture = ghost_texture_object(ghost, width, height);
    return RF_OK;
}

namespace {
int raster_entry(const float* vertexes, const uint32_t* tile_offsets, const uint32_t* tile_entries,
                 const uint32_t* tile_order, const float* ghost, const float* spectrum, const rf_raster_args* args,
                 float* image, void* stream) {
    using namespace rf;
    if (!vertexes || !tile_offsets || !ghost || !spectrum || !args || !image) return RF_ERR_INVALID_ARG;
    if (!aligned16(vertexes) || !aligned16(image)) return RF_ERR_INVALID_ARG;
    RasterParams p;
    if (!make_params(*args, p)) return RF_ERR_INVALID_ARG;
    if (p.WS > kBatchRecords || p.maxW * p.WS > 4096) return RF_ERR_INVALID_ARG;
    switch (tile_size_of(*args)) {
        case 32:
            return launch_raster<32>(vertexes, tile_offsets, tile_entries, tile_order, ghost, spectrum, p, image,
                                     (cudaStream_t)stream);
        case 16:
            return launch_raster<16>(vertexes, tile_offsets, tile_entries, tile_order, ghost, spectrum, p, image,
                                     (cudaStream_t)stream);
        default:
            return RF_ERR_NOT_SUPPORTED;
    }
}
}  // namespace

extern "C" int rf_raster(const float* vertexes, const uint32_t* tile_offsets, const uint32_t* tile_entries,
                         const float* ghost, const float* spectrum, const rf_raster_args* args, float* image,
                         void* stream) {
    return raster_entry(vertexes, tile_offsets, tile_entries, nullptr, ghost, spectrum, args, image, stream);
}

extern "C" int rf_raster_ordered(const float* vertexes, const uint32_t* tile_offsets, const uint32_t* tile_entries,
                                 const uint32_t* tile_order, const float* ghost, const float* spectrum,
                                 const rf_raster_args* args, float* image, void* stream) {
    if (!tile_order) return RF_ERR_INVALID_ARG;
    return raster_entry(vertexes, tile_offsets, tile_entries, tile_order, ghost, spectrum, args, image, stream);
}

extern "C" int rf_raster_masks(const float* vertexes, const uint64_t* masks, int32_t batch_count, const float* ghost,
                               const float* spectrum, const rf_raster_args* args, float* image, void* stream) {
    using namespace rf;
    if (!vertexes || !masks || !ghost || !spectrum || !args || !image || batch_count < 0) return RF_ERR_INVALID_ARG;
    RasterParams p;
    if (!make_params(*args, p)) return RF_ERR_INVALID_ARG;
    const long long prim_total = (long long)args->path_count * (args->grid_count - 1) * (args->grid_count - 1);
    dim3 grid((p.width + 15) / 16, (p.height + 15) / 16);
    k_raster_masks<<<grid, 256, 0, (cudaStream_t)stream>>>((const float4*)vertexes, (const unsigned long long*)masks,
                                                           batch_count, args->bin_size, prim_total, ghost, spectrum,
                                                           p, fragment_consts(p), (float4*)image);
    return launch_status();
}

extern "C" int rf_raster_backward(const float* vertexes, const uint32_t* tile_offsets, const uint32_t* tile_entries,
                                  const float* ghost, const float* spectrum, const rf_raster_args* args,
                                  const float* image, const float* grad_image, float* grad_vertexes, void* stream) {
    using namespace rf;
    if (!vertexes || !tile_offsets || !ghost || !spectrum || !args || !image || !grad_image || !grad_vertexes)
        return RF_ERR_INVALID_ARG;
    if (!aligned16(vertexes) || !aligned16(image) || !aligned16(grad_image) || ((uintptr_t)grad_vertexes & 3u) != 0)
        return RF_ERR_INVALID_ARG;
    RasterParams p;
    if (!make_params(*args, p)) return RF_ERR_INVALID_ARG;
    if (p.WS > kBatchRecords || p.maxW * p.WS > 4096) return RF_ERR_INVALID_ARG;
    const int T = tile_size_of(*args);
    if (T != 32 && T != 16) return RF_ERR_NOT_SUPPORTED;
    cudaStream_t s = (cudaStream_t)stream;
    const long long n_vertices = (long long)args->path_count * args->grid_count * args->grid_count *
                                 args->wavelength_count + 1;
    RF_TRY(cuda_status(cudaMemsetAsync(grad_vertexes, 0, sizeof(float) * 8 * (size_t)n_vertices, s)));
    p.T = T;
    p.ntx = (p.width + T - 1) / T;
    const int nty = (p.height + T - 1) / T;
    const size_t smem = sizeof(Rec) * 2 * kBatchRecords + (sizeof(long long) + sizeof(float)) * 3 * kBatchRecords +
                        sizeof(float) * (3 * p.maxW * p.WS + ((p.WS + 3) & ~3)) +
                        sizeof(float) * (96 * (T * T / 32) + 2 * kBatchRecords * 4 * kGradAttrs +
                                         8 * kRedRows * kRedStride);
    const FragmentConsts fc = fragment_consts(p, 0.5);  // texel coordinates without ghost_footprint's shift
    const float4 *im = (const float4*)image, *gim = (const float4*)grad_image;
    // CTAs per tile: the sums are atomic, so a tile's batches can be shared out, up to 8 ways while
    // there are few tiles (one CTA per tile leaves SMs idle at the end of the launch, or
    // altogether on small images). 1 / 2 / 4 / 8 ways: 512 x 512 (1024 tiles) 3.21 / 2.93 / 2.78 /
    // 2.73 ms, 200 x 300 1.22 / 0.69 / 0.52 / 0.45 ms, 79 x 85 2.63 / 1.37 / 0.83 / 0.48 ms.
    const int parts = std::min(8, std::max(1, 8192 / (p.ntx * nty)));
    const dim3 grid((unsigned)(p.ntx * nty), (unsigned)parts);
    p.ghost_tex = ghost_texture_object(ghost, p.ghost_w, p.ghost_h);
#define RF_BACKWARD_LAUNCH(TT, SS, X)                                                                         \
    do {                                                                                                      \
        static std::atomic<size_t> allowed[kMaxDevices];                                                      \
        RF_TRY(allow_smem(k_raster_backward<TT, SS, X>, smem, allowed));                                      \
        k_raster_backward<TT, SS, X><<<grid, kThreads, smem, s>>>((const float4*)vertexes, tile_offsets,       \
                                                                  tile_entries, ghost, spectrum, p, fc, im, gim, \
                                                                  grad_vertexes);                             \
    } while (0)
    const bool tex = p.ghost_tex != 0;
    if (T == 32 && p.S == 1) {
        if (tex) RF_BACKWARD_LAUNCH(32, 1, true); else RF_BACKWARD_LAUNCH(32, 1, false);
    } else if (T == 32) {
        if (tex) RF_BACKWARD_LAUNCH(32, 0, true); else RF_BACKWARD_LAUNCH(32, 0, false);
    } else if (p.S == 1) {
        if (tex) RF_BACKWARD_LAUNCH(16, 1, true); else RF_BACKWARD_LAUNCH(16, 1, false);
    } else {
        if (tex) RF_BACKWARD_LAUNCH(16, 0, true); else RF_BACKWARD_LAUNCH(16, 0, false);
    }
#undef RF_BACKWARD_LAUNCH
    return launch_status();
}

#ifdef RF_RASTER_STATS
// Statistics build only: read (and zero) the counters of the k_raster launches since the
// last call. out[8]: record iterations, whole-block record iterations, fragments, fragments
// of whole-block records, block visits, fragments with a zero smoothstep factor, record
// iterations where every shaded pixel has one (those two with more than one sample per
// pixel), warp steps of the one-sample shading loop.
extern "C" int rf_raster_stats(unsigned long long* out) {
    using namespace rf;
    if (!out) return RF_ERR_INVALID_ARG;
    RF_TRY(cuda_status(cudaMemcpyFromSymbol(out, g_raster_stats, sizeof(unsigned long long) * kRasterStats)));
    const unsigned long long zero[kRasterStats] = {};
    RF_TRY(cuda_status(cudaMemcpyToSymbol(g_raster_stats, zero, sizeof zero)));
    return RF_OK;
}
#endif
