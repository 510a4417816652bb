// rf_trace_core.cuh — per-ray trace code shared by the trace (rf_trace.cu) and its adjoint
// (rf_adjoint.cu). Both translation units are compiled without floating-point contraction,
// so a ray recomputed by the adjoint follows the forward trace's arithmetic exactly.
//
// Follows realflare/api/tasks/cl/raytracing.cl: init_ray (178-215), the element loop of
// raytrace (218-359), intersect (123-175), refract / reflect (70-102), dispersion
// (107-120), fresnel (1-16) and fresnel_ar (18-59).
#pragma once

#include <math.h>

#include "rf_common.cuh"

namespace rf {
namespace {

constexpr int kMaxElements = 128;
constexpr int kMaxGrid = 2048;  // (float)ray_id / G is exact enough for trunc() up to 2048

struct TraceParams {
    long long n_rays;
    int E, aperture, P, W, G, R;
    float cmin, layer_n0, layer_n1;
    float dir[3];        // normalize(-direction.xyz), host-computed in FP32
    float grid[kMaxGrid];  // grid_length * ((float)i / (G - 1) - 0.5), rounded from double
};

struct alignas(16) SmemElement {
    float radius, center, height, ior;
    int coating, layers;
    float d0, d1;
};

struct Hit {
    float px, py, pz, nx, ny, nz;
    bool hit;
};

// The reciprocal, correctly rounded like sqrt_rn (rf_common.cuh): |x| in [2^-100, 2^100].
__device__ __forceinline__ float rcp_rn(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return __fmaf_rn(__fmaf_rn(-x, y, 1.0f), y, y);
}

// Inlining of the reflection-only functions (RF_CORE_COLD: the Fresnel variants) and of the
// sphere/plane intersection (RF_CORE_HOT); a unit may define them __noinline__ before
// including this file (same arithmetic either way: nothing is contracted across calls).
#ifndef RF_CORE_COLD
#define RF_CORE_COLD __forceinline__
#endif
#ifndef RF_CORE_HOT
#define RF_CORE_HOT __forceinline__
#endif
__device__ RF_CORE_HOT Hit intersect(float px, float py, float pz, float dx, float dy, float dz,
                                         const SmemElement& e) {
    Hit h;
    h.px = h.py = h.pz = h.nx = h.ny = h.nz = 0.0f;
    h.hit = false;
    if (dz == 0.0f) return h;
    const float radius = e.radius, cz = -e.center;
    if (radius == 0.0f) {
        float t = (cz - pz) / dz;
        h.px = px + dx * t;
        h.py = py + dy * t;
        h.pz = pz + dz * t;
        h.nx = 0.0f;
        h.ny = 0.0f;
        h.nz = (dz < 0.0f) ? 1.0f : -1.0f;
        h.hit = true;
        return h;
    }
    // u = (0, 0, cz) - p; products and differences as the reference rounds them (signs moved, which
    // is exact)
    const float uz = cz - pz;
    const float proj = -px * dx + -py * dy + uz * dz;
    const float u1x = dx * proj, u1y = dy * proj, u1z = dz * proj;
    const float ex = -px - u1x, ey = -py - u1y, ez = uz - u1z;
    const float d2 = ex * ex + ey * ey + ez * ez;
    const float d = sqrt_rn(d2);
    if (d > fabsf(radius) || d2 > 1e37f) return h;
    const float sgn = (radius * dz) > 0.0f ? -1.0f : 1.0f;
    const float m = sqrt_rn(radius * radius - d * d) * sgn;
    h.px = (px + u1x) - dx * m;
    h.py = (py + u1y) - dy * m;
    h.pz = (pz + u1z) - dz * m;
    const float qz = h.pz - cz;
    const float inv = rcp_rn(sqrt_rn(h.px * h.px + h.py * h.py + qz * qz)) * sgn;
    h.nx = h.px * inv;
    h.ny = h.py * inv;
    h.nz = qz * inv;
    h.hit = true;
    return h;
}

__device__ __forceinline__ float incident_angle(float dx, float dy, float dz, const Hit& h) {
    float c = -dx * h.nx + -dy * h.ny + -dz * h.nz;
    return acosf(clampf(c, -1.0f, 1.0f));
}

// The reference's reflectances (fresnel, fresnel_ar; raytracing.cl:1-59) take the incidence angle
// and evaluate sines and tangents of sums and differences of it and the refracted angles. With the
// refraction law they are rational in the cosines, which is how they are evaluated here (c0, s0:
// cosine and sine of the incidence angle, from the incidence cosine itself): no inverse and
// forward trigonometric functions, and no 0 / 0 at normal incidence (where the reference adds
// 1e-9 to the angle). Total reflection gives NaN, as the reference's arcsine does.
__device__ __forceinline__ float incident_cos(float dx, float dy, float dz, const Hit& h) {
    return clampf(-dx * h.nx + -dy * h.ny + -dz * h.nz, -1.0f, 1.0f);
}
__device__ __forceinline__ float refracted_cos(float s) {
    const float x = 1.0f - s * s;
    return x < 0.0f ? __int_as_float(0x7fffffff) : sqrt_rn(x);
}
// interface reflectances of s- and p-polarised light: -sin(i - j) / sin(i + j) and tan(i - j) /
// tan(i + j) for angles i, j with ni sin(i) = nj sin(j)
__device__ __forceinline__ void interface_r(float ni, float ci, float nj, float cj, float& rs, float& rp) {
    rs = (ni * ci - nj * cj) * rcp_rn(ni * ci + nj * cj);
    rp = (nj * ci - ni * cj) * rcp_rn(nj * ci + ni * cj);
}

// theta = incident + 1e-9 (a double sum there); only angles below 0.02 rad are close enough to 1e-9 for
// the double sum to differ from `incident`
__device__ __forceinline__ float angle_of(float incident) {
    return incident < 0.02f ? (float)((double)incident + 1e-9) : incident;
}
// The reference's form of the uncoated reflectance (see fresnel_ar_angle).
__device__ RF_CORE_COLD float fresnel_angle(float theta0, float n1, float n2) {
    float theta1 = asinf(sinf(theta0) * n1 / n2);
    float cosi = cosf(theta0);
    float cost = cosf(theta1);
    float rs = ((n1 * cosi) - (n2 * cost)) / ((n1 * cosi) + (n2 * cost));
    float rp = ((n1 * cost) - (n2 * cosi)) / ((n1 * cost) + (n2 * cosi));
    return (rs * rs + rp * rp) / 2.0f;
}

// Between equal indices (in every lens: back from the stop at the element before it) the reflectance is
// 0, which the trace does not multiply by (the reference's rule), or a rounding residue, which it
// does: a whole ghost lit or dark by last bits. There the reference's form decides.
__device__ RF_CORE_COLD float fresnel(float c0, float s0, float n1, float n2) {
    if (n1 == n2) {
        const float theta = angle_of(acosf(c0));
        __builtin_assume(fabsf(theta) < 8.0f);  // (sinf and cosf without their slow path)
        return fresnel_angle(theta, n1, n2);
    }
    float rs, rp;
    interface_r(n1, c0, n2, refracted_cos(s0 * (n1 / n2)), rs, rp);
    return (rs * rs + rp * rp) / 2.0f;
}

__device__ RF_CORE_COLD float fresnel_ar(float c0, float s0, float lambda, float d1, float n0, float n1, float n2) {
    const float s1 = s0 * n0 / n1;
    const float c1 = refracted_cos(s1), c2 = refracted_cos(s0 * n0 / n2);
    float rs01, rp01, rs12, rp12;
    interface_r(n0, c0, n1, c1, rs01, rp01);
    interface_r(n1, c1, n2, c2, rs12, rp12);
    const float ts01 = 2.0f * (n0 * c0) * rcp_rn(n0 * c0 + n1 * c1);
    const float tp01 = ts01 * (c0 * c1 + s0 * s1);  // cos(theta0 - theta1)
    const float ris = ts01 * ts01 * rs12;
    const float rip = tp01 * tp01 * rp12;
    // delay sqrt(dx^2 + dy^2) - dx sin(theta0), dy = d1 n1, dx = tan(theta1) dy
    const float dy = d1 * n1;
    const float c = cosf(4.0f * RF_MPI_F / lambda * ((fabsf(dy) - dy * s1 * s0) * rcp_rn(c1)));
    const float out_s2 = rs01 * rs01 + ris * ris + 2.0f * rs01 * ris * c;
    const float out_p2 = rp01 * rp01 + rip * rip + 2.0f * rp01 * rip * c;
    return (out_s2 + out_p2) / 2.0f;
}

// Exact two-layer thin-film reflectance (no reference counterpart; the same definition as
// the oracle): incident medium n0 | layer a | layer b | substrate n2, s/p averaged.
__device__ __forceinline__ float stack_r2(float r01, float r12, float r23, float s1, float c1, float s2, float c2) {
    float nre = r12 + r23 * c2, nim = r23 * s2;
    float dre = 1.0f + r12 * r23 * c2, dim = r12 * r23 * s2;
    float den = rcp_rn(dre * dre + dim * dim);
    float ire = (nre * dre + nim * dim) * den;
    float iim = (nim * dre - nre * dim) * den;
    float ere = ire * c1 - iim * s1, eim = ire * s1 + iim * c1;
    float tre = r01 + ere, tim = eim;
    float bre = 1.0f + r01 * ere, bim = r01 * eim;
    return (tre * tre + tim * tim) * rcp_rn(bre * bre + bim * bim);
}
__device__ RF_CORE_COLD float fresnel_two_layer(float c0, float s0, float lambda, float n0, float na, float da,
                                                   float nb, float db, float n2) {
    const float ns = n0 * s0;
    const float ca = refracted_cos(ns / na), cb = refracted_cos(ns / nb), c2 = refracted_cos(ns / n2);
    float rs01, rp01, rs12, rp12, rs23, rp23;
    interface_r(n0, c0, na, ca, rs01, rp01);
    interface_r(na, ca, nb, cb, rs12, rp12);
    interface_r(nb, cb, n2, c2, rs23, rp23);
    const float phase = 4.0f * RF_MPI_F / lambda;
    float sd1, cd1, sd2, cd2;
    sincosf(phase * na * da * ca, &sd1, &cd1);
    sincosf(phase * nb * db * cb, &sd2, &cd2);
    return (stack_r2(rs01, rs12, rs23, sd1, cd1, sd2, cd2) + stack_r2(rp01, rp12, rp23, sd1, cd1, sd2, cd2)) / 2.0f;
}

// The same reflectances evaluated from the incidence angle, operation by operation as the reference
// writes them and as the adjoint's duals differentiate them. The adjoint's re-trace and the
// forward trace of a differentiated render use these: where a gradient is a small difference of
// large terms (the light's), the reflectances' last bits show in it.
__device__ RF_CORE_COLD float fresnel_ar_angle(float theta0, float lambda, float d1, float n0, float n1, float n2) {
    float s0 = sinf(theta0);
    float theta1 = asinf(s0 * n0 / n1);
    float theta2 = asinf(s0 * n0 / n2);
    float rs01 = -sinf(theta0 - theta1) / sinf(theta0 + theta1);
    float rp01 = tanf(theta0 - theta1) / tanf(theta0 + theta1);
    float ts01 = 2.0f * sinf(theta1) * cosf(theta0) / sinf(theta0 + theta1);
    float tp01 = ts01 * cosf(theta0 - theta1);
    float rs12 = -sinf(theta1 - theta2) / sinf(theta1 + theta2);
    float rp12 = tanf(theta1 - theta2) / tanf(theta1 + theta2);
    float ris = ts01 * ts01 * rs12;
    float rip = tp01 * tp01 * rp12;
    float dy = d1 * n1;
    float dx = tanf(theta1) * dy;
    float delay = sqrtf(dx * dx + dy * dy);
    float rel_phase = 4.0f * RF_MPI_F / lambda * (delay - dx * s0);
    float c = cosf(rel_phase);
    float out_s2 = rs01 * rs01 + ris * ris + 2.0f * rs01 * ris * c;
    float out_p2 = rp01 * rp01 + rip * rip + 2.0f * rp01 * rip * c;
    return (out_s2 + out_p2) / 2.0f;
}

__device__ __forceinline__ void interface_r_div(float ni, float ci, float nj, float cj, float& rs, float& rp) {
    rs = (ni * ci - nj * cj) / (ni * ci + nj * cj);
    rp = (nj * ci - ni * cj) / (nj * ci + ni * cj);
}
__device__ __forceinline__ float stack_r2_div(float r01, float r12, float r23, float d1, float d2) {
    float s2, c2, s1, c1;
    sincosf(d2, &s2, &c2);
    sincosf(d1, &s1, &c1);
    float nre = r12 + r23 * c2, nim = r23 * s2;
    float dre = 1.0f + r12 * r23 * c2, dim = r12 * r23 * s2;
    float den = dre * dre + dim * dim;
    float ire = (nre * dre + nim * dim) / den;
    float iim = (nim * dre - nre * dim) / den;
    float ere = ire * c1 - iim * s1, eim = ire * s1 + iim * c1;
    float tre = r01 + ere, tim = eim;
    float bre = 1.0f + r01 * ere, bim = r01 * eim;
    return (tre * tre + tim * tim) / (bre * bre + bim * bim);
}
__device__ RF_CORE_COLD float fresnel_two_layer_angle(float theta0, float lambda, float n0, float na, float da,
                                                   float nb, float db, float n2) {
    float s0, c0;
    sincosf(theta0, &s0, &c0);
    float sa = n0 * s0 / na, sb = n0 * s0 / nb, s2 = n0 * s0 / n2;
    float ca = sqrtf(1.0f - sa * sa), cb = sqrtf(1.0f - sb * sb), c2 = sqrtf(1.0f - s2 * s2);
    float rs01, rp01, rs12, rp12, rs23, rp23;
    interface_r_div(n0, c0, na, ca, rs01, rp01);
    interface_r_div(na, ca, nb, cb, rs12, rp12);
    interface_r_div(nb, cb, n2, c2, rs23, rp23);
    float phase = 4.0f * RF_MPI_F / lambda;
    float d1 = phase * na * da * ca;
    float d2 = phase * nb * db * cb;
    return (stack_r2_div(rs01, rs12, rs23, d1, d2) + stack_r2_div(rp01, rp12, rp23, d1, d2)) / 2.0f;
}

// dispersion, raytracing.cl:107-120 (lambda * 1e-3 is a double expression there)
__device__ __forceinline__ float dispersion(float lambda, const float* c) {
    float l = (float)((double)lambda * 1e-3);
    float l2 = l * l;
    float d0 = (c[0] * l2) / (l2 - c[1]);
    float d1 = (c[2] * l2) / (l2 - c[3]);
    float d2 = (c[4] * l2) / (l2 - c[5]);
    return sqrtf(1.0f + d0 + d1 + d2);
}

// reflect (raytracing.cl:96-102): d + n * 2 (n . -d)
__device__ __forceinline__ void reflect_dir(float& dx, float& dy, float& dz, const Hit& h) {
    float k = 2.0f * (h.nx * -dx + h.ny * -dy + h.nz * -dz);
    dx = dx + h.nx * k;
    dy = dy + h.ny * k;
    dz = dz + h.nz * k;
}

// refract (raytracing.cl:70-86) with o = n1 / n2; the direction is zeroed past total
// internal reflection (the reference multiplies by 0 there and by 1 elsewhere)
__device__ __forceinline__ void refract_dir(float& dx, float& dy, float& dz, const Hit& h, float o) {
    const float cost = -dx * h.nx + -dy * h.ny + -dz * h.nz;
    const float sint2 = (o * o) * (1.0f - cost * cost);
    const float k = o * cost - sqrt_rn(fabsf(1.0f - sint2));
    dx = o * dx + k * h.nx;
    dy = o * dy + k * h.ny;
    dz = o * dz + k * h.nz;
    if (!(sint2 < 1.0f)) {
        dx *= 0.0f;
        dy *= 0.0f;
        dz *= 0.0f;
    }
}

// Per-frame constants of the trace.
struct TraceFrame {
    int E, aperture, W, G, R;
    float cmin, layer_n0, layer_n1;
    float dir[3];  // normalize(-direction.xyz), host-computed in FP32
};

// The reflectance of element e from the angle theta0 at which a ray hits it from a medium of index n1, the
// element's own index being n2.
__device__ __forceinline__ float reflectance_angle(float theta0, const SmemElement& e, float n1, float n2,
                                                   float wavelength, const TraceFrame& f) {
    const float nc = fmaxf(sqrtf(n1 * n2), f.cmin);
    const float d1 = e.layers == 1 ? e.d0 : (float)e.coating / (4.0f * nc);
    if (e.layers == 2) return fresnel_two_layer_angle(theta0, wavelength, n1, f.layer_n0, e.d0, f.layer_n1, e.d1, n2);
    if (e.layers == 1 || e.coating > 0) return fresnel_ar_angle(theta0, wavelength, d1, n1, nc, n2);
    return fresnel_angle(theta0, n1, n2);
}
// Two layers without thickness between equal indices, which is no coating either (see fresnel): the reference's form
// of the stack (fresnel_two_layer_angle) with the phases' sines 0 and cosines 1.
__device__ __forceinline__ float bare_layers_r2(float r01, float r12, float r23) {
    const float nre = r12 + r23, dre = 1.0f + r12 * r23;
    const float ere = (nre * dre) / (dre * dre);
    const float tre = r01 + ere, bre = 1.0f + r01 * ere;
    return (tre * tre) / (bre * bre);
}
__device__ RF_CORE_COLD float bare_layers(float c, float n, float na, float nb) {
    const float theta = angle_of(acosf(c));
    __builtin_assume(fabsf(theta) < 8.0f);
    float s0, c0;
    sincosf(theta, &s0, &c0);
    const float sa = n * s0 / na, sb = n * s0 / nb, s2 = n * s0 / n;
    const float ca = sqrtf(1.0f - sa * sa), cb = sqrtf(1.0f - sb * sb), c2 = sqrtf(1.0f - s2 * s2);
    float rs01, rp01, rs12, rp12, rs23, rp23;
    interface_r_div(n, c0, na, ca, rs01, rp01);
    interface_r_div(na, ca, nb, cb, rs12, rp12);
    interface_r_div(nb, cb, n, c2, rs23, rp23);
    return (bare_layers_r2(rs01, rs12, rs23) + bare_layers_r2(rp01, rp12, rp23)) / 2.0f;
}

// The same from the cosine and sine of the angle.
__device__ __forceinline__ float reflectance_cos(float c0, float s0, const SmemElement& e, float n1, float n2,
                                                 float wavelength, const TraceFrame& f) {
    const float nc = fmaxf(sqrtf(n1 * n2), f.cmin);
    const float d1 = e.layers == 1 ? e.d0 : (float)e.coating / (4.0f * nc);
    if (e.layers == 2 && n1 == n2 && e.d0 == 0.0f && e.d1 == 0.0f) return bare_layers(c0, n1, f.layer_n0, f.layer_n1);
    if (e.layers == 2) return fresnel_two_layer(c0, s0, wavelength, n1, f.layer_n0, e.d0, f.layer_n1, e.d1, n2);
    if (e.layers == 1 || e.coating > 0) return fresnel_ar(c0, s0, wavelength, d1, n1, nc, n2);
    return fresnel(c0, s0, n1, n2);
}
// The reflectance of element e for a ray (dx, dy, dz) that hits it from a medium of index n1, the
// element's own index being n2. kAngles: from the incidence angle.
template <bool kAngles>
__device__ __forceinline__ float surface_reflectance(float dx, float dy, float dz, const Hit& h, const SmemElement& e,
                                                     float n1, float n2, float wavelength, const TraceFrame& f) {
    if (kAngles) return reflectance_angle(angle_of(incident_angle(dx, dy, dz, h)), e, n1, n2, wavelength, f);
    const float c0 = incident_cos(dx, dy, dz, h);
    return reflectance_cos(c0, sqrt_rn((1.0f - c0) * (1.0f + c0)), e, n1, n2, wavelength, f);
}

// Observer of a traced ray: step() sees the ray entering each element (element index,
// position, direction), hit() each successful intersection (loop step index, the hit, the
// incoming direction, whether the element is flat), rrel() each candidate of the running
// maximum before it is taken, reflect() each reflection. The adjoint records steps, the
// intersection trace records hits.

// A wavelength's entry for one element: its index and the index ratios n1 / n2 a ray refracted there
// sees going towards the light (dz < 0: n1 is the element before) or the sensor (the element after);
// an index outside the lens is 1.
struct IorEntry {
    float ior, down, up;
};
template <class IorOf>
__device__ __forceinline__ IorEntry ior_entry(int el, int E, IorOf ior_of) {
    IorEntry r;
    r.ior = ior_of(el);
    r.down = (el > 0 ? ior_of(el - 1) : 1.0f) / r.ior;
    r.up = (el + 1 < E ? ior_of(el + 1) : 1.0f) / r.ior;
    return r;
}

// One ray: init_ray (raytracing.cl:178-215) from grid point (grid_x, grid_y), then the
// element loop of raytrace (218-359). ior_row: this ray's wavelength row of the (wavelength,
// element) index table in shared memory, or nullptr to evaluate dispersion per element.
// ratio_row: the row's index ratios, or nullptr to divide. kAngles: the reflectances from angles.
template <bool kAngles, class Recorder>
__device__ __forceinline__ void trace_ray_rec(const SmemElement* __restrict__ se, const float* ior_row,
                                              const float2* ratio_row, bool disperse,
                                              const float* __restrict__ coef_base, float wavelength, int2 path,
                                              float grid_x, float grid_y, const TraceFrame& f, float out[6],
                                              Recorder& rec) {
    const int E = f.E;
    auto ior_of = [&](int el) -> float {
        if (ior_row) return ior_row[el];
        float n = se[el].ior;
        if (disperse && n > 1.0f) n = dispersion(wavelength, coef_base + (size_t)el * 16);
        return n;
    };

    float px = grid_x, py = -grid_y, pz = 1.0f;
    {
        Hit h0 = intersect(px, py, pz, 0.0f, 0.0f, -1.0f, se[0]);
        px = h0.px;  // zero when the grid point misses element 0
        py = h0.py;
        pz = h0.pz;
    }
    float dx = f.dir[0], dy = f.dir[1], dz = f.dir[2];
    px = px - dx;
    py = py - dy;
    pz = pz - dz;
    float apt_x = 0.0f, apt_y = 0.0f, rrel = 0.0f, refl = 1.0f;

    int delta = 1;
    int target = path.x, target2 = path.y;  // the element the ray reflects at next, and then
    // rrel = max |xy| / height: an element whose ratio is below the maximum by more than the
    // roundings (2^-20) is passed over by comparing squares; the others are evaluated exactly
    float rrel2 = 0.0f;
    int lens_id, inter_id = 0;  // inter_id: loop steps so far (raytracing.cl:256)
    for (lens_id = 0; lens_id >= 0 && lens_id < E; lens_id += delta, inter_id++) {
        const SmemElement& e = se[lens_id];
        rec.step(lens_id, px, py, pz, dx, dy, dz);
        Hit h = intersect(px, py, pz, dx, dy, dz, e);
        if (!h.hit) break;
        rec.hit(inter_id, h, dx, dy, dz, e.radius == 0.0f);
        px = h.px;
        py = h.py;
        pz = h.pz;
        if (lens_id == f.aperture) {
            apt_x = h.px / e.height;
            apt_y = h.py / e.height;
            continue;
        }
        const float xy2 = h.px * h.px + h.py * h.py;
        if (!(xy2 < rrel2 * (e.height * e.height))) {
            const float r_here = sqrtf(xy2) / e.height;
            rec.rrel(r_here, rrel);
            rrel = fmaxf(rrel, r_here);
            rrel2 = rrel * rrel * (1.0f - 0x1p-20f);
        }
        if (lens_id == E - 1) continue;
        if (lens_id == target) {
            target = target2;
            target2 = -1;
            delta = -delta;
            const int n_index = (dz < 0.0f) ? lens_id - 1 : lens_id + 1;
            const float n1 = (0 <= n_index && n_index < E) ? ior_of(n_index) : 1.0f;
            const float n2 = ior_of(lens_id);
            rec.reflect();
            const float reflectance = surface_reflectance<kAngles>(dx, dy, dz, h, e, n1, n2, wavelength, f);
            reflect_dir(dx, dy, dz, h);
            if (reflectance > 0.0f) refl *= reflectance;
        } else {
            float o;
            if (ratio_row) {
                const float2 q = ratio_row[lens_id];
                o = dz < 0.0f ? q.x : q.y;
            } else {
                const int n_index = (dz < 0.0f) ? lens_id - 1 : lens_id + 1;
                o = ((0 <= n_index && n_index < E) ? ior_of(n_index) : 1.0f) / ior_of(lens_id);
            }
            refract_dir(dx, dy, dz, h, o);
            if (dz == 0.0f) break;
        }
    }
    if (lens_id >= 0 && lens_id < E) refl = __int_as_float(0x7fffffff);
    out[0] = px;
    out[1] = py;
    out[2] = apt_x;
    out[3] = apt_y;
    out[4] = rrel;
    out[5] = refl;
}

// A thread traces one grid point and wavelength along several ghost paths at once. Paths differ only
// from their reflections on: the way to the first reflecting element serves every path that
// reflects there or later, the way back from it every path of that first element, and only the last
// leg from the second reflection is a path's own. Sorted by (first element, second element
// descending) the paths are the leaves of a tree of depth two that is walked once, a ray that goes
// on past a reflection being kept meanwhile. Every ray sees the operations of its own trace in
// their order, so nothing changes in the results; 120 paths of 18 elements take 16 at a time 1860
// surface interactions instead of 3648, 276 of 26 elements 5890 instead of 12064, and half the
// first reflections' reflectances are shared.
constexpr int kMaxPaths = kMaxTracePaths;
static_assert(kMaxPaths <= 32, "one lane of a warp per path");
struct PathList {
    // first and second reflecting element (E, -1: none is reached), the path's index, the next path
    // that differs and the next with another first element
    int x[kMaxPaths], y[kMaxPaths], id[kMaxPaths], next[kMaxPaths], next_x[kMaxPaths];
};
// Paths [first, first + count) (count <= kMaxPaths) into l; the first warp of a block calls it.
__device__ __forceinline__ void stage_paths(const int2* __restrict__ paths, int first, int count, int E, int aperture,
                                            PathList& l) {
    const int lane = threadIdx.x & 31;
    int x = E + 1, y = 0;
    if (lane < count) {
        // no reflection at the stop or the last element, nor a second one outside the way back
        const int2 q = __ldg(paths + first + lane);
        const bool reflects = q.x >= 0 && q.x < E - 1 && q.x != aperture;
        x = reflects ? q.x : E;
        y = reflects && q.y >= 0 && q.y < q.x && q.y != aperture ? q.y : -1;
    }
    int rank = 0, next = 0, next_x = 0;
#pragma unroll
    for (int k = 0; k < kMaxPaths; k++) {
        const int ox = __shfl_sync(0xffffffffu, x, k), oy = __shfl_sync(0xffffffffu, y, k);
        rank += ox < x || (ox == x && (oy > y || (oy == y && k < lane)));
        next += k < count && (ox < x || (ox == x && oy >= y));
        next_x += k < count && ox <= x;
    }
    if (lane < count) {
        l.x[rank] = x;
        l.y[rank] = y;
        l.id[rank] = first + lane;
        l.next[rank] = next;
        l.next_x[rank] = next_x;
    }
}
// Walks the paths of l. The walk is the warp's; a lane whose ray has failed waits. Ray: State (the ray),
// hit(element, state) (intersects and moves the ray there; false: missed), refract(element, state)
// (false: the ray ends), reflect(element, state), store(path, state, whether it reached the end).
template <class Ray>
__device__ __forceinline__ void trace_paths(Ray& ray, typename Ray::State s, bool alive, const PathList& l, int count,
                                            int E, int aperture) {
    typename Ray::State kept[2];  // rays that go on past a reflection, per leg
    bool kept_alive[2];
    int i = 0, leg = 0, at = 0, step = 1, turn = l.x[0], last_x = 0, last_y = 0;
    for (;;) {
        if (alive) alive = ray.hit(at, s);
        if (at == turn) {  // (never the stop or the last element)
            if (leg == 0 ? l.next_x[i] < count : l.next[i] < l.next_x[i]) {  // paths after this one go on
                typename Ray::State c = s;
                kept_alive[leg] = alive && ray.refract(at, c);
                kept[leg] = c;
            }
            if (alive) ray.reflect(at, s);
            step = -step;
            if (leg++ == 0) last_x = at, turn = l.y[i];
            else last_y = at, turn = -1;
        } else if (at != aperture && at != E - 1) {
            if (alive) alive = ray.refract(at, s);
        }
        at += step;
        while ((unsigned)at >= (unsigned)E || !__any_sync(0xffffffffu, alive)) {
            // the ray is the last for these paths (those it would have turned at, where it failed)
            const int end = leg == 2 ? l.next[i] : (leg == 1 ? l.next_x[i] : count);
            const int group = l.next_x[i];
            for (; i < end; i++) ray.store(l.id[i], s, alive);
            if (end == count) return;
            leg = leg == 2 && end < group ? 1 : 0;
            s = kept[leg];
            alive = kept_alive[leg];
            step = leg == 0 ? 1 : -1;
            at = (leg == 0 ? last_x : last_y) + step;
            turn = leg == 0 ? l.x[i] : l.y[i];
        }
    }
}
// A ray in FP32.
template <bool kAngles>
struct FloatRay {
    struct State {
        float px, py, pz, dx, dy, dz, apt_x, apt_y, rrel, rrel2, refl;  // rrel2: see trace_ray_rec
    };
    const SmemElement* se;
    const float* ior_row;     // this wavelength's row of the (wavelength, element) index table, or nullptr
    const float2* ratio_row;  // and of the index ratios
    bool disperse;
    const float* coef_base;
    float wavelength;
    TraceFrame f;
    float* out;  // rays + the ray's place in a path
    long long per_path, plane;
    bool mine;  // the lane has a ray
    Hit h;

    __device__ __forceinline__ float ior_of(int el) const {
        if (ior_row) return ior_row[el];
        float n = se[el].ior;
        if (disperse && n > 1.0f) n = dispersion(wavelength, coef_base + (size_t)el * 16);
        return n;
    }
    // init_ray, raytracing.cl:178-215
    __device__ __forceinline__ State start(float grid_x, float grid_y) const {
        const Hit h0 = intersect(grid_x, -grid_y, 1.0f, 0.0f, 0.0f, -1.0f, se[0]);
        State s;  // the origin when the grid point misses element 0
        s.dx = f.dir[0], s.dy = f.dir[1], s.dz = f.dir[2];
        s.px = h0.px - s.dx, s.py = h0.py - s.dy, s.pz = h0.pz - s.dz;
        s.apt_x = s.apt_y = s.rrel = s.rrel2 = 0.0f;
        s.refl = 1.0f;
        return s;
    }
    __device__ __forceinline__ bool hit(int at, State& s) {
        const SmemElement& e = se[at];
        h = intersect(s.px, s.py, s.pz, s.dx, s.dy, s.dz, e);
        if (!h.hit) return false;
        s.px = h.px, s.py = h.py, s.pz = h.pz;
        if (at == f.aperture) {
            s.apt_x = h.px / e.height;
            s.apt_y = h.py / e.height;
        } else {
            const float xy2 = h.px * h.px + h.py * h.py;
            if (!(xy2 < s.rrel2 * (e.height * e.height))) {
                s.rrel = fmaxf(s.rrel, sqrtf(xy2) / e.height);
                s.rrel2 = s.rrel * s.rrel * (1.0f - 0x1p-20f);
            }
        }
        return true;
    }
    __device__ __forceinline__ bool refract(int at, State& s) {
        float o;
        if (ratio_row) {
            const float2 q = ratio_row[at];
            o = s.dz < 0.0f ? q.x : q.y;
        } else {
            const int n_index = (s.dz < 0.0f) ? at - 1 : at + 1;
            o = ((0 <= n_index && n_index < f.E) ? ior_of(n_index) : 1.0f) / ior_of(at);
        }
        refract_dir(s.dx, s.dy, s.dz, h, o);
        return s.dz != 0.0f;
    }
    __device__ __forceinline__ void reflect(int at, State& s) {
        const int n_index = (s.dz < 0.0f) ? at - 1 : at + 1;
        const float n1 = (0 <= n_index && n_index < f.E) ? ior_of(n_index) : 1.0f;
        const float reflectance =
            surface_reflectance<kAngles>(s.dx, s.dy, s.dz, h, se[at], n1, ior_of(at), wavelength, f);
        reflect_dir(s.dx, s.dy, s.dz, h);
        if (reflectance > 0.0f) s.refl *= reflectance;
    }
    __device__ __forceinline__ void store(int path, const State& s, bool alive) const {
        if (!mine) return;
        float* q = out + path * per_path;
        q[0] = s.px;
        q[plane] = s.py;
        q[2 * plane] = s.apt_x;
        q[3 * plane] = s.apt_y;
        q[4 * plane] = s.rrel;
        q[5 * plane] = alive ? s.refl : __int_as_float(0x7fffffff);
    }
};

// Wavelength rows that kTraceThreads * rays consecutive rays can span, and the shared memory of
// their tables (12 bytes per row and element); none past kMaxTableBytes.
constexpr int kMaxTableBytes = 40 * 1024;
__host__ __device__ inline int table_rows(long long rays, int R, int W) {
    const long long rows = (rays + R - 2) / R + 1;
    return (int)(rows < W ? rows : W);
}
inline size_t table_bytes(long long rays, int R, int W, int E) {
    const size_t bytes = sizeof(IorEntry) * (size_t)table_rows(rays, R, W) * E;
    return bytes <= kMaxTableBytes ? bytes : 0;
}

// Stage the lens elements and the refractive indices and ratios of wavelength rows [row0, row0 +
// span) (row r = wavelength (row0 + r) % W) in shared memory; table false: too many rows. ior is
// [span][E], ratio [span][E] after it.
__device__ __forceinline__ void stage_lens(const rf_lens_element* __restrict__ elements, const float* __restrict__ wavelengths,
                                           int E, int W, long long row0, int span, bool table, bool disperse,
                                           SmemElement* se, float2* ratio, float* ior) {
    for (int i = threadIdx.x; i < E; i += kTraceThreads) {
        const rf_lens_element& e = elements[i];
        se[i].radius = e.radius;
        se[i].center = e.center;
        se[i].height = e.height;
        se[i].ior = e.ior;
        se[i].coating = e.coating;
        se[i].layers = e.coating_layers;
        se[i].d0 = e.coating_thickness[0];
        se[i].d1 = e.coating_thickness[1];
    }
    if (table) {
        for (int k = threadIdx.x; k < span * E; k += kTraceThreads) {
            int row = k / E, el = k % E;
            int wl = (int)((row0 + row) % W);
            float n = elements[el].ior;
            if (disperse && n > 1.0f) n = dispersion(wavelengths[wl], elements[el].coefficients);
            ior[row * E + el] = n;
        }
        __syncthreads();
        for (int k = threadIdx.x; k < span * E; k += kTraceThreads) {
            const int row = k / E, el = k % E;
            const IorEntry r = ior_entry(el, E, [&](int i) { return ior[row * E + i]; });
            ratio[k] = make_float2(r.down, r.up);
        }
    }
}

// Kernel parameters of a trace (host): counts, coating constants, the light direction
// normalize(direction.xyz * -1) in FP32 without fused multiply-adds (the host code is
// compiled with -ffp-contract=off: the value the oracle computes) and the grid
// coordinates grid_length * (i / (G - 1) - 0.5), evaluated in double as the reference does.
inline bool trace_params(const rf_trace_args& a, TraceParams& p) {
    if (a.grid_count < 2 || a.grid_count > kMaxGrid) return false;
    p.R = a.grid_count * a.grid_count;
    p.n_rays = (long long)a.path_count * a.wavelength_count * p.R;
    p.E = a.element_count;
    p.aperture = a.aperture_index;
    p.P = a.path_count;
    p.W = a.wavelength_count;
    p.G = a.grid_count;
    p.cmin = a.coating_min_ior;
    p.layer_n0 = a.coating_layer_ior[0];
    p.layer_n1 = a.coating_layer_ior[1];
    float vx = -a.direction[0], vy = -a.direction[1], vz = -a.direction[2];
    float dd = vx * vx + vy * vy + vz * vz;
    float inv = 1.0f / sqrtf(dd);
    p.dir[0] = vx * inv;
    p.dir[1] = vy * inv;
    p.dir[2] = vz * inv;
    for (int i = 0; i < a.grid_count; i++) {
        float f = (float)i / (float)(a.grid_count - 1);
        p.grid[i] = (float)((double)a.grid_length * ((double)f - 0.5));
    }
    return true;
}

}  // namespace
}  // namespace rf
