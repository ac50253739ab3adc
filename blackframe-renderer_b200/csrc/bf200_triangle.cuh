// Ray / triangle test of the walks: exact edge signs, correctly rounded parameter and barycentrics, and the
// single-precision rule that spares certain misses the double test.
#pragma once

#include "bf200_geometry.cuh"

namespace bf200 {

constexpr double kU = 1.1102230246251565e-16;  // 2^-53

struct Dets {
    double p[3][3];
    double d[3];
};

// Exact evaluation of the four determinants as double expansions and an exact decision.
// Returns kTriHit with t (and barycentrics if requested), kTriMiss, or kTriFailure when a
// coordinate difference is not exact in double (exponent gap above 29 bits).
__device__ __forceinline__ int slow_triangle_decision(float4 v0, float4 v1, float4 v2, F3 o, F3 d, float t_min,
                                                      float t_max, float approx_t, bool want_bary, TriangleHit& hit) {
    Dets q;
    const double ox = o.x, oy = o.y, oz = o.z;
    q.p[0][0] = double(v0.x) - ox; q.p[0][1] = double(v0.y) - oy; q.p[0][2] = double(v0.z) - oz;
    q.p[1][0] = double(v1.x) - ox; q.p[1][1] = double(v1.y) - oy; q.p[1][2] = double(v1.z) - oz;
    q.p[2][0] = double(v2.x) - ox; q.p[2][1] = double(v2.y) - oy; q.p[2][2] = double(v2.z) - oz;
    q.d[0] = d.x; q.d[1] = d.y; q.d[2] = d.z;
    Expansion<double, 32> e0, e1, e2, vol;
    if (!exp_det3(e0, q.p[1], q.p[2], q.d) || !exp_det3(e1, q.p[2], q.p[0], q.d) ||
        !exp_det3(e2, q.p[0], q.p[1], q.d) || !exp_det3(vol, q.p[0], q.p[1], q.p[2])) {
        return kTriFailure;
    }
    Expansion<double, 96> det;
    det.size = 0;
    if (!exp_add_expansion(det, e0, 1.0) || !exp_add_expansion(det, e1, 1.0) || !exp_add_expansion(det, e2, 1.0)) {
        return kTriFailure;
    }
    const int ds = exp_sign(det);
    if (ds == 0) {
        return kTriMiss;  // coplanar or parallel: the accel skips both
    }
    const int s0 = exp_sign(e0), s1 = exp_sign(e1), s2 = exp_sign(e2);
    const bool nonneg = s0 >= 0 && s1 >= 0 && s2 >= 0;
    const bool nonpos = s0 <= 0 && s1 <= 0 && s2 <= 0;
    if (!nonneg && !nonpos) {
        return kTriMiss;
    }
    double dv = 0.0, vv = 0.0;
    for (int i = 0; i < det.size; ++i) dv += det.c[i];
    for (int i = 0; i < vol.size; ++i) vv += vol.c[i];
    float seed = isfinite(approx_t) && approx_t != 0.0F ? approx_t : static_cast<float>(vv / dv);
    float t = 0.0F;
    if (exp_sign(vol) == 0) {
        t = 0.0F;
    } else {
        if (seed == 0.0F || !isfinite(seed)) {
            return kTriFailure;
        }
        if (!exact_round_quotient(vol, det, seed, t)) {
            return kTriFailure;
        }
    }
    if (isnan(t) || t < t_min || t > t_max) {
        return kTriMiss;
    }
    hit.t = t;
    if (want_bary) {
        const Expansion<double, 32>* es[3] = {&e0, &e1, &e2};
        float out[3];
        for (int k = 0; k < 3; ++k) {
            if (exp_sign(*es[k]) == 0) {
                out[k] = 0.0F;
                continue;
            }
            double ev = 0.0;
            for (int i = 0; i < es[k]->size; ++i) ev += es[k]->c[i];
            if (!exact_round_quotient(*es[k], det, static_cast<float>(ev / dv), out[k])) {
                return kTriFailure;
            }
        }
        hit.b0 = out[0];
        hit.b1 = out[1];
        hit.b2 = out[2];
    }
    return kTriHit;
}

// The out-of-line copy of the exact test. It takes the vertices and the ray by value, rebuilds the
// differences itself and returns its result by value, so the fast path that calls it keeps
// everything in registers.
struct SlowResult {
    int code;
    TriangleHit hit;
};

static __device__ __noinline__ SlowResult exact_triangle_slow(float4 v0, float4 v1, float4 v2, F3 o, F3 d, float t_min,
                                                       float t_max, float approx_t, bool want_bary) {
    SlowResult r;
    r.code = slow_triangle_decision(v0, v1, v2, o, d, t_min, t_max, approx_t, want_bary, r.hit);
    return r;
}

__device__ __forceinline__ int slow_path(float4 v0, float4 v1, float4 v2, F3 o, F3 d, float t_min, float t_max,
                                         float approx_t, bool want_bary, TriangleHit& hit) {
    const SlowResult r = exact_triangle_slow(v0, v1, v2, o, d, t_min, t_max, approx_t, want_bary);
    if (r.code == kTriHit) {
        hit = r.hit;
    }
    return r.code;
}

// The float nearest to num/den when a forward error bound proves it; otherwise NaN. Bounds below 2^-46
// of their values, the usual case, leave the quotient within 2^-44 of its own size: one division
// decides, and an interval that rounds to one float holds the same float as the narrower one of the
// general case.
static __device__ __noinline__ float certain_round_general(double num, double num_bound, double den, double den_bound);
__device__ __forceinline__ float certain_round(double num, double num_bound, double den, double den_bound) {
    if (num_bound <= fabs(num) * 0x1p-46 && den_bound <= fabs(den) * 0x1p-46) {
        const double q = num / den;
        const double slack = fabs(q) * 0x1p-44;
        const float lo = __double2float_rn(q - slack), hi = __double2float_rn(q + slack);
        if (lo == hi && q != 0.0) {
            return lo;
        }
    }
    return certain_round_general(num, num_bound, den, den_bound);
}
static __device__ __noinline__ float certain_round_general(double num, double num_bound, double den, double den_bound) {
    if (!(fabs(num) > 2.0 * num_bound) || !(fabs(den) > 2.0 * den_bound)) {
        return __int_as_float(0x7fc00000);
    }
    const double q = num / den;
    const double rel = num_bound / fabs(num) + den_bound / fabs(den) + 4.0 * kU;
    if (!(rel < 0x1p-27)) {
        return __int_as_float(0x7fc00000);
    }
    const double lo = q - fabs(q) * (2.0 * rel);
    const double hi = q + fabs(q) * (2.0 * rel);
    const float flo = __double2float_rn(lo);
    const float fhi = __double2float_rn(hi);
    return flo == fhi ? flo : __int_as_float(0x7fc00000);
}

// Returns kTriHit (t set), kTriMiss or kTriFailure. Object-space floats in; the decision and
// the parameter equal those of the exact test in Triangle.hpp:683-822.
// d . (p x f) and a bound on its evaluation error: edge differences, products and the two
// subtractions / additions round at most seven times along any term, so the error is below
// 8u * sum |d_i| (|p_j f_k| + |p_k f_j|); 16u of that sum is returned as the bound.
__device__ __forceinline__ double edge_function(const double (&p)[3], double fx, double fy, double fz,
                                                const double (&dd)[3], double& bound) {
    const double cx = p[1] * fz - p[2] * fy, cy = p[2] * fx - p[0] * fz, cz = p[0] * fy - p[1] * fx;
    const double bx = fabs(p[1] * fz) + fabs(p[2] * fy), by = fabs(p[2] * fx) + fabs(p[0] * fz),
                 bz = fabs(p[0] * fy) + fabs(p[1] * fx);
    bound = 16.0 * kU * ((fabs(dd[0]) * bx + fabs(dd[1]) * by) + fabs(dd[2]) * bz);
    return (dd[0] * cx + dd[1] * cy) + dd[2] * cz;
}

__device__ __forceinline__ int triangle_test(float4 v0, float4 v1, float4 v2, F3 o, F3 d, float t_min, float t_max,
                                             bool want_bary, TriangleHit& hit) {
    const double ox = o.x, oy = o.y, oz = o.z;
    const double p0[3] = {double(v0.x) - ox, double(v0.y) - oy, double(v0.z) - oz};
    const double p1[3] = {double(v1.x) - ox, double(v1.y) - oy, double(v1.z) - oz};
    const double p2[3] = {double(v2.x) - ox, double(v2.y) - oy, double(v2.z) - oz};
    const double dd[3] = {d.x, d.y, d.z};
    // Edge functions e0 = det(p1, p2, d), e1 = det(p2, p0, d), e2 = det(p0, p1, d), evaluated as
    // e0 = d . (p1 x (v2 - v1)), e1 = d . (p2 x (v0 - v2)), e2 = d . (p0 x (v1 - v0)): the same
    // exact values (p_j = p_i + v_j - v_i), with terms of the size (distance x edge) instead of
    // distance squared, so their error bounds stay small for small distant triangles.
    double e[3], bound[3];
    e[0] = edge_function(p1, double(v2.x) - double(v1.x), double(v2.y) - double(v1.y),
                         double(v2.z) - double(v1.z), dd, bound[0]);
    e[1] = edge_function(p2, double(v0.x) - double(v2.x), double(v0.y) - double(v2.y),
                         double(v0.z) - double(v2.z), dd, bound[1]);
    e[2] = edge_function(p0, double(v1.x) - double(v0.x), double(v1.y) - double(v0.y),
                         double(v1.z) - double(v0.z), dd, bound[2]);
    int pos = 0, neg = 0;
    bool ambiguous = false;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (e[k] > bound[k]) {
            ++pos;
        } else if (e[k] < -bound[k]) {
            ++neg;
        } else {
            ambiguous = true;
        }
    }
    if (pos > 0 && neg > 0) {
        return kTriMiss;
    }
    // A coordinate difference that is not exact in double makes the slow path unusable; such
    // inputs (exponent gaps above 29 bits) are reported as a lane failure.
    const auto exact_diffs = [&]() {
        return (p0[0] + ox == double(v0.x)) && (p0[1] + oy == double(v0.y)) && (p0[2] + oz == double(v0.z)) &&
               (p1[0] + ox == double(v1.x)) && (p1[1] + oy == double(v1.y)) && (p1[2] + oz == double(v1.z)) &&
               (p2[0] + ox == double(v2.x)) && (p2[1] + oy == double(v2.y)) && (p2[2] + oz == double(v2.z));
    };
    if (ambiguous) {
        if (!exact_diffs()) {
            return kTriFailure;
        }
        return slow_path(v0, v1, v2, o, d, t_min, t_max, __int_as_float(0x7fc00000), want_bary, hit);
    }
    // vol = det(p0, p1, p2) and det = e0 + e1 + e2 have the exact values p0 . N and d . N with
    // N = (v1 - v0) x (v2 - v0) (the scalar triple product identities). Evaluated in that form
    // their rounding error scales with the triangle's own size instead of its distance from the ray
    // origin, so small distant triangles certify their parameter without the exact fallback; the
    // quotient certified is still the exact one, so t is unchanged. Error bound: each edge
    // difference and product rounds once (u), each cross component and three-term dot product
    // rounds twice and three times more, at most 8u of the magnitudes summed below; 16u is used.
    const double e1x = double(v1.x) - double(v0.x), e1y = double(v1.y) - double(v0.y),
                 e1z = double(v1.z) - double(v0.z);
    const double e2x = double(v2.x) - double(v0.x), e2y = double(v2.y) - double(v0.y),
                 e2z = double(v2.z) - double(v0.z);
    const double nx = e1y * e2z - e1z * e2y, ny = e1z * e2x - e1x * e2z, nz = e1x * e2y - e1y * e2x;
    const double ax = fabs(e1y * e2z) + fabs(e1z * e2y), ay = fabs(e1z * e2x) + fabs(e1x * e2z),
                 az = fabs(e1x * e2y) + fabs(e1y * e2x);
    const double vol = (p0[0] * nx + p0[1] * ny) + p0[2] * nz;
    const double vol_bound = 16.0 * kU * ((fabs(p0[0]) * ax + fabs(p0[1]) * ay) + fabs(p0[2]) * az);
    const double det = (dd[0] * nx + dd[1] * ny) + dd[2] * nz;
    const double det_bound = 16.0 * kU * ((fabs(dd[0]) * ax + fabs(dd[1]) * ay) + fabs(dd[2]) * az);
    float t = certain_round(vol, vol_bound, det, det_bound);
    if (isnan(t)) {
        if (!exact_diffs()) {
            return kTriFailure;
        }
        return slow_path(v0, v1, v2, o, d, t_min, t_max, __double2float_rn(vol / det), want_bary, hit);
    }
    if (t < t_min || t > t_max) {
        return kTriMiss;
    }
    hit.t = t;
    if (want_bary) {
        // The edge functions do not change when multiples of d are taken from the vertices. Moved by
        // the hit's t d (exact vertex differences, then one rounding of the small result), the vertices
        // lie within the triangle's size of the origin instead of the ray's length away, and the error
        // bounds shrink with them (nine roundings along a term instead of eight, still below the 16u
        // returned): from the far origin, weights of small distant triangles below about 2^-11 could not be
        // certified, and their exact evaluations kept k_hits waiting (BVH-stress frame, 16 samples: trace and hits 89.7 ->
        // 79.5 ms; Cornell box with spheres, 256 spp: 30.8 -> 29.1 ms).
        const auto exact_back = [&](double p, double o, float v) { return double(v) - p == o; };
        const bool exact = exact_diffs() && exact_back(p0[0], ox, v0.x) && exact_back(p0[1], oy, v0.y) &&
                           exact_back(p0[2], oz, v0.z) && exact_back(p1[0], ox, v1.x) && exact_back(p1[1], oy, v1.y) &&
                           exact_back(p1[2], oz, v1.z) && exact_back(p2[0], ox, v2.x) && exact_back(p2[1], oy, v2.y) &&
                           exact_back(p2[2], oz, v2.z);
        if (exact) {
            const double along = t;
            const double q0[3] = {fma(-along, dd[0], p0[0]), fma(-along, dd[1], p0[1]), fma(-along, dd[2], p0[2])};
            const double q1[3] = {fma(-along, dd[0], p1[0]), fma(-along, dd[1], p1[1]), fma(-along, dd[2], p1[2])};
            const double q2[3] = {fma(-along, dd[0], p2[0]), fma(-along, dd[1], p2[1]), fma(-along, dd[2], p2[2])};
            e[0] = edge_function(q1, double(v2.x) - double(v1.x), double(v2.y) - double(v1.y),
                                 double(v2.z) - double(v1.z), dd, bound[0]);
            e[1] = edge_function(q2, -e2x, -e2y, -e2z, dd, bound[1]);
            e[2] = edge_function(q0, e1x, e1y, e1z, dd, bound[2]);
        }
        const float b0 = certain_round(e[0], bound[0], det, det_bound);
        const float b1 = certain_round(e[1], bound[1], det, det_bound);
        const float b2 = certain_round(e[2], bound[2], det, det_bound);
        if (isnan(b0) || isnan(b1) || isnan(b2)) {
            if (!exact_diffs()) {
                return kTriFailure;
            }
            return slow_path(v0, v1, v2, o, d, t_min, t_max, t, true, hit);
        }
        hit.b0 = b0;
        hit.b1 = b1;
        hit.b2 = b2;
    }
    return kTriHit;
}

// Whether two edge functions certainly have opposite signs by single precision, so that the ray misses
// the triangle (what triangle_test, in double, finds first). Vertex and edge differences, products and
// sums round at most seven times along any term of e = d . (p x f), and the terms sum to at most
// 2 |d|_1 |p|_max |f|_max, so the error is below 14.1 u |d|_1 |p|_max |f|_max; 20u is asked for. Values in
// the reach of subnormal products decide nothing, nor does anything that can overflow: 4 |p|_max |f|_max
// and its product with |d|_1 bound every intermediate and are infinite first.
__device__ __forceinline__ bool certain_miss(float4 v0, float4 v1, float4 v2, F3 o, F3 d, float d_sum) {
    const F3 p0{v0.x - o.x, v0.y - o.y, v0.z - o.z}, p1{v1.x - o.x, v1.y - o.y, v1.z - o.z},
        p2{v2.x - o.x, v2.y - o.y, v2.z - o.z};
    const F3 f0{v2.x - v1.x, v2.y - v1.y, v2.z - v1.z}, f1{v0.x - v2.x, v0.y - v2.y, v0.z - v2.z},
        f2{v1.x - v0.x, v1.y - v0.y, v1.z - v0.z};
    const auto largest = [](F3 a, F3 b, F3 c) {
        return fmaxf(fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(b.x))),
                           fmaxf(fmaxf(fabsf(b.y), fabsf(b.z)), fmaxf(fabsf(c.x), fabsf(c.y)))),
                     fabsf(c.z));
    };
    const auto edge = [&](F3 p, F3 f) {
        const F3 c{fmaf(p.y, f.z, -(p.z * f.y)), fmaf(p.z, f.x, -(p.x * f.z)), fmaf(p.x, f.y, -(p.y * f.x))};
        return fmaf(d.x, c.x, fmaf(d.y, c.y, d.z * c.z));
    };
    const float bound = fmaxf(4.0F * largest(p0, p1, p2) * largest(f0, f1, f2) * d_sum * (5.0F * 5.9604645e-8F),
                              1e-30F * (1.0F + d_sum));
    const float e0 = edge(p1, f0), e1 = edge(p2, f1), e2 = edge(p0, f2);
    return (e0 > bound || e1 > bound || e2 > bound) && (e0 < -bound || e1 < -bound || e2 < -bound);
}

}  // namespace bf200
