// ht_bound.cuh -- distance bounds of the hyperbolic object scans: world-space records of
// geodesic planes and horospheres and the culling tests on them. Shared by the hand-written
// scene kernels (ht_trace.cuh) and the generic template kernels (ht_generic.cuh, also
// compiled at run time by NVRTC). They decide only which objects are tested exactly, never a
// result: tests/cull_check/scan_check.c restates them on the CPU and checks every hop's
// winner against the full scan of the reference.
#pragma once
#include "ht_math.cuh"

namespace ht {

// ---------------------------------------------------------------- distance bounds
// The object scan only needs the exact (reference) test for objects that can be hit nearer
// than the best hit found so far. Whether and where the geodesic ray from (p, v) meets an
// object has a closed form in world space, evaluated here with explicit error terms and wide
// margins; objects it rules out are not tested. This changes which objects are evaluated,
// never the result. Per object one float4 `rec`, staged once per launch (stage_bound):
//   geodesic plane  rec = (A, 2Re B, 2Im B, C): the world plane's normalised Hermitian form,
//                   |B|^2 - A C = 1. F = rec . (|p|^2, x, y, 1) = Q and sinh(signed distance
//                   to the plane) = Q / (2t); along the unit-speed geodesic it is exactly
//                   a cosh s + b sinh s with a = F / 2t, b = W / 2t, so the ray meets the plane
//                   at s* = atanh(-a/b) when 0 <= -a/b < 1.
//   horosphere      rec = (|n21|^2, 2 Re w, -2 Im w, |n22|^2), w = conj(n22) n21, N = M^-1
//                   normalised to det 1: F = rec . (|p|^2, x, y, 1) = t / t' (t' = local
//                   height; inside the horoball when t' > 1). Along the geodesic
//                   1/t' = P cosh s + V sinh s with P = F / t, V = W / t; it crosses 1 at
//                   e^s = (P - V) / (1 + r) (entry) and (1 + r) / (P + V) (exit), r^2 = 1 - P^2 + V^2.
//   both            W = t (2 rec.x (p.v) + rec.y v.x + rec.z v.y) - F v.z
// with p = (x, y, t) the ray start, v its unit direction (v.z along the height).
// The threshold is thr = best (1 + CULL_REL) + CULL_ABS; objects with large map entries get
// NaN records (never culled) and ray starts outside a well-conditioned box disable culling.
//
// Margins. The reference computes the local ray and the hit in f32, so what it reports differs
// from the exact geometry; a test may cull only with more room than that. With eps = 2^-24,
// N^2 the largest squared entry of the map (det 1) and G = 2 N^2 K0 / t >= 1 / t' (K0 = |p|^2 + |x| +
// |y| + 1, t' the local height of the ray start):
//   - the local start is off by about 10 eps N^2 K0 / t in the hyperbolic metric, a plane's
//     |p'|^2 - 1 by 3 eps G in units of sinh(distance), and its hit point's height, sqrt(1 - |xy|^2),
//     moves the hit by eps (3 G / |p'.d'| + G^2);
//   - cosh(distance) is rounded to a multiple of 2 eps, which moves a distance d by 2 eps / d;
//   - a root is reported from -EPS on: sinh(distance) up to 1e-6 G on the wrong side of a plane.
// The additive allowance eF = mag K (K = K0^2 / t >= 2 K0) grows as these do: mag is
// BOUND_EPS / 2 max(N^2, |rec|), plus PLANE_EPS N^4 for planes, which in sinh(distance) is at least
// 2.5e-6 G + 2.4e-7 G^2, ten times the first item's linear and four times its quadratic part. On
// top of it CULL_ABS = 2e-3 covers the rounding of distances (at most 4e-4 near d = 0) and
// CULL_REL the hits far from the start, whose local height is e^-d of it; PLANE_M = 1e-3 t (5e-4
// of sinh(distance)) keeps the signs of a plane's test apart. Fixed margins in place of the
// allowance's quadratic part have to be sized for the worst map and let a hop test 20 % more
// objects. tests/cull_check/scan_check.c runs all of this against the full scan on the CPU.
constexpr float CULL_REL = 1e-2f, CULL_ABS = 2e-3f;

constexpr float BOUND_EPS = 1e-5f;   // relative error allowance of F and W (>> f32 rounding)
constexpr float PLANE_EPS = 2e-6f;   // allowance of a plane's hit point, per N^4
constexpr float PLANE_M = 1e-3f;     // additive margin of the plane tests, in units of t
constexpr float HORO_M = 1e-3f;      // relative margin of the horosphere root bounds

// Hardware approximations (PTX rcp / sqrt / lg2 / ex2 .approx, relative error near 2^-22) for
// the bound arithmetic only: every quantity they produce carries a margin of at least 1e-6
// relative (the threshold itself 1e-2), so they never decide a culling the exact values
// would not allow. The path's own arithmetic (ray maps, shape tests) never uses them.
HT_D float rcp_approx(float x) { float r; asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
HT_D float sqrt_approx(float x) { float r; asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
HT_D float lg2_approx(float x) { float r; asm("lg2.approx.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
HT_D float ex2_approx(float x) { float r; asm("ex2.approx.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
constexpr float LN2F = 0.693147180559945f, LOG2EF = 1.442695040888963f;

struct Cull { float S, E, T; };   // sinh, exp, tanh of the threshold; S = E = inf, T = 1: none

// World-space bound record of one object from its f32 map M, in FP64 (once per launch), and the
// magnitude `mag` of its error allowance.
// N = adj(M) maps world to local (c22_inverse_n, matrix_complex.cc:60-65).
HT_D float bound_mag(float4 rec, double n2, uint32_t shape) {
    const double m = fmax(n2, (double)fmaxf(fmaxf(fabsf(rec.x), fabsf(rec.y)), fmaxf(fabsf(rec.z), fabsf(rec.w))));
    return (float)(0.5 * BOUND_EPS * m + (shape == 0 ? PLANE_EPS * m * m : 0.0));
}
HT_D float4 stage_bound(const Mo &m, uint32_t shape, float &mag) {
    const double ar = m.a.x, ai = m.a.y, br = m.b.x, bi = m.b.y;
    const double cr = m.c.x, ci = m.c.y, dr = m.d.x, di = m.d.y;
    const double det_r = (ar * dr - ai * di) - (br * cr - bi * ci);
    const double det_i = (ar * di + ai * dr) - (br * ci + bi * cr);
    const double adet = sqrt(det_r * det_r + det_i * det_i);
    const double maxe = fmax(fmax(fabs(ar) + fabs(ai), fabs(br) + fabs(bi)), fmax(fabs(cr) + fabs(ci), fabs(dr) + fabs(di)));
    const float nan = __int_as_float(0x7fc00000);
    mag = 0.0f;
    if (!(maxe <= 32.0 && adet >= 0.5 && adet <= 2.0)) return make_float4(nan, nan, nan, nan);
    const double n2 = fmax(fmax(ar * ar + ai * ai, br * br + bi * bi), fmax(cr * cr + ci * ci, dr * dr + di * di)) / adet;
    // N = [[n11, n12], [n21, n22]] = [[d, -b], [-c, a]]
    const double n11r = dr, n11i = di, n12r = -br, n12i = -bi, n21r = -cr, n21i = -ci, n22r = ar, n22i = ai;
    if (shape == 0) {
        const double A = (n11r * n11r + n11i * n11i) - (n21r * n21r + n21i * n21i);
        // B = conj(n11) n12 - conj(n21) n22
        const double Br = (n11r * n12r + n11i * n12i) - (n21r * n22r + n21i * n22i);
        const double Bi = (n11r * n12i - n11i * n12r) - (n21r * n22i - n21i * n22r);
        const double C = (n12r * n12r + n12i * n12i) - (n22r * n22r + n22i * n22i);
        const float4 rec = make_float4((float)(A / adet), (float)(2.0 * Br / adet), (float)(2.0 * Bi / adet), (float)(C / adet));
        mag = bound_mag(rec, n2, shape);
        return rec;
    }
    // horosphere: scale N by 1 / sqrt|det| so the height formula holds
    const double k2 = 1.0 / adet;
    const double c2 = (n21r * n21r + n21i * n21i) * k2;
    const double wr = (n22r * n21r + n22i * n21i) * k2;   // w = conj(n22) n21
    const double wi = (n22r * n21i - n22i * n21r) * k2;
    const double n22sq = (n22r * n22r + n22i * n22i) * k2;
    const float4 rec = make_float4((float)c2, (float)(2.0 * wr), (float)(-2.0 * wi), (float)n22sq);
    mag = bound_mag(rec, n2, shape);
    return rec;
}

// Per-hop constants of the bound evaluation.
struct BoundRay {
    float x, y, t, r2, pv, vx, vy, vz;
    float K;    // (|p|^2 + |x| + |y| + 1)^2 / t: eF = mag * K
    float Kw;   // t (2 |p.v| + |vx| + |vy|) (|p|^2 + |x| + |y| + 1) / t: the part of eW that scales with mag
};
HT_D bool cull_point_ok(Q4 p) {
    return p.z >= 0x1p-20f && p.z <= 0x1p20f && fabsf(p.x) + fabsf(p.y) <= 0x1p10f * p.z &&
           fabsf(p.w) <= 1e-3f * p.z;
}
HT_D BoundRay bound_ray(Q4 p, Q4 v) {
    BoundRay b;
    b.x = p.x; b.y = p.y; b.t = p.z;
    b.r2 = fmaf(p.x, p.x, fmaf(p.y, p.y, p.z * p.z));
    b.pv = fmaf(p.x, v.x, fmaf(p.y, v.y, p.z * v.z));
    b.vx = v.x; b.vy = v.y; b.vz = v.z;
    const float K0 = b.r2 + fabsf(p.x) + fabsf(p.y) + 1.0f;
    b.K = K0 * K0 * rcp_approx(b.t);
    b.Kw = K0 * (2.0f * fabsf(b.pv) + fabsf(b.vx) + fabsf(b.vy));
    return b;
}
// eF and eW of one object (the bounds of the float error of F and W)
HT_D float bound_eF(float mag, const BoundRay &r) { return mag * r.K; }
HT_D float bound_eW(float mag, float eF, float W, const BoundRay &r) {
    return fmaf(mag, r.Kw, fmaf(eF, fabsf(r.vz), BOUND_EPS * fabsf(W)));
}
// S, E, T are upper bounds of sinh, exp, tanh of the threshold: E from ex2.approx raised by
// 1e-5 relative (more than its error plus the rounding of thr * log2(e) for thr < 89, above
// which it is +inf), S and T increasing functions of it.
HT_D Cull cull_from_dist(float d) {
    const float thr = fmaf(d, 1.0f + CULL_REL, CULL_ABS);
    Cull c;
    c.E = ex2_approx(thr * LOG2EF) * (1.0f + 1e-5f);
    c.S = 0.5f * (c.E - rcp_approx(c.E));
    c.T = 1.0f - 2.0f * rcp_approx(fmaf(c.E, c.E, 1.0f));
    return c;
}
HT_D Cull cull_none() {
    Cull c;
    c.S = c.E = __int_as_float(0x7f800000);
    c.T = 1.0f;
    return c;
}
// Cheap bound: the distance from the ray start to the object alone (any hit lies on it),
// F = rec . (|p|^2, x, y, 1) with its error allowance eF:
//   geodesic plane  culled when |F| - eF > 2 t S (sinh of the distance to the plane);
//   horosphere      culled when t > E (F + eF) or t E < F - eF (the local height t' = t / F
//                   outside [e^-thr, e^thr] even with F's error).
// The point bound as thresholds on F: an object is culled when F + eF < lo or F - eF > hi. (In the packed
// form, two slots of one shape at once, the product mag K and its sum with F may be rounded once
// instead of twice, as ht_math.cuh says of packed sums: a last place of eF, which is 1e-5 of F and more.)
//   geodesic plane  lo = -2 t S, hi = 2 t S: |F| - eF > 2 t S (|F| - eF = -(F + eF) when F < 0);
//   horosphere      lo = t / E (E an upper bound of e^thr raised by 1e-5, so this stays below
//                   t e^-thr after its rounding and the rcp approximation), hi = t E: the
//                   test t > E (F + eF) or t E < F - eF with the division moved to the threshold.
// A NaN record (ill-conditioned map) is never culled.
struct PointCut { float2 lo, hi; };
HT_D PointCut point_cut(uint32_t shape, float t, const Cull &c) {
    PointCut k;
    if (shape == 0) {
        const float h = 2.0f * t * c.S;
        k.lo = make_float2(-h, -h);
        k.hi = make_float2(h, h);
    } else {
        const float l = t * rcp_approx(c.E), h = t * c.E;
        k.lo = make_float2(l, l);
        k.hi = make_float2(h, h);
    }
    return k;
}
// The same test on one object (the scalar form of the packed loop).
HT_D bool culled_point(float4 rec, float mag, const BoundRay &r, const PointCut &k) {
    const float F = fmaf(rec.x, r.r2, fmaf(rec.y, r.x, fmaf(rec.z, r.y, rec.w)));
    const float eF = mag * r.K;
    return F + eF < k.lo.x || F - eF > k.hi.x;
}
// F, W of one object along the ray and the bounds of their float error
struct BoundFW { float F, eF, W, eW; };
HT_D BoundFW bound_fw(float4 rec, float mag, const BoundRay &r) {
    BoundFW b;
    b.F = fmaf(rec.x, r.r2, fmaf(rec.y, r.x, fmaf(rec.z, r.y, rec.w)));
    b.eF = bound_eF(mag, r);
    const float G = fmaf(2.0f * rec.x, r.pv, fmaf(rec.y, r.vx, rec.z * r.vy));
    b.W = fmaf(r.t, G, -b.F * r.vz);
    b.eW = bound_eW(mag, b.eF, b.W, r);
    return b;
}
// The ray-aware test of one object that the point bound kept.
HT_D bool culled_ray(const BoundFW &b, uint32_t shape, float t, const Cull &c) {
    const float F = b.F, eF = b.eF, W = b.W, eW = b.eW;
    if (shape == 0) {
        const float Fa = fabsf(F) - eF;       // lower bound of |2 t a|
        const float Wlo = fabsf(W) - eW, Whi = fabsf(W) + eW;
        // starts off the plane and moves away from it: |a| > 5e-4 and more, |b| > 0.001, same signs
        const bool away = (F > 0.0f) == (W > 0.0f) && Fa > fmaf(PLANE_M, t, eF) && Wlo > 0.002f * t;
        // |a| > 1.01 T |b| + 5e-4: no root (T = 1) or the root lies beyond the threshold
        const bool far = Fa > fmaf(1.01f * c.T, Whi, PLANE_M * t);
        return away || far;
    } else {
        // In the object's frame the reference's horosphere test (shape/hy/horosphere.cc:4-34)
        // looks at two roots; with P = F/t (1 / local height), V = W/t (its derivative along
        // the ray), r^2 = 1 - P^2 + V^2 their parameters are t1 = -(V + rP)/P^2 and
        // t2 = (rP - V)/P^2, and a root is reported only when its parameter is >= -EPS (it
        // accepts roots up to EPS behind the start, before dividing by |d.xy|^2). The roots
        // are the crossings at e^s = (P - V)/(1 + r) and (1 + r)/(P + V). The object is
        // culled when every root that can be reported lies farther than the threshold.
        const float Flo = F - eF, Fhi = F + eF, Wlo = W - eW, Whi = W + eW;
        const float aWlo = fmaxf(fabsf(W) - eW, 0.0f), aWhi = fabsf(W) + eW;
        if (!(Flo > 0.0f)) return false;
        const float R2lo = t * t - Fhi * Fhi + aWlo * aWlo, R2hi = t * t - Flo * Flo + aWhi * aWhi;
        if (R2hi < -HORO_M * t * t) return true;        // no crossing
        if (R2lo < HORO_M * t * t) return false;        // nearly tangent: test exactly
        const float Rlo = sqrt_approx(R2lo) * (1.0f - 1e-6f), Rhi = sqrt_approx(R2hi) * (1.0f + 1e-6f);   // r t
        // margin of the reference's own root test: 2 EPS plus its float error
        const float tol = 2e-6f * Fhi * Fhi + 1e-5f * (aWhi * t + Rhi * Fhi);
        const bool r1 = !(Wlo * t + Rlo * Flo > tol);   // root 1 may be reported
        const bool r2 = !(Wlo * t - Rhi * Fhi > tol);   // root 2 may be reported
        const float E1 = c.E * (1.0f + HORO_M);
        const bool r1_far = (Flo - Whi) > E1 * (t + Rhi) || (Fhi - Wlo) * E1 < (t + Rlo);
        const bool r2_far = (Flo + Wlo) > 0.0f && ((t + Rlo) > E1 * (Fhi + Whi) || (t + Rhi) * E1 < (Flo + Wlo));
        return (!r1 || r1_far) && (!r2 || r2_far);
    }
}

// Upper bound of e^(2 s) at the nearest crossing of one object that the reference surely
// reports (s = distance along the ray): geodesic planes crossed ahead (tanh s = |F| / |W|,
// not the plane the ray just left), horospheres entered ahead from outside or left ahead
// from inside (e^s of the crossing), with margins far above the float error of either side.
// +inf when the object has no such crossing.
HT_D float sure_crossing_e2(const BoundFW &b, uint32_t shape, bool plane_repeat, float t) {
    const float inf = __int_as_float(0x7f800000);
    const float F = b.F, eF = b.eF, W = b.W, eW = b.eW;
    if (shape == 0) {
        if (plane_repeat) return inf;   // a plane is never hit twice in a row
        const float Fa = fabsf(F) - eF, Wlo = fabsf(W) - eW;
        if (!((F > 0.0f) != (W > 0.0f) && Fa > fmaf(PLANE_M, t, eF) && Wlo > 0.02f * t)) return inf;
        const float rr = (fabsf(F) + eF) * rcp_approx(Wlo);   // >= tanh s
        if (!(rr < 0.99f)) return inf;
        return (1.0f + rr) * rcp_approx(1.0f - rr);
    }
    const float Flo = F - eF, Fhi = F + eF, Wlo = W - eW, Whi = W + eW;
    float e = inf;
    if (Fhi < 0.999f * t && Flo > 0.0f && (Flo + Wlo) > 0.0f) {   // inside: exit ahead
        const float aWlo = fmaxf(fabsf(W) - eW, 0.0f), aWhi = fabsf(W) + eW;
        const float R2lo = t * t - Fhi * Fhi + aWlo * aWlo, R2hi = t * t - Flo * Flo + aWhi * aWhi;
        if (R2lo > 1e-3f * t * t) {
            const float Rlo = sqrt_approx(R2lo) * (1.0f - 1e-6f), Rhi = sqrt_approx(R2hi) * (1.0f + 1e-6f);
            const float tol = 2e-6f * Fhi * Fhi + 1e-5f * (aWhi * t + Rhi * Fhi);
            const bool r1 = !(Wlo * t + Rlo * Flo > tol);
            const bool r2_sure = (Wlo * t - Rhi * Fhi) < -tol - 1e-3f * t * t;
            if (!r1 && r2_sure) e = (t + Rhi) * rcp_approx(Flo + Wlo) * 1.001f;
        }
    } else if (Flo > 1.01f * t && Whi < -0.01f * t) {   // outside, approaching: entry ahead
        const float it = rcp_approx(t);
        const float aVlo = -Whi * it, P = Fhi * it;
        const float D = 1.0f - P * P + aVlo * aVlo;
        if (D > 0.02f) e = (Fhi - Wlo) * it * rcp_approx(1.0f + sqrt_approx(D));
    }
    return e * e;
}
// Whether the scan has to test one object exactly, from the point bound `k` of its shape and the
// ray-aware test.
HT_D bool keep_object(float4 rec, float mag, uint32_t shape, const BoundRay &r, const PointCut &k, const Cull &c) {
    const BoundFW b = bound_fw(rec, mag, r);
    return !(b.F + b.eF < k.lo.x || b.F - b.eF > k.hi.x || culled_ray(b, shape, r.t, c));
}
// The threshold of a scan: the nearest hit found, or surely to be found, so far.
struct Limit {
    float d;        // that distance (+inf: none)
    Cull cull;
    PointCut kp, kh;
};
HT_D Limit limit_none(float t) {
    Limit l;
    l.d = __int_as_float(0x7f800000);
    l.cull = cull_none();
    l.kp = point_cut(0, t, l.cull);
    l.kh = point_cut(1, t, l.cull);
    return l;
}
HT_D void limit_lower(Limit &l, float d, float t) {
    if (!(d < l.d)) return;
    l.d = d;
    l.cull = cull_from_dist(d);
    l.kp = point_cut(0, t, l.cull);
    l.kh = point_cut(1, t, l.cull);
}
// Distance of a crossing from its e^(2 s) bound (the threshold built from it adds 1e-2 margins).
HT_D float dist_from_e2(float x) { return 0.5f * LN2F * lg2_approx(x); }

// Warp pre-cull (wavefront kernels, full warps whose lanes can all cull): each lane tests
// one slot of a 32-slot chunk against the whole warp at once — F over the box of the lanes'
// (|p|^2, x, y), the largest error allowance and the loosest thresholds of the warp — and a
// slot the warp test culls is culled by every lane's own point test, so the lanes run that
// test only on the pairs the warp keeps and reach the same candidate masks bit for bit. The
// warp test adds a slack of 2^-16 of the magnitudes involved, far above the rounding of
// either evaluation (a few units of 2^-24 each), so float rounding cannot break that
// implication. After the coherence sort a warp's rays start in one cell, the box is small,
// and most slots go in one test per warp instead of one per lane.
struct WarpBox { float r2lo, r2hi, xlo, xhi, ylo, yhi, K; };
HT_D uint32_t ord_bits(float f) {   // order-preserving map of floats (no NaN) to unsigned
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
HT_D float ord_float(uint32_t o) { return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o); }
HT_D float warp_min(float f) { return ord_float(__reduce_min_sync(0xffffffffu, ord_bits(f))); }
HT_D float warp_max(float f) { return ord_float(__reduce_max_sync(0xffffffffu, ord_bits(f))); }
HT_D WarpBox warp_box(const BoundRay &r) {
    WarpBox b;
    b.r2lo = warp_min(r.r2); b.r2hi = warp_max(r.r2);
    b.xlo = warp_min(r.x);   b.xhi = warp_max(r.x);
    b.ylo = warp_min(r.y);   b.yhi = warp_max(r.y);
    b.K = warp_max(r.K);
    return b;
}
// interval of a * u over u in [lo, hi], and a bound of |a u| there
HT_D void box_term(float a, float lo, float hi, float &flo, float &fhi, float &mag) {
    const float p = a * lo, q = a * hi;
    flo += fminf(p, q);
    fhi += fmaxf(p, q);
    mag += fmaxf(fabsf(p), fabsf(q));
}
// Slots of the chunk at c0 that some lane of the warp may keep (every lane calls this); the low
// two bits of shape[q] are 0 for planes.
HT_D uint32_t warp_survivors(const float4 *bound, const float *mags, const uint32_t *shape, uint32_t c0, uint32_t valid,
                             const WarpBox &b, const PointCut &kp, const PointCut &kh) {
    const uint32_t lane = threadIdx.x & 31;
    const float hp = warp_max(kp.hi.x);   // planes: lo = -hi
    const float lh = warp_min(kh.lo.x), hh = warp_max(kh.hi.x);
    bool keep = false;
    if (valid >> lane & 1u) {
        const uint32_t q = c0 + lane;
        const float4 rec = bound[q];
        const float e = mags[q] * b.K;
        float flo = rec.w, fhi = rec.w, mag = fabsf(rec.w);
        box_term(rec.x, b.r2lo, b.r2hi, flo, fhi, mag);
        box_term(rec.y, b.xlo, b.xhi, flo, fhi, mag);
        box_term(rec.z, b.ylo, b.yhi, flo, fhi, mag);
        const float slack = 0x1p-16f * (mag + e);
        float lo = lh, hi = hh;
        if ((shape[q] & 3u) == 0) {
            lo = -hp;
            hi = hp;
        }
        keep = !((fhi + e) + slack < lo || (flo - e) - slack > hi);   // NaN: kept
    }
    return __ballot_sync(0xffffffffu, keep);
}

// ---------------------------------------------------------------- Euclidean bounds
// The same idea for unit spheres and planes under rigid maps: world-space tests with wide margins
// that rule out objects the reference's test cannot report nearer than the best hit so far.
// Per object one float4, staged once per launch (eu_stage_bound):
//   sphere  its centre c. With m = c - p, b = m.v, the line passes the centre at a squared
//           distance q2 = |m|^2 - b^2; the roots are b -+ sqrt(1 - q2). It is missed when q2 > 1,
//           behind when b < 0 and |m| > 1, and no root is nearer than b - 1.
//   plane   its normal n (local z) and w = -n.c: h = n.p + w and n.v are the local heights of the
//           start and the direction; missed when they have one sign, else hit at -h / n.v.
// Margins: the reference's local ray differs from the exact one by at most about 1e-6 of
// (|p| + |c|) in position and, for a quaternion whose norm the staging lets pass, 1e-5 in scale;
// the tests allow 1e-4 |m|^2 + 1.6e-5 |p|_1 + 1e-3 on q2 (|c|_1 <= |p|_1 + 2 |m|), 2e-3 + 8e-6 |p|_1
// on h (planes with |c|_1 <= 250 only), 2e-5 on n.v, and 1e-4 relative + 1e-3 + 1.6e-5 |p|_1 on
// distances. Other objects get NaN records, which no test culls; rays whose direction is not of
// unit length to 2e-5, or that start beyond 10^4, are not culled at all.
// tests/cull_check/eu_check.c runs them against the full scan on the CPU.
HT_D float4 eu_stage_bound(const Hom &m, uint32_t shape) {
    const double w = m.rot.x, x = m.rot.y, y = m.rot.z, z = m.rot.w;
    const double cx = m.shift.x, cy = m.shift.y, cz = m.shift.z;
    const double c1 = fabs(cx) + fabs(cy) + fabs(cz);
    const float nan = __int_as_float(0x7fc00000);
    if (!(fabs(w * w + x * x + y * y + z * z - 1.0) <= 1e-5 && c1 <= (shape == 0 ? 250.0 : 1e4)))
        return make_float4(nan, nan, nan, nan);
    if (shape != 0) return make_float4(m.shift.x, m.shift.y, m.shift.z, 0.0f);
    const double nx = 2.0 * (x * z + w * y), ny = 2.0 * (y * z - w * x), nz = 1.0 - 2.0 * (x * x + y * y);
    return make_float4((float)nx, (float)ny, (float)nz, (float)-(nx * cx + ny * cy + nz * cz));
}
struct EuBoundRay {
    V3 p, v;
    float base;   // 1 + the margin of q2 without its |m|^2 part
    float dh;     // margin of a plane's h
    float dd;     // absolute margin of a distance
    bool can;     // the ray may be culled for
};
HT_D EuBoundRay eu_bound_ray(V3 p, V3 v) {
    EuBoundRay r;
    r.p = p;
    r.v = v;
    const float p1 = fabsf(p.x) + fabsf(p.y) + fabsf(p.z);
    r.dd = fmaf(1.6e-5f, p1, 1e-3f);
    r.base = 1.0f + r.dd;
    r.dh = fmaf(8e-6f, p1, 2e-3f);
    r.can = p1 <= 1e4f && fabsf(dot3(v, v) - 1.0f) <= 2e-5f;
    return r;
}
// The limit that a hit at distance d sets: objects whose nearest possible hit lies beyond it
// are culled.
HT_D float eu_limit(float d, const EuBoundRay &r) { return fmaf(d, 1.0f + 1e-4f, r.dd); }
// Whether one object is culled; `limit` is lowered when the object is surely hit.
HT_D bool eu_culled_sphere(float4 rec, const EuBoundRay &r, float &limit) {
    const float mx = rec.x - r.p.x, my = rec.y - r.p.y, mz = rec.z - r.p.z;
    const float b = fmaf(mx, r.v.x, fmaf(my, r.v.y, mz * r.v.z));
    const float mm = fmaf(mx, mx, fmaf(my, my, mz * mz));
    const float q2 = fmaf(-b, b, mm), top = fmaf(1e-4f, mm, r.base);
    const bool out = mm > top;
    if (q2 > top || (b < 0.0f && out) || b - 1.0f > limit) return true;
    const float s = (2.0f - top) - q2;   // lower bound of 1 - q2
    if (s > 0.0f && b > 0.0f && out) limit = fminf(limit, eu_limit(fmaf(-(1.0f - 1e-6f), sqrt_approx(s), b), r));
    return false;
}
HT_D bool eu_culled_plane(float4 rec, const EuBoundRay &r, bool repeat, float &limit) {
    const float h = fmaf(rec.x, r.p.x, fmaf(rec.y, r.p.y, fmaf(rec.z, r.p.z, rec.w)));
    const float n = fmaf(rec.x, r.v.x, fmaf(rec.y, r.v.y, rec.z * r.v.z));
    const float hlo = fabsf(h) - r.dh, an = fabsf(n);
    const bool ahead = (h > 0.0f) != (n > 0.0f);
    if (repeat || (hlo > 0.0f && ((!ahead && an > 2e-5f) || hlo > limit * (an + 2e-5f)))) return true;
    if (ahead && hlo > 0.0f && an > 0.01f) limit = fminf(limit, eu_limit((fabsf(h) + r.dh) * rcp_approx(an - 2e-5f) * (1.0f + 1e-6f), r));
    return false;
}
// The far test alone, for a candidate whose turn has come.
HT_D bool eu_far_sphere(float4 rec, const EuBoundRay &r, float limit) {
    return fmaf(rec.x - r.p.x, r.v.x, fmaf(rec.y - r.p.y, r.v.y, (rec.z - r.p.z) * r.v.z)) - 1.0f > limit;
}

}  // namespace ht
