// ht_math.cuh -- device float math for the render path, in the reference's evaluation order.
//
// Every helper keeps the operation order and rounding points of the reference's kernel
// library (kernel/ocl/algebra/*.cc, transform/*.cc) so that, compiled with FMA
// contraction off (-fmad=false) and IEEE division / square root, each result is
// bit-identical to the reference compiled for the host. Transcendentals are the
// exception: logf is CUDA's, cos and sin are evaluated in FP64 and rounded once (see below);
// the host libm's float versions return other values on a small fraction of arguments.
#pragma once
#ifdef __CUDACC_RTC__
// Runtime compilation (NVRTC) has no C++ standard headers; these are the only ones used.
typedef unsigned char uint8_t;
typedef unsigned int uint32_t;
typedef unsigned long long uint64_t;
typedef int int32_t;
typedef unsigned long long uintptr_t;
#else
#include <cstdint>
#endif

namespace ht {

struct C2 { float x, y; };
struct Q4 { float x, y, z, w; };   // x = real part; (y, z, w) = (i, j, k)
struct V3 { float x, y, z; };
struct Col { float x, y, z; };
struct Mo { C2 a, b, c, d; };      // (a p + b)(c p + d)^-1
struct Hom { V3 shift; Q4 rot; };  // Chain<Shift3, Rotation3>: p -> rot(p) + shift

#define HT_D __device__ __forceinline__

HT_D Q4 q4(float x, float y, float z, float w) { Q4 r; r.x = x; r.y = y; r.z = z; r.w = w; return r; }
HT_D V3 v3(float x, float y, float z) { V3 r; r.x = x; r.y = y; r.z = z; return r; }

// ------------------------------------------------------------------- RNG
// kernel/ocl/random.cc:8-14
HT_D uint32_t rng_next(uint32_t &s) { s = 1103515245u * s + 12345u; return s; }
HT_D float rng_uniform(uint32_t &s) {
    return __uint2float_rn(rng_next(s)) / 4294967296.0f;
}

// ------------------------------------------------------------------- vectors
// dot = (((0 + a0 b0) + a1 b1) + ...): kernel/ocl/algebra/vector_math.hpp:8-15
HT_D float dot2(float ax, float ay, float bx, float by) {
    float c = 0.0f; c += ax * bx; c += ay * by; return c;
}
HT_D float dot3(V3 a, V3 b) { float c = 0.0f; c += a.x * b.x; c += a.y * b.y; c += a.z * b.z; return c; }
HT_D float dot4(Q4 a, Q4 b) {
    float c = 0.0f; c += a.x * b.x; c += a.y * b.y; c += a.z * b.z; c += a.w * b.w; return c;
}
HT_D Q4 normalize4(Q4 a) { float l = sqrtf(dot4(a, a)); return q4(a.x / l, a.y / l, a.z / l, a.w / l); }
HT_D V3 cross3(V3 a, V3 b) {
    return v3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// ------------------------------------------------------------------- quaternions
// kernel/ocl/algebra/quaternion.cc:4-56
HT_D Q4 q_conj(Q4 a) { return q4(a.x, -a.y, -a.z, -a.w); }
HT_D Q4 q_mul(Q4 a, Q4 b) {
    return q4(a.x * b.x - a.y * b.y - a.z * b.z - a.w * b.w,
              a.x * b.y + a.y * b.x + a.z * b.w - a.w * b.z,
              a.x * b.z + a.z * b.x - a.y * b.w + a.w * b.y,
              a.x * b.w + a.w * b.x + a.y * b.z - a.z * b.y);
}
HT_D Q4 cq_mul(C2 a, Q4 b) {
    return q4(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x, a.x * b.z - a.y * b.w, a.x * b.w + a.y * b.z);
}
HT_D Q4 q_add(Q4 a, Q4 b) { return q4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
HT_D Q4 q_sub(Q4 a, Q4 b) { return q4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w); }
HT_D Q4 q_addc(Q4 a, C2 b) { return q4(a.x + b.x, a.y + b.y, a.z + 0.0f, a.w + 0.0f); }  // + q_new(c, C0)

// Packed FP32: two operations an instruction, each half rounded as the scalar operation is. ptxas
// (12.9) contracts a packed product and sum into one FMA whatever their rounding modifiers and
// -fmad say; a sum as an FMA with a factor of 1 or -1 that it cannot know (a constant bank
// operand) is the same sum and stays apart from the product.
static __constant__ float2 c_plus = {1.0f, 1.0f}, c_minus = {-1.0f, -1.0f};
HT_D float2 both(float a) { return make_float2(a, a); }
HT_D float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
HT_D float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
HT_D float2 add2(float2 a, float2 b) { return __ffma2_rn(a, c_plus, b); }
HT_D float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, c_minus, a); }
// Two quaternions side by side.
struct QQ { float2 x, y, z, w; };
HT_D QQ qq(Q4 a, Q4 b) {
    QQ r;
    r.x = make_float2(a.x, b.x); r.y = make_float2(a.y, b.y); r.z = make_float2(a.z, b.z); r.w = make_float2(a.w, b.w);
    return r;
}
HT_D Q4 qq_first(const QQ &a) { return q4(a.x.x, a.y.x, a.z.x, a.w.x); }
HT_D Q4 qq_second(const QQ &a) { return q4(a.x.y, a.y.y, a.z.y, a.w.y); }
HT_D QQ cqq_mul(C2 a, const QQ &b) {   // cq_mul of both
    const float2 x = both(a.x), y = both(a.y);
    QQ r;
    r.x = sub2(mul2(x, b.x), mul2(y, b.y));
    r.y = add2(mul2(x, b.y), mul2(y, b.x));
    r.z = sub2(mul2(x, b.z), mul2(y, b.w));
    r.w = add2(mul2(x, b.w), mul2(y, b.z));
    return r;
}
HT_D QQ qq_mul(const QQ &a, const QQ &b) {   // q_mul of both
    QQ r;
    r.x = sub2(sub2(sub2(mul2(a.x, b.x), mul2(a.y, b.y)), mul2(a.z, b.z)), mul2(a.w, b.w));
    r.y = sub2(add2(add2(mul2(a.x, b.y), mul2(a.y, b.x)), mul2(a.z, b.w)), mul2(a.w, b.z));
    r.z = add2(sub2(add2(mul2(a.x, b.z), mul2(a.z, b.x)), mul2(a.y, b.w)), mul2(a.w, b.y));
    r.w = sub2(add2(add2(mul2(a.x, b.w), mul2(a.w, b.x)), mul2(a.y, b.z)), mul2(a.z, b.y));
    return r;
}

// ------------------------------------------------------------------- division
// Correctly rounded quotients that share one reciprocal (Markstein's correction step):
//   y = RN(1/b),  q0 = RN(a*y),  r = b*q0 - a (exact with an FMA),  q = RN(q0 - r*y) = RN(a/b)
// (P. Markstein, "IA-64 and Elementary Functions", 2000; Muller et al., "Handbook of
// Floating-Point Arithmetic", 2nd ed., section 4.7, Markstein's theorem). Divisors here are
// squared norms and lengths (b > 0); taking the residual as b*q0 - a keeps IEEE's sign of a
// zero quotient without a select (a = -0: q0 = -0, r = +0, q = -0 + -0). The identity needs
// every intermediate to be a normal number: each divisor lies in [2^-60, 2^60] and each
// numerator is zero or at least 2^-60 (then |q0| >= 2^-120 and the residual's last place is at
// least 2^-108). A numerator so large that q0 overflows makes q NaN, and NaN reaches the
// length of the result, whose own range check fails. A group with any value outside redoes its
// divisions with IEEE division. The numerators' check costs one add and half a 3-input minimum
// per quotient (2 * bits - 1 drops the sign and maps zero to the largest word): about 4.5
// instructions per quotient in place of 9 with a range test of every q0, 17 quotients per ray
// map, three to nine maps per hop. Measured together with sincos_turn and the estimate's loop
// per shape (ht_trace.cuh): 1080p / 200 objects, 8 passes 17.24 -> 16.09 ms; 800x600 / 18
// objects, 64 passes 27.2 -> 24.4 ms; 24 mixed views batched 61.2 -> 57.2 ms.
// tests/test_gpu_math.py compares qdiv with IEEE division on billions of inputs.
struct Rcp { float b, y; };
struct DivCheck {   // of one group of quotients
    uint32_t least;   // over the numerators: 2 * bits - 1
    bool bad;         // a divisor out of range
};
constexpr uint32_t DIV_LEAST = 2u * 0x21800000u - 1u;   // the word of 2^-60
HT_D DivCheck div_check() { DivCheck c; c.least = 0xFFFFFFFFu; c.bad = false; return c; }
HT_D bool div_failed(const DivCheck &c) { return c.bad | (c.least < DIV_LEAST); }
HT_D uint32_t div_word(float a) { const uint32_t b = __float_as_uint(a); return b + b - 1u; }
HT_D bool in_safe_range(float x) {
    const float ax = fabsf(x);
    return ax >= 0x1p-60f && ax <= 0x1p60f;
}
HT_D Rcp rcp_of(float b, bool &bad) {
    bad |= !in_safe_range(b);
    Rcp r;
    r.b = b;
    r.y = __frcp_rn(b);
    return r;
}
HT_D Rcp rcp_of(float b, DivCheck &c) { return rcp_of(b, c.bad); }
HT_D float qdiv_unchecked(float a, const Rcp &r) {
    const float q0 = a * r.y;
    const float e = fmaf(r.b, q0, -a);
    return fmaf(-e, r.y, q0);
}
HT_D float2 qdiv2_unchecked(float2 a, const Rcp &r) {   // two quotients, packed
    const float2 y = both(r.y), q0 = __fmul2_rn(a, y);
    return __ffma2_rn(neg2(__ffma2_rn(both(r.b), q0, neg2(a))), y, q0);
}
HT_D float qdiv(float a, const Rcp &r, DivCheck &c) {
    c.least = min(c.least, div_word(a));
    return qdiv_unchecked(a, r);
}
// One quotient with a check of its own, for a divisor of either sign.
HT_D float qdiv(float a, const Rcp &r, bool &bad) {
    bad |= (div_word(a) < DIV_LEAST) | (fabsf(a * r.y) > 0x1p60f) | (a == 0.0f & r.b < 0.0f);
    return qdiv_unchecked(a, r);
}
template <bool PACKED = false> HT_D Q4 qdiv4(Q4 a, const Rcp &r, DivCheck &c) {
    c.least = min(min(c.least, div_word(a.x)), min(min(div_word(a.y), div_word(a.z)), div_word(a.w)));
    if constexpr (PACKED) {
        const float2 xy = qdiv2_unchecked(make_float2(a.x, a.y), r), zw = qdiv2_unchecked(make_float2(a.z, a.w), r);
        return q4(xy.x, xy.y, zw.x, zw.y);
    }
    return q4(qdiv_unchecked(a.x, r), qdiv_unchecked(a.y, r), qdiv_unchecked(a.z, r), qdiv_unchecked(a.w, r));
}
// normalize3 and normalize4 through one correctly rounded reciprocal of the length.
static __device__ __noinline__ V3 normalize3_ieee(V3 a) { float l = sqrtf(dot3(a, a)); return v3(a.x / l, a.y / l, a.z / l); }
HT_D V3 normalize3(V3 a) {
    DivCheck c = div_check();
    const Rcp r = rcp_of(sqrtf(dot3(a, a)), c);
    c.least = min(min(div_word(a.x), div_word(a.y)), div_word(a.z));
    if (div_failed(c)) return normalize3_ieee(a);
    return v3(qdiv_unchecked(a.x, r), qdiv_unchecked(a.y, r), qdiv_unchecked(a.z, r));
}
template <bool PACKED = false> HT_D Q4 normalize4_fast(Q4 a, DivCheck &c) {
    float l = sqrtf(dot4(a, a));
    Rcp r = rcp_of(l, c);
    return qdiv4<PACKED>(a, r, c);
}

// q_inverse(d) = conj(d) / |d|^2 through one reciprocal (the four divisions share it).
static __device__ __noinline__ Q4 q_inverse_ieee(Q4 d) {
    const float d2 = dot4(d, d);
    return q4(d.x / d2, (-d.y) / d2, (-d.z) / d2, (-d.w) / d2);
}
HT_D Q4 q_inverse(Q4 d) {
    DivCheck chk = div_check();
    const Rcp r = rcp_of(dot4(d, d), chk);
    const Q4 q = qdiv4(q4(d.x, -d.y, -d.z, -d.w), r, chk);
    return div_failed(chk) ? q_inverse_ieee(d) : q;
}

// ------------------------------------------------------------------- Moebius
// mo_apply_q and mo_deriv_q (kernel/ocl/transform/moebius.cc:20-42) share the numerator u,
// the denominator d, |d|^2 and q_inverse(d) = conj(d) / |d|^2.
struct HyRay { Q4 p, v; };

// Reference evaluation with IEEE division everywhere (the fallback of the maps below). `twice`:
// mo_apply_dir normalizes, ray_map.inl:19 again.
static __device__ __noinline__ HyRay hy_map_ieee(const Mo m, const Q4 p, const Q4 v, bool twice) {
    Q4 u = q_addc(cq_mul(m.a, p), m.b);
    Q4 d = q_addc(cq_mul(m.c, p), m.d);
    float d2 = dot4(d, d);
    Q4 di = q4(d.x / d2, (-d.y) / d2, (-d.z) / d2, (-d.w) / d2);   // q_inverse(d)
    HyRay o;
    o.p = q_mul(u, di);                                             // mo_apply_q
    Q4 g1 = q_mul(cq_mul(m.a, v), di);                              // q_div(cq_mul(a, v), d)
    Q4 cv = cq_mul(m.c, v);
    Q4 g21 = q_conj(cv);
    float k = (2.0f * dot4(d, cv)) / d2;
    Q4 dc = q_conj(d);
    Q4 g22 = q4(k * dc.x, k * dc.y, k * dc.z, k * dc.w);
    Q4 t = q_sub(g21, g22);
    Q4 g2 = q_mul(u, q4(t.x / d2, t.y / d2, t.z / d2, t.w / d2));
    o.v = normalize4(q_add(g1, g2));
    if (twice) o.v = normalize4(o.v);
    return o;
}
static __device__ __forceinline__ HyRay ray_hy_map_ieee(const Mo m, const Q4 p, const Q4 v) { return hy_map_ieee(m, p, v, true); }

// ray_<hy>_map (geometry/ray_map.inl:15-21; TWICE) and the camera map (view/mapped.inl:20-26:
// direction = mo_apply_dir, one normalize, then start): the nine divisions by |d|^2 share one
// reciprocal, each normalize shares one; results are bit-identical to hy_map_ieee.
// PACKED: the position and the direction side by side through the two products that they share
// and the quotients two at a time, 15 % fewer instructions. The hand-written kernels take it
// (24 mixed views batched 35.75 -> 35.34 ms, 800x600 64 passes 18.44 -> 17.81, 1080p / 200 objects, 8
// passes 9.21 -> 9.01); the generic kernels, which have 64 registers for more state, lose 3 % to
// the register pairs (64 tiled objects at 1080p 22.1 -> 22.8 ms) and keep the scalar form.
template <bool TWICE, bool PACKED> HT_D HyRay hy_map(const Mo &m, const QQ &pv) {
    DivCheck chk = div_check();
    const Q4 p = qq_first(pv), v = qq_second(pv);
    Q4 u, d, cv, g1;
    QQ av;
    if constexpr (PACKED) {
        const QQ cpv = cqq_mul(m.c, pv);
        av = cqq_mul(m.a, pv);
        u = q_addc(qq_first(av), m.b);
        d = q_addc(qq_first(cpv), m.d);
        cv = qq_second(cpv);
    } else {
        u = q_addc(cq_mul(m.a, p), m.b);
        d = q_addc(cq_mul(m.c, p), m.d);
    }
    const Rcp rd = rcp_of(dot4(d, d), chk);
    const Q4 di = qdiv4<PACKED>(q4(d.x, -d.y, -d.z, -d.w), rd, chk);
    HyRay o;
    if constexpr (PACKED) {
        const QQ og = qq_mul(qq(u, qq_second(av)), qq(di, di));
        o.p = qq_first(og);
        g1 = qq_second(og);
    } else {
        o.p = q_mul(u, di);
        g1 = q_mul(cq_mul(m.a, v), di);
        cv = cq_mul(m.c, v);
    }
    const Q4 g21 = q_conj(cv), dc = q_conj(d);
    const float k = qdiv(2.0f * dot4(d, cv), rd, chk);
    const Q4 g22 = q4(k * dc.x, k * dc.y, k * dc.z, k * dc.w);
    const Q4 g2 = q_mul(u, qdiv4<PACKED>(q_sub(g21, g22), rd, chk));
    o.v = normalize4_fast<PACKED>(q_add(g1, g2), chk);
    if (TWICE) o.v = normalize4_fast<PACKED>(o.v, chk);
    if (div_failed(chk)) return hy_map_ieee(m, p, v, TWICE);
    return o;
}
HT_D HyRay ray_hy_map(const Mo &m, Q4 p, Q4 v) { return hy_map<true, false>(m, qq(p, v)); }
HT_D HyRay view_hy_map(const Mo &m, Q4 p, Q4 v) { return hy_map<false, false>(m, qq(p, v)); }
HT_D HyRay view_hy_map_packed(const Mo &m, Q4 p, Q4 v) { return hy_map<false, true>(m, qq(p, v)); }
// The same map, out of line: the object scan and the hit path share this one copy of its
// code (instruction-cache footprint; an inlined copy in the scan measured slower). The packed
// one takes its arguments in the pairs that it works on.
static __device__ __noinline__ HyRay ray_hy_map_call(const Mo m, const Q4 p, const Q4 v) { return ray_hy_map(m, p, v); }
static __device__ __noinline__ HyRay ray_hy_map_packed(const Mo m, const QQ pv) { return hy_map<true, true>(m, pv); }

HT_D Q4 mo_apply_pos(const Mo &m, Q4 p) {   // mo_apply_q (transform/moebius.cc:20-25)
    return q_mul(q_addc(cq_mul(m.a, p), m.b), q_inverse(q_addc(cq_mul(m.c, p), m.d)));
}

// c22_inverse_n (kernel/ocl/algebra/matrix_complex.cc:60-65): adjugate, det = 1 assumed.
HT_D Mo mo_inverse(const Mo &m) {
    Mo r;
    r.a = m.d;
    r.b.x = -m.b.x; r.b.y = -m.b.y;
    r.c.x = -m.c.x; r.c.y = -m.c.y;
    r.d = m.a;
    return r;
}

// ------------------------------------------------------------------- Euclidean maps
// rot3_apply_pos = (q (0, p) q*).yzw (transform/rotation.cc); chain.inl:36-73; shift.cc
struct EuRay { V3 p, v; };
HT_D V3 rot3_apply(Q4 q, V3 p) {
    Q4 r = q_mul(q_mul(q, q4(0.0f, p.x, p.y, p.z)), q_conj(q));
    return v3(r.y, r.z, r.w);
}
HT_D V3 hom3_apply_pos(const Hom &m, V3 p) {
    V3 r = rot3_apply(m.rot, p);
    return v3(r.x + m.shift.x, r.y + m.shift.y, r.z + m.shift.z);
}
HT_D EuRay ray_eu_map(const Hom &m, V3 p, V3 v) {
    EuRay o;
    o.p = hom3_apply_pos(m, p);
    o.v = normalize3(rot3_apply(m.rot, v));
    return o;
}
// The same map, out of line: the object scan and the hit path share this one copy of its code.
// Packed: the position and the direction are turned side by side (1917x1077, 25 objects, 16 passes:
// 4.77 -> 4.60 ms).
static __device__ __noinline__ EuRay ray_eu_map_call(const Hom m, const V3 p, const V3 v) {
    const Q4 c = q_conj(m.rot);
    const QQ r = qq_mul(qq_mul(qq(m.rot, m.rot), qq(q4(0.0f, p.x, p.y, p.z), q4(0.0f, v.x, v.y, v.z))), qq(c, c));
    EuRay o;
    o.p = v3(r.y.x + m.shift.x, r.z.x + m.shift.y, r.w.x + m.shift.z);
    o.v = normalize3(v3(r.y.y, r.z.y, r.w.y));
    return o;
}
HT_D Hom hom3_inverse(const Hom &m) {
    Hom s;
    s.shift = v3(-m.shift.x, -m.shift.y, -m.shift.z);
    s.rot = q_conj(m.rot);
    s.shift = rot3_apply(s.rot, s.shift);
    return s;
}

// ------------------------------------------------------------------- hyperbolic geometry
// kernel/ocl/geometry/hyperbolic.cc:20-33, split in two: hy_distance(a, b) =
// hy_dist_from_x(hy_x(a, b)). The object scan compares x and evaluates the logarithm only
// for a candidate that can be nearer than the current one; that equals comparing the
// distances because hy_dist_from_x, as compiled here, is non-decreasing on [1, inf]
// (checked exhaustively over every float in tests/test_gpu_math.py).
HT_D float hy_x(Q4 a, Q4 b) {
    Q4 d = q_sub(a, b);
    return 1.0f + dot4(d, d) / (2.0f * a.z * b.z);
}
// CUDA's single-precision logf. Evaluating it in FP64 and rounding once (what the host libm's
// logf returns) was measured: the share of pixels that differ from the reference over 16
// passes of the 1080p frame stayed 0.365 % (the flips come from cos / sin, below), and the
// headline kernel lost 4.5 % (the generic kernel 30 %).
HT_D float hy_dist_from_x(float x) {
    return logf(x + sqrtf(x * x - 1.0f));
}
HT_D float hy_distance(Q4 a, Q4 b) { return hy_dist_from_x(hy_x(a, b)); }
HT_D Q4 hy_dir_at(Q4 p, Q4 d, Q4 h) {
    float lpxy = sqrtf(dot2(p.x - h.x, p.y - h.y, p.x - h.x, p.y - h.y));
    float ldxy = sqrtf(dot2(d.x, d.y, d.x, d.y));
    float k = h.z / p.z;
    return q4(k * d.x, k * d.y, d.z - lpxy / p.z * ldxy, 0.0f);
}

// ------------------------------------------------------------------- samplers / rotations
// (float)sin(x) and (float)cos(x) of a float angle in [0, 2 pi], evaluated in FP64 and rounded
// once: quarter turns taken off with pi/2 in two parts (Cody and Waite), then the Taylor series
// on [-pi/4, pi/4] (the first term left out is below 2^-58 of the result). A sampler's angles
// are 2 pi u of a 32-bit state, so every one of them was compared with CUDA's FP64 sincos
// (tests/test_gpu_sincos.py): the same floats. That function also serves large angles, which
// costs the hop kernels twice the instructions and a slow path in their instruction stream.
HT_D void sincos_turn(float angle, float &sn, float &cs) {
    const double x = (double)angle;
    const double k = rint(x * 0.63661977236758134308);
    const double r = fma(-k, 6.12323399573676603587e-17, fma(-k, 1.57079632679489655800, x));
    const double z = r * r;
    double s = fma(z, 1.0 / 355687428096000.0, -1.0 / 1307674368000.0);
    double c = fma(z, 1.0 / 20922789888000.0, -1.0 / 87178291200.0);
    s = fma(z, s, 1.0 / 6227020800.0);
    c = fma(z, c, 1.0 / 479001600.0);
    s = fma(z, s, -1.0 / 39916800.0);
    c = fma(z, c, -1.0 / 3628800.0);
    s = fma(z, s, 1.0 / 362880.0);
    c = fma(z, c, 1.0 / 40320.0);
    s = fma(z, s, -1.0 / 5040.0);
    c = fma(z, c, -1.0 / 720.0);
    s = fma(z, s, 1.0 / 120.0);
    c = fma(z, c, 1.0 / 24.0);
    s = fma(z, s, -1.0 / 6.0);
    c = fma(z, c, -0.5);
    const float fs = (float)fma(r * z, s, r), fc = (float)fma(z, c, 1.0);
    const int q = (int)k;
    const float a = q & 1 ? fc : fs, b = q & 1 ? fs : fc;
    sn = q & 2 ? -a : a;
    cs = (q + 1) & 2 ? -b : b;
}
// random_hemisphere_cosine (kernel/ocl/random.cc:37-39,53-59). cos/sin are evaluated in
// FP64 and rounded once: this lands on the correctly rounded float, which the host libm
// the reference is built against matches far more often than a float kernel does.
HT_D V3 hemisphere_cosine(uint32_t &s) {
    float phi = 2.0f * 3.14159265358979323846f * rng_uniform(s);
    float sqr_cos_theta = rng_uniform(s);
    float cos_theta = sqrtf(sqr_cos_theta);
    float sin_theta = sqrtf(1.0f - sqr_cos_theta);
    float sd, cd;
    sincos_turn(phi, sd, cd);
    return v3(cd * sin_theta, sd * sin_theta, cos_theta);
}
// rot3_look_at_cont / rot3_look_at / rot3_from_axis (kernel/ocl/transform/rotation.cc)
HT_D Q4 rot3_look_at_cont(V3 d) {
    V3 z = v3(0.0f, 0.0f, -1.0f);
    float c2 = dot3(d, z);
    float c = sqrtf((1.0f + c2) / 2.0f);
    float sm = 1.0f / (2.0f * c);
    V3 x = cross3(z, d);
    return q4(c, sm * x.x, sm * x.y, sm * x.z);
}
HT_D Q4 rot3_look_at(V3 d) {
    if (d.z < 0.0f) return rot3_look_at_cont(d);
    Q4 a = rot3_look_at_cont(v3(-d.x, -d.y, -d.z));
    // rot3_from_axis(x, pi): the FP64 sine and cosine of (float)pi / 2, each rounded to float
    Q4 b = q4(-0x1.777a5cp-25f, 1.0f, 0.0f, 0.0f);
    return q_mul(a, b);
}

}  // namespace ht
