// ht_trace.cuh -- scene access and the per-hop path logic for the two scene recipes.
//
// Device-side restatement of render/scene.inl:16-44 (hop loop), object/vector.inl:24-74
// (nearest-hit scan), object/mapped.inl:24-51, object/covered.inl:23-56, the shapes in
// shape/hy/{plane,horosphere}.cc and shape/eu/{plane,sphere}.cc, the mixture material
// (material/mixture/impl.inl:16-27 with colored.inl, lambertian.cc, specular.cc,
// emissive.inl, absorbing.cc), the point camera (view/point/impl.inl:18-25,
// view/mapped.inl:20-26) and the constant background (background/constant.inl:18-21).
//
// Scheduling differs from the reference, results do not:
//  * the object scan keeps the best candidate's distance, index and local ray, and computes
//    its hit point and normal from that ray afterwards -- the same inputs through the same
//    operations give the same bits, so this equals keeping every candidate's light/cache copy;
//  * only the winner is mapped back to world space (the reference maps every candidate
//    back, mapped.inl:34, but only the kept copy is observable);
//  * inverse maps are computed once per launch and staged in shared memory.
#pragma once
#include "ht_math.cuh"
#include "ht_bound.cuh"

namespace ht {

constexpr int RECIPE_HY = 1;
constexpr int RECIPE_EU = 2;
constexpr float EPSF = 1e-6f;   // EPS for real = float (kernel/ocl/algebra/real.hh:19-25)
constexpr uint32_t HASH_NEVER = 0xFFFFFFFFu;  // hash_never (kernel/ocl/hash.cc:22-24)
constexpr uint32_t OBJ_STRIDE = 128;
constexpr uint32_t FLAG_JITTER_YX = 1u;

// Serialized scene byte offsets (see hypertrace_b200/scene.py for the derivation).
template <int R> struct Layout;
template <> struct Layout<RECIPE_HY> {
    static constexpr uint32_t FOV = 32, BG = 64, COUNT = 96, OBJECTS = 128;
};
template <> struct Layout<RECIPE_EU> {
    static constexpr uint32_t FOV = 32, BG = 48, COUNT = 64, OBJECTS = 80;
};
// Object record offsets (Mapped<Covered<Choice, Mixture>, Map>).
constexpr uint32_t O_DIFFUSE_COLOR = 32, O_DIFFUSE = 48, O_SPECULAR = 64, O_EMISSION = 80,
                   O_LUMINOUS = 96, O_SHAPE = 112;

struct Material {
    Col diffuse_color;
    float diffuse, specular, luminous;
    Col emission;
};

HT_D float ldf(const uint8_t *base, uint32_t off) { return __ldg(reinterpret_cast<const float *>(base + off)); }
HT_D float4 ldf4(const uint8_t *base, uint32_t off) { return __ldg(reinterpret_cast<const float4 *>(base + off)); }
HT_D uint32_t ldu(const uint8_t *base, uint32_t off) { return __ldg(reinterpret_cast<const uint32_t *>(base + off)); }

HT_D Material load_material(const uint8_t *obj) {
    Material m;
    float4 dc = ldf4(obj, O_DIFFUSE_COLOR);
    m.diffuse_color.x = dc.x; m.diffuse_color.y = dc.y; m.diffuse_color.z = dc.z;
    m.diffuse = ldf(obj, O_DIFFUSE);
    m.specular = ldf(obj, O_SPECULAR);
    float4 em = ldf4(obj, O_EMISSION);
    m.emission.x = em.x; m.emission.y = em.y; m.emission.z = em.z;
    m.luminous = ldf(obj, O_LUMINOUS);
    return m;
}

HT_D Mo load_mo(const uint8_t *p) {
    float4 a = ldf4(p, 0), b = ldf4(p, 16);
    Mo m;
    m.a.x = a.x; m.a.y = a.y; m.b.x = a.z; m.b.y = a.w;
    m.c.x = b.x; m.c.y = b.y; m.d.x = b.z; m.d.y = b.w;
    return m;
}
HT_D Hom load_hom(const uint8_t *p) {
    float4 a = ldf4(p, 0), b = ldf4(p, 16);
    Hom h;
    h.shift = v3(a.x, a.y, a.z);
    h.rot = q4(b.x, b.y, b.z, b.w);
    return h;
}
HT_D Mo mo_from(float4 a, float4 b) {
    Mo m;
    m.a.x = a.x; m.a.y = a.y; m.b.x = a.z; m.b.y = a.w;
    m.c.x = b.x; m.c.y = b.y; m.d.x = b.z; m.d.y = b.w;
    return m;
}
HT_D Hom hom_from(float4 a, float4 b) {
    Hom h;
    h.shift = v3(a.x, a.y, a.z);
    h.rot = q4(b.x, b.y, b.z, b.w);
    return h;
}

// Mixture interact: one uniform draw picks the component; returns false when the path ends
// (Emissive<Absorbing>, or the draw falls past every portion).
HT_D bool mixture_interact(const Material &m, uint32_t &rng, V3 normal, V3 &dir, Col &intensity,
                           Col &emission) {
    float alpha = rng_uniform(rng);
    alpha -= m.diffuse;
    if (alpha < 0.0f) {
        intensity.x *= m.diffuse_color.x;
        intensity.y *= m.diffuse_color.y;
        intensity.z *= m.diffuse_color.z;
        if (dot3(dir, normal) > 0.0f) normal = v3(-normal.x, -normal.y, -normal.z);
        V3 rnd = hemisphere_cosine(rng);
        Q4 rot = rot3_look_at(v3(-normal.x, -normal.y, -normal.z));
        dir = rot3_apply(rot, rnd);
        return true;
    }
    alpha -= m.specular;
    if (alpha < 0.0f) {
        float k = 2.0f * dot3(dir, normal);
        dir = v3(dir.x - k * normal.x, dir.y - k * normal.y, dir.z - k * normal.z);
        return true;
    }
    alpha -= m.luminous;
    if (alpha < 0.0f) {
        emission.x += intensity.x * m.emission.x;
        emission.y += intensity.y * m.emission.y;
        emission.z += intensity.z * m.emission.z;
        return false;
    }
    return false;
}

// The interaction on a path's last hop: the same draws (the pixel's RNG goes on from them) and the
// emission, without the direction that nothing will follow -- and so without the hit point and
// the ray maps that only it needs.
HT_D void mixture_last(const Material &m, uint32_t &rng, const Col &intensity, Col &emission) {
    float alpha = rng_uniform(rng);
    alpha -= m.diffuse;
    if (alpha < 0.0f) {
        rng_next(rng);
        rng_next(rng);
        return;
    }
    alpha -= m.specular;
    if (alpha < 0.0f) return;
    alpha -= m.luminous;
    if (alpha < 0.0f) {
        emission.x += intensity.x * m.emission.x;
        emission.y += intensity.y * m.emission.y;
        emission.z += intensity.z * m.emission.z;
    }
}

// Staged scene, per slot in shared memory (hyperbolic scenes: planes first, then
// horospheres, each by distance from the camera; Euclidean scenes: slot = scene index).
struct StagedScene {
    const float4 *inv;       // shared, 2 per slot
    const uint32_t *shape;   // shared
    const float4 *bound;     // shared, 1 per slot: world-space form for distance bounds
    const float4 *pa, *pb;   // shared, per pair of slots: {x0, x1, y0, y1}, {z0, z1, w0, w1} of bound
    const float2 *pmag;      // shared, per pair of slots: {mag0, mag1}
    const float *mag;        // shared, 1 per slot: the record's error magnitude (bound_mag)
    const uint32_t *orig;    // shared, 1 per slot: the object's index in the scene
    float4 *win;             // shared, this thread's 2 float4: the scan winner's local ray
    const uint8_t *objects;  // global, OBJ_STRIDE per object (forward maps, materials), by scene index
    uint32_t n;              // objects
    uint32_t ns;             // slots: n, plus the dummy slot of a hyperbolic scene with an odd plane count
    uint32_t n_planes;       // hyperbolic: slots [0, n_planes) are planes, horospheres from the next even slot
    uint32_t dummy;          // the dummy slot, or 0xFFFFFFFF
    float fov;
    Col background;
    float4 cam0, cam1;       // camera map (Moebius or Homogenous3) as stored
};

// -------------------------------------------------------------------------- hyperbolic
struct HyPath { Q4 p, v; };

// Plane test up to the hit point (shape/hy/plane.cc:4-37 without the direction update);
// returns x of the hit distance (see hy_x), or -1 on a miss.
HT_D float plane_hy_x(Q4 p, Q4 d) {
    float pd = dot4(p, d);
    if (fabsf(pd) < EPSF) return -1.0f;
    float s = 1.0f - dot4(p, p);
    float t = s / (2.0f * pd);
    if (t < -EPSF) return -1.0f;
    float hx = p.x + d.x * t, hy = p.y + d.y * t;
    float pxy2 = dot2(hx, hy, hx, hy);
    if (pxy2 > 1.0f) return -1.0f;
    Q4 h = q4(hx, hy, sqrtf(1.0f - pxy2), 0.0f);
    return hy_x(p, h);
}
// Horosphere test up to the hit point (shape/hy/horosphere.cc:4-34); x or -1.
HT_D float horosphere_x(Q4 p, Q4 d, bool repeat) {
    float dxy = sqrtf(dot2(d.x, d.y, d.x, d.y));
    if (p.z < dxy) return -1.0f;
    float dt = sqrtf(p.z * p.z - dxy * dxy);
    float t = p.z * d.z - dt;
    float w = repeat ? EPSF : -EPSF;   // EPS * (2*repeat - 1)
    if (t < w) {
        t += 2.0f * dt;
        if (t < w) return -1.0f;
    }
    t /= dxy * dxy;
    Q4 h = q4(p.x + d.x * t, p.y + d.y * t, 1.0f, 0.0f);
    return hy_x(p, h);
}
// Full tests for the winning object: hit point, transported direction, local normal.
HT_D void plane_hy_hit(Q4 p, Q4 d, HyPath &hit, Q4 &normal) {
    float pd = dot4(p, d);
    float s = 1.0f - dot4(p, p);
    float t = s / (2.0f * pd);
    float hx = p.x + d.x * t, hy = p.y + d.y * t;
    float pxy2 = dot2(hx, hy, hx, hy);
    Q4 h = q4(hx, hy, sqrtf(1.0f - pxy2), 0.0f);
    hit.p = h;
    hit.v = hy_dir_at(p, d, h);
    normal = q4(-h.x, -h.y, -h.z, -h.w);
}
HT_D void horosphere_hit(Q4 p, Q4 d, bool repeat, HyPath &hit, Q4 &normal) {
    float dxy = sqrtf(dot2(d.x, d.y, d.x, d.y));
    float dt = sqrtf(p.z * p.z - dxy * dxy);
    float t = p.z * d.z - dt;
    float w = repeat ? EPSF : -EPSF;
    if (t < w) t += 2.0f * dt;
    t /= dxy * dxy;
    Q4 h = q4(p.x + d.x * t, p.y + d.y * t, 1.0f, 0.0f);
    hit.p = h;
    hit.v = hy_dir_at(p, d, h);
    normal = q4(0.0f, 0.0f, -1.0f, 0.0f);
}

// Camera ray: view/point/impl.inl:18-25 (hy_origin = j, hyperbolic.cc:4-6) then the
// camera Moebius map (view/mapped.inl:20-26).
// Out of line: once per sample, and keeping its code out of the hop kernel's instruction
// stream measured 3 % faster at 1920x1080 / 200 objects.
static __device__ __noinline__ HyPath camera_hy(const StagedScene &s, float px, float py, float size, uint32_t &rng,
                                                uint32_t flags) {
    float u0 = rng_uniform(rng);
    float u1 = rng_uniform(rng);
    float jx = (flags & FLAG_JITTER_YX) ? u1 : u0;
    float jy = (flags & FLAG_JITTER_YX) ? u0 : u1;
    float sx = px + size * (jx - 0.5f);
    float sy = py + size * (jy - 0.5f);
    V3 ld = normalize3(v3(sx, sy, -1.0f / s.fov));
    HyRay r = view_hy_map_packed(mo_from(s.cam0, s.cam1), q4(0.0f, 0.0f, 1.0f, 0.0f), q4(ld.x, ld.y, ld.z, 0.0f));
    HyPath o; o.p = r.p; o.v = r.v;
    return o;
}

// One hop (one iteration of render/scene.inl:25-41). Returns true while the path goes on; `last`:
// it ends here whatever is hit.
// `hit` reports whether the scan found an object (for the hop statistics).
// ---------------------------------------------------------------- the scan's packed point bound
// Objects the upper estimate looks at: the first half of them planes, the others horospheres, the
// nearest to the camera of each (stage_scene's slot order). 1080p / 200 objects, 8 passes: 8 objects
// 11.84 ms, 12 11.29, 16 11.56, 24 12.10; 24 mixed views batched 41.1, 41.0, 41.9, 44.0 ms. In scene
// order 24 to 40 objects were best, and the scan tested 3.2-4.9 objects per hop where it now
// tests 1.4-2.2 (16.3 and 55.3 ms before the slot order, the allowances of ht_bound.cuh and the
// warp-uniform ray-aware tests). Scenes of more than 1024 objects stay in scene order and take the
// same 12: with all of that together 1025, 1500 and 2500 objects at 1280x720, 4 passes take 7.3, 39.4 and
// 19.9 ms (8.8, 60.5 and 24.4 before it, with 24).
constexpr uint32_t HT_EST_OBJECTS = 12;
struct PairRay { float2 r2, x, y, K; };   // the bound ray's constants, each in both halves
HT_D PairRay pair_ray(const BoundRay &r) {
    PairRay p;
    p.r2 = make_float2(r.r2, r.r2);
    p.x = make_float2(r.x, r.x);
    p.y = make_float2(r.y, r.y);
    p.K = make_float2(r.K, r.K);
    return p;
}
HT_D uint32_t survivors2(float4 a, float4 b, float2 mag, const PairRay &r, const PointCut &k) {
    // F = rec.x r2 + (rec.y x + (rec.z y + rec.w)), as culled_point evaluates it
    float2 F = __ffma2_rn(make_float2(b.x, b.y), r.y, make_float2(b.z, b.w));
    F = __ffma2_rn(make_float2(a.z, a.w), r.x, F);
    F = __ffma2_rn(make_float2(a.x, a.y), r.r2, F);
    const float2 e = __fmul2_rn(mag, r.K);                      // eF, once for both sides
    const float2 up = __fadd2_rn(F, e);                          // F + eF
    const float2 dn = __fadd2_rn(F, make_float2(-e.x, -e.y));   // F - eF
    const bool c0 = up.x < k.lo.x || dn.x > k.hi.x;
    const bool c1 = up.y < k.lo.y || dn.y > k.hi.y;
    return (c0 ? 0u : 1u) | (c1 ? 0u : 2u);
}
// Upper estimate of the nearest hit that the reference surely reports (the least
// sure_crossing_e2) among the first HT_EST_OBJECTS / 2 planes and the first HT_EST_OBJECTS / 2
// horospheres of the staged slots, +inf when none qualifies. A threshold derived from it
// (cull_from_dist) then culls before the first exact test.
// SHAPE: the slots' shape (planes come first, then horospheres), so each loop carries one
// shape's test only.
template <uint32_t SHAPE>
HT_D float est_range(const StagedScene &s, uint32_t q0, uint32_t q1, const BoundRay &r, uint32_t prev_hash, float best) {
#pragma unroll 1
    for (uint32_t q = q0; q < q1; ++q)   // warp-uniform: broadcast loads
        best = fminf(best, sure_crossing_e2(bound_fw(s.bound[q], s.mag[q], r), SHAPE, SHAPE == 0 && s.orig[q] == prev_hash, r.t));
    return best;
}
HT_D float upper_estimate(const StagedScene &s, const BoundRay &r, uint32_t prev_hash) {
    const uint32_t half = HT_EST_OBJECTS / 2, h0 = (s.n_planes + 1) & ~1u;
    float best = est_range<0>(s, 0, min(half, s.n_planes), r, prev_hash, __int_as_float(0x7f800000));
    best = est_range<1>(s, h0, min(h0 + half, s.ns), r, prev_hash, best);
    return best < __int_as_float(0x7f800000) ? dist_from_e2(best) : best;
}

// WARP: the warp pre-cull is compiled in; `full_warp` (all 32 lanes of the warp are in this
// call together, uniform across the warp) turns it on. 1: callers whose warps are nearly always
// full, the others look at every object; 2: warps that are not full take the point bound by lane.
template <int WARP = 0>
HT_D bool hop_hy(const StagedScene &s, HyPath &ray, uint32_t &rng, uint32_t &prev_hash,
                 Col &intensity, Col &emission, bool &hit, uint32_t &n_exact, bool last, bool full_warp = false) {
    // Nearest hit with ties to the lowest scene index (object/vector.inl:37-50): candidates
    // are compared on (distance, index), so the order of the slots does not matter; x =
    // cosh(distance) is compared first and the logarithm taken only when x can win; objects
    // whose distance bound rules them out are not tested.
    float min_dist = -1.0f;
    float min_x = __int_as_float(0x7f800000);   // +inf
    uint32_t kmin = 0, kmin_orig = 0xFFFFFFFFu;
    const Q4 p = ray.p, v = ray.v;
    const bool can_cull = cull_point_ok(p);
    const BoundRay br = bound_ray(p, v);
    Limit lim = limit_none(br.t);
    if (can_cull) limit_lower(lim, upper_estimate(s, br, prev_hash), br.t);   // before the first exact test
    const uint32_t h0 = (s.n_planes + 1) & ~1u;   // the first horosphere's slot
    bool warp_pre = false;
    WarpBox wb;
    if constexpr (WARP != 0) {
        if (full_warp) {
            __syncwarp();
            warp_pre = __all_sync(0xffffffffu, can_cull);
            if (warp_pre) wb = warp_box(br);
        }
    }
#pragma unroll 1
    for (uint32_t c0 = 0; c0 < s.ns; c0 += 32) {
        const uint32_t cn = min(32u, s.ns - c0);
        uint32_t valid = cn == 32 ? 0xFFFFFFFFu : (1u << cn) - 1u;
        if (s.dummy - c0 < 32u) valid &= ~(1u << (s.dummy - c0));
        uint32_t mask = valid;
        if (can_cull) {
            uint32_t m = valid;   // objects to look at one by one
            if constexpr (WARP != 0) {
                // those that the warp keeps: one object at a time for all lanes, so loads are
                // broadcasts and a shape's test runs without divergence (each lane taking its own
                // survivors of the point bound: 1080p / 200 objects, 8 passes 15.0 against 14.1 ms)
                if (warp_pre) {   // uniform: every lane can cull
                    __syncwarp();
                    m = warp_survivors(s.bound, s.mag, s.shape, c0, valid, wb, lim.kp, lim.kh);
                }
            }
            if (WARP != 1 && !warp_pre) {
                // this lane's survivors of the point bound, two slots at once
                m = 0;
                // kept rolled: the kernel is bound by instruction fetch as much as by issue
#pragma unroll 1
                for (uint32_t j = 0; j < cn; j += 2) {   // warp-uniform: broadcast loads
                    const uint32_t pq = (c0 + j) >> 1;
                    m |= survivors2(s.pa[pq], s.pb[pq], s.pmag[pq], pair_ray(br), c0 + j >= s.n_planes ? lim.kh : lim.kp) << j;
                }
                m &= valid;
            }
            mask = 0;
            while (m) {
                const uint32_t j = __ffs(m) - 1, q = c0 + j;
                m &= m - 1;
                const uint32_t shape = q >= h0 ? 1u : 0u;
                if (keep_object(s.bound[q], s.mag[q], shape, br, shape == 0 ? lim.kp : lim.kh, lim.cull)) mask |= 1u << j;
            }
        }
        while (mask) {   // this lane's candidates, in slot order
            const uint32_t q = c0 + (__ffs(mask) - 1);
            mask &= mask - 1;
            const uint32_t shape = q >= h0 ? 1u : 0u;
            if (can_cull && culled_point(s.bound[q], s.mag[q], br, shape == 0 ? lim.kp : lim.kh)) continue;
            const uint32_t k = s.orig[q];
            const bool repeat = (k == prev_hash);
            if (shape == 0 && repeat) continue;   // a geodesic plane is never hit twice in a row
            ++n_exact;
            // the out-of-line copy of the map, shared with the hit path: one copy of its code
            // (the kernel is bound by instruction fetch as much as by issue)
            HyRay l = ray_hy_map_packed(mo_from(s.inv[2 * q], s.inv[2 * q + 1]), qq(p, v));
            const float x = shape == 0 ? plane_hy_x(l.p, l.v) : horosphere_x(l.p, l.v, repeat);
            // x above the best's gives a distance no smaller (hy_dist_from_x is non-decreasing),
            // which can only win a tie, and only from a lower scene index
            if (x >= 1.0f && (x <= min_x || k < kmin_orig)) {
                const float dist = hy_dist_from_x(x);
                if (dist > -EPSF && (min_dist <= -EPSF || dist < min_dist || (dist == min_dist && k < kmin_orig))) {
                    min_dist = dist;
                    min_x = x;
                    kmin = q;
                    kmin_orig = k;
                    limit_lower(lim, dist, br.t);
                    s.win[0] = make_float4(l.p.x, l.p.y, l.p.z, l.p.w);   // kept for the hit
                    s.win[1] = make_float4(l.v.x, l.v.y, l.v.z, l.v.w);
                }
            }
        }
    }
    if (!(min_dist > -EPSF)) {
        hit = false;
        emission.x += s.background.x * intensity.x;
        emission.y += s.background.y * intensity.y;
        emission.z += s.background.z * intensity.z;
        return false;
    }
    hit = true;
    const uint8_t *obj = s.objects + (size_t)kmin_orig * OBJ_STRIDE;
    if (last) {
        mixture_last(load_material(obj), rng, intensity, emission);
        return false;
    }
    const Mo inv = mo_from(s.inv[2 * kmin], s.inv[2 * kmin + 1]);
    const Mo fwd = load_mo(obj);
    const bool repeat = (kmin_orig == prev_hash);
    HyRay l;   // the winner's local ray, as the scan computed it (the same map, the same bits)
    {
        const float4 a = s.win[0], b = s.win[1];
        l.p = q4(a.x, a.y, a.z, a.w);
        l.v = q4(b.x, b.y, b.z, b.w);
    }
    HyPath lh;
    Q4 normal;
    if (s.shape[kmin] == 0) plane_hy_hit(l.p, l.v, lh, normal);
    else horosphere_hit(l.p, l.v, repeat, lh, normal);
    HyRay w = ray_hy_map_packed(fwd, qq(lh.p, lh.v));          // detect: map back (mapped.inl:34)
    HyRay loc = ray_hy_map_packed(inv, qq(w.p, w.v));          // interact: to local (mapped.inl:46-47)
    Material m = load_material(obj);
    V3 dir = v3(loc.v.x, loc.v.y, loc.v.z);          // light_hy_to_local (light/hy.cc:3-8)
    bool ret = mixture_interact(m, rng, v3(normal.x, normal.y, normal.z), dir, intensity, emission);
    HyRay out = ray_hy_map_packed(fwd, qq(loc.p, q4(dir.x, dir.y, dir.z, 0.0f)));  // mapped.inl:49
    ray.p = out.p;
    ray.v = out.v;
    if (!ret) return false;
    prev_hash = kmin_orig;   // the hasher state after hash_usize(0, index) is the index
    return true;
}

// -------------------------------------------------------------------------- euclidean
struct EuPath { V3 p, v; };

HT_D float sphere_eu_dist(V3 pos, V3 dir, bool repeat) {   // shape/eu/sphere.cc:3-29
    float b = -dot3(dir, pos);
    V3 g = v3(pos.x + dir.x * b, pos.y + dir.y * b, pos.z + dir.z * b);
    float d = 1.0f - dot3(g, g);
    if (d < 0.0f) return -1.0f;
    d = sqrtf(d);
    float e = b - d;
    float w = repeat ? EPSF : -EPSF;
    if (e < w) {
        e = b + d;
        if (e < w) return -1.0f;
    }
    return e;
}
HT_D float plane_eu_dist(V3 pos, V3 dir) {   // shape/eu/plane.cc:3-21 (repeat handled by caller)
    if (pos.z * dir.z > 0.0f) return -1.0f;
    return -pos.z / dir.z;
}

HT_D EuPath camera_eu(const StagedScene &s, float px, float py, float size, uint32_t &rng, uint32_t flags) {
    float u0 = rng_uniform(rng);
    float u1 = rng_uniform(rng);
    float jx = (flags & FLAG_JITTER_YX) ? u1 : u0;
    float jy = (flags & FLAG_JITTER_YX) ? u0 : u1;
    float sx = px + size * (jx - 0.5f);
    float sy = py + size * (jy - 0.5f);
    V3 ld = normalize3(v3(sx, sy, -1.0f / s.fov));
    Hom cam = hom_from(s.cam0, s.cam1);
    EuPath o;
    o.v = rot3_apply(cam.rot, ld);                       // hom3_apply_dir: not normalized
    o.p = hom3_apply_pos(cam, v3(0.0f, 0.0f, 0.0f));
    return o;
}

HT_D bool hop_eu(const StagedScene &s, EuPath &ray, uint32_t &rng, uint32_t &prev_hash,
                 Col &intensity, Col &emission, bool &hit, uint32_t &n_exact, bool last) {
    // Per chunk of 32 objects: the bounds of every object (warp-uniform, broadcast loads; 20
    // instructions against 110 of an exact test), then each lane's survivors in index order, so
    // that the reference's comparison (object/vector.inl:37-50) is unchanged. 25 objects: 0.8 exact
    // tests per hop; 1917x1077, 16 passes 10.63 -> 4.91 ms (with normalize3's shared reciprocal and
    // the winner's local ray kept, which leaves three maps of the hit path instead of four).
    float min_dist = -1.0f;
    uint32_t kmin = 0;
    const V3 p = ray.p, v = ray.v;
    const EuBoundRay br = eu_bound_ray(p, v);
    float limit = __int_as_float(0x7f800000);   // +inf
    for (uint32_t c0 = 0; c0 < s.n; c0 += 32) {
        const uint32_t cn = min(32u, s.n - c0);
        uint32_t mask = cn == 32 ? 0xFFFFFFFFu : (1u << cn) - 1u;
        if (br.can) {
            mask = 0;
#pragma unroll 1
            for (uint32_t j = 0; j < cn; ++j) {
                const float4 rec = s.bound[c0 + j];
                const bool out = s.shape[c0 + j] == 0 ? eu_culled_plane(rec, br, c0 + j == prev_hash, limit)
                                                      : eu_culled_sphere(rec, br, limit);
                mask |= (out ? 0u : 1u) << j;
            }
        }
        while (mask) {
            const uint32_t k = c0 + (__ffs(mask) - 1);
            mask &= mask - 1;
            const uint32_t shape = s.shape[k];
            const bool repeat = (k == prev_hash);
            if (shape == 0 ? repeat : br.can && eu_far_sphere(s.bound[k], br, limit)) continue;
            ++n_exact;
            const EuRay l = ray_eu_map_call(hom_from(s.inv[2 * k], s.inv[2 * k + 1]), p, v);
            const float dist = shape == 0 ? plane_eu_dist(l.p, l.v) : sphere_eu_dist(l.p, l.v, repeat);
            if (dist > -EPSF && (min_dist <= -EPSF || dist < min_dist)) {
                min_dist = dist;
                kmin = k;
                limit = fminf(limit, eu_limit(dist, br));
                s.win[0] = make_float4(l.p.x, l.p.y, l.p.z, 0.0f);   // kept for the hit
                s.win[1] = make_float4(l.v.x, l.v.y, l.v.z, 0.0f);
            }
        }
    }
    if (!(min_dist > -EPSF)) {
        hit = false;
        emission.x += s.background.x * intensity.x;
        emission.y += s.background.y * intensity.y;
        emission.z += s.background.z * intensity.z;
        return false;
    }
    hit = true;
    const uint8_t *obj = s.objects + (size_t)kmin * OBJ_STRIDE;
    if (last) {
        mixture_last(load_material(obj), rng, intensity, emission);
        return false;
    }
    const Hom inv = hom_from(s.inv[2 * kmin], s.inv[2 * kmin + 1]);
    const Hom fwd = load_hom(obj);
    EuRay l;   // the winner's local ray, as the scan computed it; min_dist is its test's root
    {
        const float4 a = s.win[0], b = s.win[1];
        l.p = v3(a.x, a.y, a.z);
        l.v = v3(b.x, b.y, b.z);
    }
    const float e = min_dist;
    EuPath lh;
    V3 normal;
    lh.v = l.v;
    if (s.shape[kmin] == 0) {
        lh.p = v3(l.p.x + l.v.x * e, l.p.y + l.v.y * e, 0.0f);
        normal = v3(0.0f, 0.0f, -1.0f);
    } else {
        V3 h = normalize3(v3(l.p.x + l.v.x * e, l.p.y + l.v.y * e, l.p.z + l.v.z * e));
        lh.p = h;
        normal = h;
    }
    EuRay w = ray_eu_map_call(fwd, lh.p, lh.v);
    EuRay loc = ray_eu_map_call(inv, w.p, w.v);
    Material m = load_material(obj);
    V3 dir = loc.v;
    bool ret = mixture_interact(m, rng, normal, dir, intensity, emission);
    EuRay out = ray_eu_map_call(fwd, loc.p, dir);
    ray.p = out.p;
    ray.v = out.v;
    if (!ret) return false;
    prev_hash = kmin;
    return true;
}

}  // namespace ht
