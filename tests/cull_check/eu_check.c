/* eu_check.c -- test infrastructure: a CPU restatement of the Euclidean scan's bounds
 * (hypertrace_b200/csrc/ht_bound.cuh: eu_stage_bound, eu_bound_ray, eu_culled_sphere,
 * eu_culled_plane, eu_far_sphere) run against the full scan on every hop of sampled paths: the
 * culled scan must pick the object that the full scan picks, at the same distance. Shape tests
 * and ray maps come from the oracle's restatement of the reference (oracle/htoracle.c); in
 * adversarial mode each value that the kernel takes from a PTX approximation is pushed 2^-21
 * relative the way that culls more.
 *
 * usage: eu_check <scene bytes> <width> <height> <hops> <pixels> <global seed> <adversarial 0|1>
 * prints: hops <n> exact_per_hop <x> wrong <k> objects <n>
 */
#include "../../oracle/htoracle.c"
#include <stdio.h>

static int ADV = 0;
static float adv(float x, int dir) { return ADV ? x * (1.0f + (float)dir * 4.76837158203125e-7f) : x; }
typedef struct { float x, y, z, w; } f4;
typedef struct { vec3 p, v; float base, dh, dd; int can; } ebr_t;

static f4 eu_stage_bound(hom3 m, uint32_t shape) {
    double w = m.rot.x, x = m.rot.y, y = m.rot.z, z = m.rot.w, cx = m.shift.x, cy = m.shift.y, cz = m.shift.z;
    double c1 = fabs(cx) + fabs(cy) + fabs(cz);
    f4 nanr = {NAN, NAN, NAN, NAN};
    if (!(fabs(w * w + x * x + y * y + z * z - 1.0) <= 1e-5 && c1 <= (shape == 0 ? 250.0 : 1e4))) return nanr;
    if (shape != 0) { f4 r = {m.shift.x, m.shift.y, m.shift.z, 0.0f}; return r; }
    double nx = 2.0 * (x * z + w * y), ny = 2.0 * (y * z - w * x), nz = 1.0 - 2.0 * (x * x + y * y);
    f4 r = {(float)nx, (float)ny, (float)nz, (float)-(nx * cx + ny * cy + nz * cz)};
    return r;
}
static ebr_t eu_bound_ray(vec3 p, vec3 v) {
    ebr_t r;
    r.p = p; r.v = v;
    float p1 = fabsf(p.x) + fabsf(p.y) + fabsf(p.z);
    r.dd = fmaf(1.6e-5f, p1, 1e-3f);
    r.base = 1.0f + r.dd;
    r.dh = fmaf(8e-6f, p1, 2e-3f);
    r.can = p1 <= 1e4f && fabsf(dot3(v, v) - 1.0f) <= 2e-5f;
    return r;
}
static float eu_limit(float d, const ebr_t *r) { return fmaf(d, 1.0f + 1e-4f, r->dd); }
static int eu_culled_sphere(f4 rec, const ebr_t *r, float *limit) {
    float mx = rec.x - r->p.x, my = rec.y - r->p.y, mz = rec.z - r->p.z;
    float b = fmaf(mx, r->v.x, fmaf(my, r->v.y, mz * r->v.z));
    float mm = fmaf(mx, mx, fmaf(my, my, mz * mz));
    float q2 = fmaf(-b, b, mm), top = fmaf(1e-4f, mm, r->base);
    int out = mm > top;
    if (q2 > top || (b < 0.0f && out) || b - 1.0f > *limit) return 1;
    float s = (2.0f - top) - q2;
    if (s > 0.0f && b > 0.0f && out) *limit = fminf(*limit, eu_limit(fmaf(-(1.0f - 1e-6f), adv(sqrtf(s), +1), b), r));
    return 0;
}
static int eu_culled_plane(f4 rec, const ebr_t *r, int repeat, float *limit) {
    float h = fmaf(rec.x, r->p.x, fmaf(rec.y, r->p.y, fmaf(rec.z, r->p.z, rec.w)));
    float n = fmaf(rec.x, r->v.x, fmaf(rec.y, r->v.y, rec.z * r->v.z));
    float hlo = fabsf(h) - r->dh, an = fabsf(n);
    int ahead = (h > 0.0f) != (n > 0.0f);
    if (repeat || (hlo > 0.0f && ((!ahead && an > 2e-5f) || hlo > *limit * (an + 2e-5f)))) return 1;
    if (ahead && hlo > 0.0f && an > 0.01f)
        *limit = fminf(*limit, eu_limit((fabsf(h) + r->dh) * adv(1.0f / (an - 2e-5f), -1) * (1.0f + 1e-6f), r));
    return 0;
}
static int eu_far_sphere(f4 rec, const ebr_t *r, float limit) {
    return fmaf(rec.x - r->p.x, r->v.x, fmaf(rec.y - r->p.y, r->v.y, (rec.z - r->p.z) * r->v.z)) - 1.0f > limit;
}
static uint32_t fmix32(uint32_t h) {
    h ^= h >> 16; h *= 0x85EBCA6Bu; h ^= h >> 13; h *= 0xC2B2AE35u; h ^= h >> 16; return h;
}

int main(int argc, char **argv) {
    if (argc < 8) { fprintf(stderr, "usage\n"); return 2; }
    FILE *f = fopen(argv[1], "rb");
    if (!f) { fprintf(stderr, "scene file\n"); return 2; }
    static uint8_t buf[1 << 24];
    size_t len = fread(buf, 1, sizeof buf, f);
    fclose(f);
    uint32_t W = (uint32_t)atoi(argv[2]), H = (uint32_t)atoi(argv[3]), hops = (uint32_t)atoi(argv[4]);
    uint32_t npix = (uint32_t)atoi(argv[5]), gseed = (uint32_t)strtoul(argv[6], NULL, 10);
    ADV = atoi(argv[7]);
    scene_t sc;
    if (scene_parse(2, buf, len, 32, &sc)) { fprintf(stderr, "scene parse\n"); return 2; }
    f4 *rec = malloc(sizeof(f4) * (sc.n + 1));
    for (uint32_t k = 0; k < sc.n; ++k) rec[k] = eu_stage_bound(sc.hom[k], sc.mat[k].shape);
    long long n_hops = 0, n_exact = 0, wrong = 0;
    for (uint32_t pi = 0; pi < npix; ++pi) {
        uint32_t px = (uint32_t)(((uint64_t)pi * 2654435761u) % ((uint64_t)W * H));
        uint32_t rng = fmix32(gseed ^ fmix32(px));
        uint32_t x = px % W, y = px / W;
        R pxr = ((R)(2u * x + 1u) - (R)W) / (R)H, pyr = ((R)H - (R)(2u * y + 1u)) / (R)H, size = (R)2 / (R)H;
        R u0 = rng_uniform(&rng), u1 = rng_uniform(&rng);
        vec3 ld = normalize3(v3(pxr + size * (u0 - (R)0.5f), pyr + size * (u1 - (R)0.5f), (R)-1 / sc.fov));
        ray_eu ray;
        ray.dir = hom3_apply_dir(sc.cam_hom, ld);
        ray.start = hom3_apply_pos(sc.cam_hom, v3(0, 0, 0));
        col3 inten = {1, 1, 1}, em = {0, 0, 0};
        uint32_t prev = 0xFFFFFFFFu;
        for (uint32_t h = 0; h < hops; ++h) {
            ++n_hops;
            R min_dist = -1; uint32_t min_index = 0; ray_eu min_local = ray; vec3 min_normal = v3(0, 0, 0);
            for (uint32_t k = 0; k < sc.n; ++k) {
                int rep = (k == prev);
                ray_eu local = ray_eu_map(ray, sc.hom_inv[k]);
                vec3 nrm;
                R d = sc.mat[k].shape == 0 ? plane_eu_detect(rep, &nrm, &local) : sphere_eu_detect(rep, &nrm, &local);
                if (d > -EPS && (min_dist <= -EPS || d < min_dist)) { min_dist = d; min_index = k; min_local = local; min_normal = nrm; }
            }
            ebr_t br = eu_bound_ray(ray.start, ray.dir);
            float limit = INFINITY;
            R cd = -1; uint32_t ck = 0;
            for (uint32_t c0 = 0; c0 < sc.n; c0 += 32) {
                uint32_t cn = sc.n - c0 < 32 ? sc.n - c0 : 32, mask = 0;
                for (uint32_t j = 0; j < cn; ++j) {
                    uint32_t k = c0 + j;
                    int out = !br.can ? 0 : sc.mat[k].shape == 0 ? eu_culled_plane(rec[k], &br, k == prev, &limit)
                                                                 : eu_culled_sphere(rec[k], &br, &limit);
                    if (!out) mask |= 1u << j;
                }
                for (uint32_t j = 0; j < cn; ++j) {
                    uint32_t k = c0 + j;
                    if (!(mask >> j & 1)) continue;
                    int rep = (k == prev);
                    if (sc.mat[k].shape == 0 ? rep : br.can && eu_far_sphere(rec[k], &br, limit)) continue;
                    ++n_exact;
                    ray_eu local = ray_eu_map(ray, sc.hom_inv[k]);
                    vec3 nrm;
                    R d = sc.mat[k].shape == 0 ? plane_eu_detect(rep, &nrm, &local) : sphere_eu_detect(rep, &nrm, &local);
                    if (d > -EPS && (cd <= -EPS || d < cd)) { cd = d; ck = k; limit = fminf(limit, eu_limit((float)d, &br)); }
                }
            }
            if ((cd > -EPS) != (min_dist > -EPS) || (cd > -EPS && (cd != min_dist || ck != min_index))) ++wrong;
            if (!(min_dist > -EPS)) break;
            ray_eu hit = ray_eu_map(min_local, sc.hom[min_index]);
            ray_eu loc = ray_eu_map(hit, sc.hom_inv[min_index]);
            vec3 d3 = loc.dir;
            int ret = mixture_interact(&sc.mat[min_index], &rng, min_normal, &d3, &inten, &em);
            loc.dir = d3;
            ray = ray_eu_map(loc, sc.hom[min_index]);
            if (!ret) break;
            prev = min_index;
        }
    }
    printf("hops %lld exact_per_hop %.3f wrong %lld objects %u\n", n_hops, n_hops ? (double)n_exact / n_hops : 0.0, wrong, sc.n);
    scene_free(&sc);
    return 0;
}
