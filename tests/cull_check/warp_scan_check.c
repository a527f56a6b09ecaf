/* warp_scan_check.c -- test infrastructure: the warp pre-cull of the present hyperbolic scans
 * (hypertrace_b200/csrc/ht_bound.cuh: warp_box, warp_survivors) on the records, allowances and
 * thresholds that scan_check.c restates, checked against the lanes' own point test (keep_object).
 *
 * The kernels drop a slot for a whole warp when F over the box of the lanes' (|p|^2, x, y), widened
 * by the warp's largest error allowance and a slack of 2^-16 of the magnitudes, lies outside the loosest
 * thresholds of the warp. That changes nothing only if every lane's own test culls the slot too,
 * in float arithmetic. Both are evaluated operation by operation (build with -ffp-contract=off) on
 *   - hop 0 of tiles of 8 x 4 pixels and the later hop depths in queue order, as the wavefront, one-pass
 *     and generic kernels hold them;
 *   - the same depths sorted by direction cell, as the coherence sort leaves them;
 *   - tight warps: a ray and 31 copies whose starts differ by a few units in the last place, where
 *     the slack is all that lies between the two tests;
 * each with the thresholds of the estimate and with nearer ones, as hits leave them.
 *
 * usage: warp_scan_check <scene bytes> <width> <height> <hops> <tiles> <global seed> <slack, in units of 2^-16>
 * prints: warps <n> slots <n> culled <n> violations <n> tight_warps <n> tight_violations <n>
 */
#define main scan_check_main
#include "scan_check.c"
#undef main
#include <string.h>

static float SLACK = 0x1p-16f;

typedef struct {
    bray_t br;
    float hp, lh, hh;   /* thresholds: planes -hp / hp, horospheres lh / hh */
    int can;
    uint32_t cell;
} lane_t;
typedef struct { quat p, v; uint32_t prev; } path_t;

static void box_term(float a, float lo, float hi, float *flo, float *fhi, float *mag) {
    float p = a * lo, q = a * hi;
    *flo += fminf(p, q);
    *fhi += fmaxf(p, q);
    *mag += fmaxf(fabsf(p), fabsf(q));
}
static int warp_culls(f4 rec, float mag, uint32_t shape, const lane_t *w) {
    float r2lo = INFINITY, r2hi = -INFINITY, xlo = INFINITY, xhi = -INFINITY, ylo = INFINITY, yhi = -INFINITY;
    float K = -INFINITY, hp = -INFINITY, lh = INFINITY, hh = -INFINITY;
    for (int l = 0; l < 32; ++l) {
        r2lo = fminf(r2lo, w[l].br.r2); r2hi = fmaxf(r2hi, w[l].br.r2);
        xlo = fminf(xlo, w[l].br.x);    xhi = fmaxf(xhi, w[l].br.x);
        ylo = fminf(ylo, w[l].br.y);    yhi = fmaxf(yhi, w[l].br.y);
        K = fmaxf(K, w[l].br.K);
        hp = fmaxf(hp, w[l].hp); lh = fminf(lh, w[l].lh); hh = fmaxf(hh, w[l].hh);
    }
    float e = mag * K, flo = rec.w, fhi = rec.w, m = fabsf(rec.w);
    box_term(rec.x, r2lo, r2hi, &flo, &fhi, &m);
    box_term(rec.y, xlo, xhi, &flo, &fhi, &m);
    box_term(rec.z, ylo, yhi, &flo, &fhi, &m);
    float slack = SLACK * (m + e), lo = lh, hi = hh;
    if (shape == 0) { lo = -hp; hi = hp; }
    return ((fhi + e) + slack < lo) || ((flo - e) - slack > hi);
}
static int lane_culls(f4 rec, float mag, uint32_t shape, const lane_t *l) {
    fw_t b = bound_fw(rec, mag, &l->br);
    float lo = l->lh, hi = l->hh;
    if (shape == 0) { lo = -l->hp; hi = l->hp; }
    return (b.F + b.eF < lo) || (b.F - b.eF > hi);
}
static uint32_t dir_cell(quat v) {   /* the face that the direction points at, 4 x 4 cells of it */
    float ax = fabsf(v.x), ay = fabsf(v.y), az = fabsf(v.z), m, a, b;
    uint32_t face;
    if (ax >= ay && ax >= az) { face = v.x > 0.0f; m = ax; a = v.y; b = v.z; }
    else if (ay >= az)        { face = 2u + (v.y > 0.0f); m = ay; a = v.z; b = v.x; }
    else                      { face = 4u + (v.z > 0.0f); m = az; a = v.x; b = v.y; }
    float r = m > 0.0f ? 1.0f / m : 0.0f;
    return face * 16u + (uint32_t)fminf(fmaxf((a * r + 1.0f) * 2.0f, 0.0f), 3.0f) * 4u + (uint32_t)fminf(fmaxf((b * r + 1.0f) * 2.0f, 0.0f), 3.0f);
}
/* `nearer`: the threshold is that of a hit at this share of the estimate */
static lane_t lane_of(quat p, quat v, uint32_t prev, const staged_t *ss, const uint32_t *slot_obj, uint32_t n, uint32_t np, float nearer) {
    lane_t l;
    memset(&l, 0, sizeof l);
    l.br = bound_ray(p, v);
    l.can = cull_point_ok(p);
    l.cell = dir_cell(v);
    cull_t c = cull_none();
    if (l.can) {
        float u = upper_estimate(ss, slot_obj, n, np, &l.br, prev);
        if (u < INFINITY) c = cull_from_dist(u * nearer);
    }
    l.hp = 2.0f * l.br.t * c.S;
    l.lh = l.br.t * (1.0f / c.E);
    l.hh = l.br.t * c.E;
    return l;
}
static void check_warp(const lane_t *w, const staged_t *ss, uint32_t n, long long *slots, long long *culled, long long *violations) {
    for (int l = 0; l < 32; ++l)
        if (!w[l].can) return;   /* the kernels run the warp test only when every lane can cull */
    for (uint32_t q = 0; q < n; ++q) {
        ++*slots;
        if (!warp_culls(ss->bound[q], ss->mag[q], ss->shape[q], w)) continue;
        ++*culled;
        for (int l = 0; l < 32; ++l)
            if (!lane_culls(ss->bound[q], ss->mag[q], ss->shape[q], &w[l])) ++*violations;
    }
}
static int by_cell(const void *a, const void *b) {
    const lane_t *x = a, *y = b;
    return x->cell < y->cell ? -1 : x->cell > y->cell;
}

int main(int argc, char **argv) {
    if (argc < 8) { fprintf(stderr, "usage\n"); return 2; }
    FILE *f = fopen(argv[1], "rb");
    if (!f) { fprintf(stderr, "scene file\n"); return 2; }
    static uint8_t buf[1 << 24];
    size_t len = fread(buf, 1, sizeof buf, f);
    fclose(f);
    uint32_t W = (uint32_t)atoi(argv[2]), H = (uint32_t)atoi(argv[3]), hops = (uint32_t)atoi(argv[4]), tiles = (uint32_t)atoi(argv[5]);
    uint32_t gseed = (uint32_t)strtoul(argv[6], NULL, 10);
    SLACK = (float)atof(argv[7]) * 0x1p-16f;
    scene_t sc;
    if (scene_parse(1, buf, len, 32, &sc)) { fprintf(stderr, "scene parse\n"); return 2; }
    /* the slots: planes, then horospheres, each by distance from the camera */
    uint32_t n = sc.n, np = 0, ns = 0;
    uint32_t *slot_obj = malloc(sizeof(uint32_t) * (n + 1));
    float *key = malloc(sizeof(float) * (n + 1));
    staged_t ss = {malloc(sizeof(f4) * (n + 1)), malloc(sizeof(float) * (n + 1)), malloc(sizeof(uint32_t) * (n + 1))};
    bray_t at = bound_ray(mo_apply_q(sc.cam_mo, q4(0, 0, 1, 0)), q4(1, 0, 0, 0));
    for (uint32_t k = 0; k < n; ++k) {
        float mag, F = bound_fw(stage_bound(sc.mo[k], sc.mat[k].shape, &mag), 0.0f, &at).F / at.t;
        float d = sc.mat[k].shape == 0 ? fabsf(F) : fmaxf(F, 1.0f / F);
        key[k] = d >= 0.0f ? d : 0.0f;
        np += sc.mat[k].shape == 0;
    }
    for (uint32_t want = 0; want < 2; ++want)
        for (uint32_t k = 0; k < n; ++k)
            if (sc.mat[k].shape == want) {
                uint32_t i = ns++;
                while (i > (want ? np : 0) && key[slot_obj[i - 1]] > key[k]) { slot_obj[i] = slot_obj[i - 1]; --i; }
                slot_obj[i] = k;
            }
    for (uint32_t q = 0; q < n; ++q) {
        ss.shape[q] = sc.mat[slot_obj[q]].shape;
        ss.bound[q] = stage_bound(sc.mo[slot_obj[q]], ss.shape[q], &ss.mag[q]);
    }
    /* the queues of every hop depth */
    path_t **queue = malloc(sizeof(path_t *) * hops);
    uint32_t *count = calloc(hops, sizeof(uint32_t));
    for (uint32_t h = 0; h < hops; ++h) queue[h] = malloc(sizeof(path_t) * 32 * tiles);
    for (uint32_t i = 0; i < 32 * tiles; ++i) {
        uint32_t tile = (uint32_t)(((uint64_t)(i / 32) * 2654435761u) % ((uint64_t)(W / 8) * (H / 4)));
        uint32_t x = tile % (W / 8) * 8 + (i & 7), y = tile / (W / 8) * 4 + (i >> 3 & 3);
        uint32_t rng = fmix32(gseed ^ fmix32(y * W + x));
        R pxr = ((R)(2u * x + 1u) - (R)W) / (R)H, pyr = ((R)H - (R)(2u * y + 1u)) / (R)H, size = (R)2 / (R)H;
        R u0 = rng_uniform(&rng), u1 = rng_uniform(&rng);
        vec3 ld = normalize3(v3(pxr + size * (u0 - (R)0.5f), pyr + size * (u1 - (R)0.5f), (R)-1 / sc.fov));
        ray_hy ray;
        ray.dir = normalize4(mo_deriv_q(sc.cam_mo, q4(0, 0, 1, 0), q4(ld.x, ld.y, ld.z, 0)));
        ray.start = mo_apply_q(sc.cam_mo, q4(0, 0, 1, 0));
        col3 inten = {1, 1, 1}, em = {0, 0, 0};
        uint32_t prev = 0xFFFFFFFFu;
        for (uint32_t h = 0; h < hops; ++h) {
            path_t path = {ray.start, ray.dir, prev};
            queue[h][count[h]++] = path;
            R min_dist = -1; uint32_t min_index = 0; ray_hy min_local = ray; quat min_normal = q4(0, 0, 0, 0);
            for (uint32_t k = 0; k < n; ++k) {
                ray_hy local = ray_hy_map(ray, sc.mo_inv[k]);
                quat nrm;
                R d = sc.mat[k].shape == 0 ? plane_hy_detect(k == prev, &nrm, &local) : horosphere_detect(k == prev, &nrm, &local);
                if (d > -EPS && (min_dist <= -EPS || d < min_dist)) { min_dist = d; min_index = k; min_local = local; min_normal = nrm; }
            }
            if (!(min_dist > -EPS)) break;
            ray_hy hit = ray_hy_map(min_local, sc.mo[min_index]), loc = ray_hy_map(hit, sc.mo_inv[min_index]);
            vec3 d3 = v3(loc.dir.x, loc.dir.y, loc.dir.z), n3 = v3(min_normal.x, min_normal.y, min_normal.z);
            int ret = mixture_interact(&sc.mat[min_index], &rng, n3, &d3, &inten, &em);
            loc.dir = q4(d3.x, d3.y, d3.z, 0);
            ray = ray_hy_map(loc, sc.mo[min_index]);
            if (!ret) break;
            prev = min_index;
        }
    }
    long long warps = 0, slots = 0, culled = 0, viol = 0, twarps = 0, tslots = 0, tculled = 0, tviol = 0;
    lane_t *lanes = malloc(sizeof(lane_t) * 32 * tiles);
    for (uint32_t h = 0; h < hops; ++h)
        for (int near = 0; near < 2; ++near) {
            const uint32_t m = count[h];
            for (uint32_t i = 0; i < m; ++i)
                lanes[i] = lane_of(queue[h][i].p, queue[h][i].v, queue[h][i].prev, &ss, slot_obj, n, np, near ? 0.3f + 0.02f * (float)(i % 32) : 1.0f);
            for (int sorted = 0; sorted < (h ? 2 : 1); ++sorted) {
                if (sorted) qsort(lanes, m, sizeof(lane_t), by_cell);
                for (uint32_t i = 0; i + 32 <= m; i += 32) {
                    ++warps;
                    check_warp(lanes + i, &ss, n, &slots, &culled, &viol);
                }
            }
            for (uint32_t i = 0; i < m; i += 29) {
                lane_t w[32];
                for (int l = 0; l < 32; ++l) {
                    quat p = queue[h][i].p;
                    int kx = l % 5 - 2, ky = (l / 5) % 5 - 2, kz = (l / 25) % 3 - 1;
                    for (int k = 0; k < abs(kx); ++k) p.x = nextafterf(p.x, kx > 0 ? INFINITY : -INFINITY);
                    for (int k = 0; k < abs(ky); ++k) p.y = nextafterf(p.y, ky > 0 ? INFINITY : -INFINITY);
                    for (int k = 0; k < abs(kz); ++k) p.z = nextafterf(p.z, kz > 0 ? INFINITY : -INFINITY);
                    w[l] = lane_of(p, queue[h][i].v, queue[h][i].prev, &ss, slot_obj, n, np, near ? 0.5f : 1.0f);
                }
                /* and thresholds right at the value that the test compares, slot by slot */
                ++twarps;
                check_warp(w, &ss, n, &tslots, &tculled, &tviol);
                for (uint32_t q = 0; q < n && w[0].can; q += 3) {
                    fw_t b = bound_fw(ss.bound[q], ss.mag[q], &w[7].br);
                    staged_t one = {ss.bound + q, ss.mag + q, ss.shape + q};
                    for (int l = 0; l < 32; ++l) {
                        if (ss.shape[q] == 0) w[l].hp = fabsf(b.F) - b.eF;
                        else { w[l].lh = b.F + b.eF; w[l].hh = b.F - b.eF; }
                    }
                    check_warp(w, &one, 1, &tslots, &tculled, &tviol);
                }
            }
        }
    printf("warps %lld slots %lld culled %lld violations %lld tight_warps %lld tight_violations %lld\n", warps, slots, culled, viol, twarps, tviol);
    return 0;
}
