// htcuda.cu -- kernels and the C ABI of libhtcuda.so (declared in include/htcuda.h).
//
// Kernels:
//   render_plain<R>      one thread per pixel, one pass: the reference's `render` kernel
//                        (kernel/ocl/render/render.cl:6-27) launched over a (W,H) grid.
//   render_wave<R, FH>   one launch per hop depth of a pass (FH: hop 0 from the pixels, or a
//                        later hop from a queue of ray states); survivors are appended to
//                        the other queue with warp-aggregated atomics, so warps scan with
//                        full lanes. The form of all but small calls.
//   k_stage, k_batch_stage  the scene's staged image for these launches, once per call.
//   k_sort_*, k_bsort_*  the coherence sort of a hop depth's queue.
//   render_batch_wave<RF, FH>  the same over many views at once, one launch per pass index,
//                        hop depth and recipe, tiles of the views' queues cut on the device.
//   render_persistent<R> one launch for P passes: warps pull pixels from a queue, each lane
//                        runs its pixel's P samples in order and regenerates a finished path
//                        in place (the allocation-free entry point uses it).
//   post kernels         extract / gamma / pack (processing/src/canvas.rs:126-135,176-186,
//                        processing/src/filter/gamma.rs:10-19) and their fused form.
// Every render kernel holds the scene's inverse object maps, distance-bound records and
// shape indices in shared memory: staged by each block of the one-pass and persistent kernels,
// copied from the image by the wavefront kernels (per view change in the batched ones). Each pixel's samples take the same
// float operations in the same order in every form, so all forms give the same bits.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/htcuda.h"
#include "ht_trace.cuh"
#include "ht_host.hpp"

using namespace ht;

// ============================================================================ errors
thread_local std::string g_last_error;

// Minimum resident blocks per SM requested from ptxas for the render kernels (register cap). The
// scan is latency-bound on dependent FP32 chains, so resident warps matter, but a hyperbolic
// ray map and the scan's thresholds hold many values; Euclidean paths need far fewer.
// Measured (ms; 1080p / 200 objects, 8 passes, and 24 mixed views for the batch; Euclidean: 1917x1077,
// 25 objects, 16 passes):
//   later hops   hyperbolic 4 blocks 8.99, 5 9.11; Euclidean (hop 0 at 9) 5 4.48, 6 4.38, 7 4.48
//   hop 0        hyperbolic 5 8.91, 6 8.99, 7 9.03; Euclidean (later hops at 6) 8 4.38, 9 4.38, 10 4.51
//                (4 and 6 for the later hops and hop 0 of both geometries: 4.59)
//   batched      hyperbolic 4 34.85, 5 34.49, 6 35.9; Euclidean 5 34.6, 6 34.45, 7 34.55
//   one pass     5 and 6 alike (800x600: 384 us), 4 1 % slower
constexpr int MINB_PERSIST = 6, MINB_PLAIN = 5;
constexpr int minb_wave(bool eu, bool first) { return eu ? (first ? 9 : 6) : (first ? 5 : 4); }
constexpr int minb_batch(bool eu) { return eu ? 6 : 5; }

// Launches of one call that follow each other directly overlap at their edges (programmatic
// dependent launch). A kernel waits for the end of the one before it (wait_previous) and then lets
// the next one start (launch_next), whose blocks take the places that this one's leave, load
// the scene and wait in turn. So before its wait a kernel may read what the launch before the
// last, or anything earlier, wrote: the scene's bytes and image. And nothing that the launch before
// writes may be a `const __restrict__` argument: that promises data which no one changes while the
// kernel runs, and the kernel runs before its wait (test_overlap_qualifiers.py). 1080p / 200 objects, 8 passes:
// 10.7 -> 9.9 ms; 640x480, the same scene, unsorted: 486 -> 396 us per pass.
__device__ __forceinline__ void launch_next() { cudaTriggerProgrammaticLaunchCompletion(); }
__device__ __forceinline__ void wait_previous() { cudaGridDependencySynchronize(); }
template <class... P, class... A>
static cudaError_t launch(bool overlap, void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = st;
    cudaLaunchAttribute a = {};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &a;
    c.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

constexpr uint32_t SORT_MIN = 131072;   // paths from which on a queue of a single view is sorted

// Device error word bits.
constexpr uint32_t ERR_SCENE = 1u;
constexpr uint32_t ERR_SMEM = 2u;

struct htc_program {
    int recipe;
    uint32_t hops;
    int address_width;
    uint32_t flags;
    uint32_t *d_err;     // device error word
    int num_sms;
    int max_smem;
    GenericProgram *generic;   // scene types served by render_generic (htgeneric.cu), else NULL
    void *wave_buf;            // two wavefront queues (WAVE_SLOT_BYTES per slot each), grown on demand
    size_t wave_slots;         // slots per queue
    uint32_t *d_wave_ctr;      // 2 counters per hop depth, two sets
    void *sort_buf;            // coherence sort of the hyperbolic queues (SortBuf), as many slots as they have
    float4 *image;             // the scene's image (stage_image), of the largest that can be staged
    int device;                // whose pool it uses (render_wave_pooled); -1: none
    int double_support;        // scene bytes in the double_support layout, narrowed before rendering
    uint8_t *narrow_buf;       // the narrowed (f32 layout) scene, grown on demand
    size_t narrow_bytes;
    std::mutex narrow_mutex;   // from a call's narrowing to its last launch
    cudaEvent_t narrow_done;   // the last call's use of narrow_buf
};

// ============================================================================ staging
// Loads the scene header and the per-object data the scan reads into shared memory. Returns
// false (uniformly across the block) when the scene bytes fail validation.
//
// Hyperbolic scenes are staged in scan order, geodesic planes first, then horospheres, each by
// their distance from the camera (scenes of 7 to STAGE_SORT_MAX objects; index order for fewer, where the
// order gains nothing and its keys cost 3 objects at 1024x700 66 -> 71 us a pass, and beyond):
// the paths of a view stay near it, so the first few slots of a shape nearly always hold a sure
// crossing close to the winner's (upper_estimate), and the later chunks fall to the warp
// pre-cull. When the plane count is odd a dummy slot follows the planes,
// so that every pair of slots (2p, 2p + 1) holds one shape and the point-bound loop can test
// two objects per packed FP32 instruction. `orig[slot]` is the object's index in the scene:
// the scan compares hits on (distance, index), the reference's nearest-hit rule
// (object/vector.inl:37-50), so the order of the slots never changes the winner. Euclidean
// scenes are staged in index order (slot = index).
//
// Shared-memory layout for up to n objects (n + 1 slots, smem_bytes(n) bytes): inverse maps
// (2 float4 per slot), bound records (float4), the bound records again as pairs of slots
// ({x0, x1, y0, y1}, {z0, z1, w0, w1} per pair) and their magnitudes ({m0, m1}), then shape,
// bound magnitude and scene index per slot (u32 / f32 / u32), then 2 float4 per thread of a
// 128-thread block (the scan's winner, local frame).
constexpr uint32_t BLOCK_THREADS = 128;
constexpr uint32_t STAGE_SORT_MAX = 2 * BLOCK_THREADS * 4;   // words of the winners' slots, the sort's scratch
struct SceneSmem {
    float4 *inv, *bound, *pa, *pb;
    float2 *pmag;
    uint32_t *shape, *orig;
    float *mag;
    float4 *win;
    float4 *end;   // first float4 past the layout
};
__host__ __device__ constexpr uint32_t scene_slots(uint32_t n) { return n + 1; }
__host__ __device__ constexpr size_t scene_win_offset(uint32_t n) {
    return ((size_t)scene_slots(n) * 60u + (size_t)((scene_slots(n) + 1) / 2) * 40u + 15u) & ~(size_t)15u;
}
__device__ __forceinline__ SceneSmem carve_scene(float4 *smem, uint32_t n) {
    const uint32_t ns = scene_slots(n), np = (ns + 1) / 2;
    SceneSmem c;
    c.inv = smem;
    c.bound = c.inv + 2 * ns;
    c.pa = c.bound + ns;
    c.pb = c.pa + np;
    c.pmag = reinterpret_cast<float2 *>(c.pb + np);
    c.shape = reinterpret_cast<uint32_t *>(c.pmag + np);
    c.mag = reinterpret_cast<float *>(c.shape + ns);
    c.orig = reinterpret_cast<uint32_t *>(c.mag + ns);
    c.win = smem + scene_win_offset(n) / 16;
    c.end = c.win + 2 * BLOCK_THREADS;
    return c;
}

// Stages object k (shape `shape`) into slot q.
template <int R>
__device__ __forceinline__ void stage_object(const uint8_t *obj, uint32_t shape, uint32_t k, uint32_t q,
                                             const SceneSmem &sm) {
    sm.shape[q] = shape;
    sm.orig[q] = k;
    float4 rec = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float mag = 0.0f;
    if (R == RECIPE_HY) {
        const Mo fwd = load_mo(obj);
        Mo inv = mo_inverse(fwd);
        sm.inv[2 * q] = make_float4(inv.a.x, inv.a.y, inv.b.x, inv.b.y);
        sm.inv[2 * q + 1] = make_float4(inv.c.x, inv.c.y, inv.d.x, inv.d.y);
        rec = stage_bound(fwd, shape, mag);
    } else {
        const Hom fwd = load_hom(obj);
        const Hom inv = hom3_inverse(fwd);
        rec = eu_stage_bound(fwd, shape);
        sm.inv[2 * q] = make_float4(inv.shift.x, inv.shift.y, inv.shift.z, 0.0f);
        sm.inv[2 * q + 1] = make_float4(inv.rot.x, inv.rot.y, inv.rot.z, inv.rot.w);
    }
    sm.bound[q] = rec;
    sm.mag[q] = mag;
    float *pa = reinterpret_cast<float *>(&sm.pa[q >> 1]), *pb = reinterpret_cast<float *>(&sm.pb[q >> 1]);
    const uint32_t o = q & 1u;
    pa[o] = rec.x; pa[2 + o] = rec.y; pb[o] = rec.z; pb[2 + o] = rec.w;
    reinterpret_cast<float *>(&sm.pmag[q >> 1])[o] = mag;
}

// The rest of a staged scene whose counts are set.
template <int R>
__device__ __forceinline__ void staged_scene(const uint8_t *scene, StagedScene &s, const SceneSmem &sm, uint32_t tid) {
    using L = Layout<R>;
    s.inv = sm.inv;
    s.bound = sm.bound;
    s.pa = sm.pa;
    s.pb = sm.pb;
    s.pmag = sm.pmag;
    s.shape = sm.shape;
    s.mag = sm.mag;
    s.orig = sm.orig;
    s.win = sm.win + 2 * tid;
    s.objects = scene + L::OBJECTS;
    s.ns = s.n + (s.dummy != 0xFFFFFFFFu ? 1u : 0u);
    s.fov = ldf(scene, L::FOV);
    const float4 bg = ldf4(scene, L::BG);
    s.background.x = bg.x; s.background.y = bg.y; s.background.z = bg.z;
    s.cam0 = ldf4(scene, 0);
    s.cam1 = ldf4(scene, 16);
}
template <int R>
__device__ bool stage_scene(const uint8_t *scene, size_t scene_size, uint32_t max_objects,
                            int address_width, uint32_t *err, StagedScene &s, const SceneSmem &sm,
                            uint32_t *s_hdr) {
    using L = Layout<R>;
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        uint32_t ok = 1;
        uint32_t n = 0;
        if (scene_size < L::OBJECTS) ok = 0;
        if (ok) {
            n = ldu(scene, L::COUNT);
            if (address_width == 64 && ldu(scene, L::COUNT + 4) != 0) ok = 0;
            if ((scene_size - L::OBJECTS) / OBJ_STRIDE < n) ok = 0;
            if (n > max_objects) ok = 0;
        }
        s_hdr[0] = ok;
        s_hdr[1] = n;
    }
    __syncthreads();
    const uint32_t n = s_hdr[1];
    const bool header_ok = s_hdr[0] != 0;
    __syncthreads();
    if (!header_ok) {
        if (threadIdx.x == 0 && threadIdx.y == 0) atomicOr(err, ERR_SCENE);
        return false;
    }
    const uint32_t tid = threadIdx.x + blockDim.x * threadIdx.y;
    const uint32_t nthreads = blockDim.x * blockDim.y;
    const uint8_t *objects = scene + L::OBJECTS;
    bool bad = false;
    uint32_t n_planes = 0, dummy = 0xFFFFFFFFu;
    if (R == RECIPE_HY) {
        // pass 1: the number of planes, and every object's sort key (shape, distance from the
        // camera; both shapes' distances grow with |F| or max(F, 1 / F) of the bound record)
        uint32_t *keys = reinterpret_cast<uint32_t *>(sm.win);
        // (up to HT_EST_OBJECTS / 2 objects the estimate looks at all of them, whatever their order)
        const bool by_distance = n > HT_EST_OBJECTS / 2 && n <= STAGE_SORT_MAX;
        const Q4 cam = mo_apply_pos(load_mo(scene), q4(0.0f, 0.0f, 1.0f, 0.0f));
        const BoundRay at = bound_ray(cam, q4(1.0f, 0.0f, 0.0f, 0.0f));
        for (uint32_t r0 = 0; r0 < n; r0 += nthreads) {
            const uint32_t k = r0 + tid;
            const uint8_t *obj = objects + (size_t)k * OBJ_STRIDE;
            const uint32_t shape = k < n ? ldu(obj, O_SHAPE) : 1u;
            if (by_distance && k < n) {
                float mag;
                const float F = bound_fw(stage_bound(load_mo(obj), min(shape, 1u), mag), 0.0f, at).F / at.t;
                const float d = shape == 0 ? fabsf(F) : fmaxf(F, 1.0f / F);
                keys[k] = (shape == 0 ? 0u : 0x80000000u) | (d >= 0.0f ? __float_as_uint(d) : 0u);   // NaN records first
            }
            n_planes += (uint32_t)__syncthreads_count(shape == 0 ? 1 : 0);
        }
        // pass 2: slot = rank among the keys (ties by index); horospheres start at an even slot.
        // Beyond the sort: rank among the planes, from a ballot per warp and the warps' counts in
        // s_hdr[2..], or among the horospheres
        const uint32_t gap = n_planes & 1u, h0 = n_planes + gap;
        const uint32_t lane = tid & 31u, warp = tid >> 5, nwarps = (nthreads + 31) >> 5;
        uint32_t before = 0;   // planes among the objects before this block-wide step
        for (uint32_t r0 = 0; r0 < n; r0 += nthreads) {
            const uint32_t k = r0 + tid;
            const bool in = k < n;
            const uint8_t *obj = objects + (size_t)k * OBJ_STRIDE;
            const uint32_t shape = in ? ldu(obj, O_SHAPE) : 1u;
            uint32_t slot = 0;
            if (by_distance) {
                const uint32_t mine = in ? keys[k] : 0u;
                for (uint32_t j = 0; j < n; ++j) {   // broadcast loads
                    const uint32_t other = keys[j];
                    slot += other < mine || (other == mine && j < k) ? 1u : 0u;
                }
                slot += shape == 0 ? 0u : gap;
            } else {
                const uint32_t ballot = __ballot_sync(0xffffffffu, in && shape == 0);
                if (lane == 0) s_hdr[2 + warp] = (uint32_t)__popc(ballot);
                __syncthreads();
                uint32_t rank = before + (uint32_t)__popc(ballot & ((1u << lane) - 1u)), total = 0;
                for (uint32_t w = 0; w < nwarps; ++w) {
                    const uint32_t c = s_hdr[2 + w];
                    if (w < warp) rank += c;
                    total += c;
                }
                __syncthreads();
                before += total;
                slot = shape == 0 ? rank : h0 + (k - rank);
            }
            if (in) {
                if (address_width == 64 && ldu(obj, O_SHAPE + 4) != 0) bad = true;
                if (shape > 1) bad = true;
                stage_object<R>(obj, shape > 1 ? 1u : shape, k, slot, sm);
            }
        }
        if (n_planes & 1u) {   // the dummy slot: never a candidate (masked), NaN bound record
            dummy = n_planes;
            if (tid == 0) {
                const float nan = __int_as_float(0x7fc00000);
                sm.shape[dummy] = 0;
                sm.orig[dummy] = 0xFFFFFFFFu;
                sm.bound[dummy] = make_float4(nan, nan, nan, nan);
                sm.mag[dummy] = 0.0f;
                float *pa = reinterpret_cast<float *>(&sm.pa[dummy >> 1]), *pb = reinterpret_cast<float *>(&sm.pb[dummy >> 1]);
                pa[1] = 0.0f; pa[3] = 0.0f; pb[1] = 0.0f; pb[3] = 0.0f;   // the odd half of its pair
                reinterpret_cast<float *>(&sm.pmag[dummy >> 1])[1] = 0.0f;
            }
        }
    } else {
        for (uint32_t k = tid; k < n; k += nthreads) {
            const uint8_t *obj = objects + (size_t)k * OBJ_STRIDE;
            const uint32_t shape = ldu(obj, O_SHAPE);
            if (address_width == 64 && ldu(obj, O_SHAPE + 4) != 0) bad = true;
            if (shape > 1) bad = true;
            stage_object<R>(obj, shape > 1 ? 1u : shape, k, k, sm);
        }
    }
    const int any_bad = __syncthreads_or(bad ? 1 : 0);
    if (any_bad) {
        if (tid == 0) atomicOr(err, ERR_SCENE);
        return false;
    }
    s.n = n;
    s.n_planes = R == RECIPE_HY ? n_planes : 0u;
    s.dummy = dummy;
    staged_scene<R>(scene, s, sm, tid);
    return true;
}

// The staged layout of one scene in global memory, made once per call: a header {valid, objects,
// planes, dummy slot}, then carve_scene's arrays for `max_objects` objects (without the winners'
// slots). The wavefront kernels copy it into shared memory instead of staging the scene in every
// block of every launch, and carry no staging code.
constexpr uint32_t STAGE_THREADS = 256;
__host__ __device__ constexpr size_t image_words(uint32_t max_objects) { return 1 + scene_win_offset(max_objects) / 16; }   // float4
template <int R>
__device__ __forceinline__ void stage_image(const uint8_t *scene, size_t scene_size, uint32_t max_objects,
                                            int address_width, uint32_t *err, float4 *image) {
    __shared__ uint32_t s_hdr[2 + STAGE_THREADS / 32];
    __shared__ float4 s_sort[2 * BLOCK_THREADS];
    SceneSmem sm = carve_scene(image + 1, max_objects);
    sm.win = s_sort;
    StagedScene s;
    s.n = s.n_planes = 0;
    s.dummy = 0xFFFFFFFFu;
    const bool ok = stage_scene<R>(scene, scene_size, max_objects, address_width, err, s, sm, s_hdr);
    if (threadIdx.x == 0) *reinterpret_cast<uint4 *>(image) = make_uint4(ok ? 1u : 0u, s.n, s.n_planes, s.dummy);
}
template <int R>
__global__ void __launch_bounds__(STAGE_THREADS) k_stage(const uint8_t *__restrict__ scene, size_t scene_size,
                                                        uint32_t max_objects, int address_width, uint32_t *err, float4 *image) {
    stage_image<R>(scene, scene_size, max_objects, address_width, err, image);
}
// The whole block; false when the scene failed validation.
template <int R>
__device__ __forceinline__ bool load_scene(const float4 *image, const uint8_t *scene, uint32_t max_objects,
                                           StagedScene &s, const SceneSmem &sm) {
    const uint4 hdr = *reinterpret_cast<const uint4 *>(image);
    if (!hdr.x) return false;
    const uint32_t words = (uint32_t)(scene_win_offset(max_objects) / 16);
    for (uint32_t i = threadIdx.x; i < words; i += BLOCK_THREADS) sm.inv[i] = image[1 + i];   // sm.inv: the first array
    s.n = hdr.y;
    s.n_planes = hdr.z;
    s.dummy = hdr.w;
    staged_scene<R>(scene, s, sm, threadIdx.x);
    __syncthreads();
    return true;
}

template <int R> struct PathOf;
template <> struct PathOf<RECIPE_HY> { using T = HyPath; };
template <> struct PathOf<RECIPE_EU> { using T = EuPath; };

template <int R>
__device__ __forceinline__ typename PathOf<R>::T camera(const StagedScene &s, float px, float py,
                                                        float size, uint32_t &rng, uint32_t flags) {
    if constexpr (R == RECIPE_HY) return camera_hy(s, px, py, size, rng, flags);
    else return camera_eu(s, px, py, size, rng, flags);
}
// WARP / full_warp: the hyperbolic scan's warp pre-cull (hop_hy), for callers whose warps enter
// together (1) or may (2).
template <int R, int WARP = 0>
__device__ __forceinline__ bool hop(const StagedScene &s, typename PathOf<R>::T &ray, uint32_t &rng,
                                    uint32_t &prev_hash, Col &intensity, Col &emission, bool &hit,
                                    uint32_t &n_exact, bool last, bool full_warp = false) {
    if constexpr (R == RECIPE_HY)
        return hop_hy<WARP>(s, ray, rng, prev_hash, intensity, emission, hit, n_exact, last, full_warp);
    else return hop_eu(s, ray, rng, prev_hash, intensity, emission, hit, n_exact, last);
}

// Pixel centre and size (render.cl:12-18).
__device__ __forceinline__ void pixel_pos(uint32_t x, uint32_t y, uint32_t W, uint32_t H, float &px,
                                          float &py, float &size) {
    px = (__uint2float_rn(2u * x + 1u) - __uint2float_rn(W)) / __uint2float_rn(H);
    py = (__uint2float_rn(H) - __uint2float_rn(2u * y + 1u)) / __uint2float_rn(H);
    size = 2.0f / __uint2float_rn(H);
}

__device__ __forceinline__ void flush_stats(uint64_t *stats, uint32_t samples32, uint32_t hops32,
                                            uint32_t hits32, uint32_t exact32, uint32_t n_objects) {
    if (!stats) return;
    uint64_t samples = samples32, hops = hops32, hits = hits32, exact = exact32;
    for (int off = 16; off > 0; off >>= 1) {
        samples += __shfl_down_sync(0xffffffffu, samples, off);
        hops += __shfl_down_sync(0xffffffffu, hops, off);
        hits += __shfl_down_sync(0xffffffffu, hits, off);
        exact += __shfl_down_sync(0xffffffffu, exact, off);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd((unsigned long long *)&stats[HTC_STAT_SAMPLES], (unsigned long long)samples);
        atomicAdd((unsigned long long *)&stats[HTC_STAT_HOPS], (unsigned long long)hops);
        atomicAdd((unsigned long long *)&stats[HTC_STAT_OBJECT_TESTS], (unsigned long long)(hops * n_objects));
        atomicAdd((unsigned long long *)&stats[HTC_STAT_HITS], (unsigned long long)hits);
        atomicAdd((unsigned long long *)&stats[HTC_STAT_EXACT_TESTS], (unsigned long long)exact);
    }
}

// ============================================================================ plain
template <int R>
__global__ void __launch_bounds__(128, MINB_PLAIN) render_plain(
    const uint8_t *__restrict__ scene, size_t scene_size, uint32_t max_objects, int address_width,
    uint32_t W, uint32_t H, uint32_t hops, uint32_t flags, float4 *__restrict__ canvas,
    uint32_t *__restrict__ seeds, uint64_t *stats, uint32_t *err) {
    extern __shared__ float4 smem[];
    __shared__ uint32_t s_hdr[2 + BLOCK_THREADS / 32];
    const SceneSmem sm = carve_scene(smem, max_objects);
    StagedScene s;
    if (!stage_scene<R>(scene, scene_size, max_objects, address_width, err, s, sm, s_hdr)) return;

    // 128 threads = 32 x 4 pixels, 8 x 4 a warp, whose rays stay close together: the scan takes the
    // warp's own bound first while no lane's path has ended (320x240, one pass, 77 and 200 objects 184 and
    // 213 us -> 177 and 199; 400x300 227 and 292 -> 217 and 268).
    const uint32_t x = blockIdx.x * 32 + (threadIdx.x >> 5) * 8 + (threadIdx.x & 7);
    const uint32_t y = blockIdx.y * 4 + (threadIdx.x >> 3 & 3);
    const bool inside = x < W && y < H;
    uint32_t n_samples = 0, n_hops = 0, n_hits = 0, n_exact = 0;
    if (inside) {
        const uint32_t idx = x + W * y;
        float px, py, size;
        pixel_pos(x, y, W, H, px, py, size);
        uint32_t rng = seeds[idx];
        auto ray = camera<R>(s, px, py, size, rng, flags);
        Col intensity = {1.0f, 1.0f, 1.0f};
        Col emission = {0.0f, 0.0f, 0.0f};
        uint32_t prev_hash = HASH_NEVER;
        for (uint32_t i = 0; i < hops; ++i) {
            bool hit;
            n_hops += 1;
            bool go = hop<R, 2>(s, ray, rng, prev_hash, intensity, emission, hit, n_exact, i + 1 == hops, __activemask() == 0xffffffffu);
            n_hits += hit ? 1 : 0;
            if (!go) break;
        }
        n_samples = 1;
        float4 c = canvas[idx];
        c.x += emission.x; c.y += emission.y; c.z += emission.z; c.w += 1.0f;
        canvas[idx] = c;
        seeds[idx] = rng;
    }
    flush_stats(stats, n_samples, n_hops, n_hits, n_exact, s.n);
}

// ============================================================================ persistent
constexpr uint32_t NO_PIXEL = 0xFFFFFFFFu;

// Counters of one thread, flushed once per launch.
struct LaneStats {
    uint32_t samples = 0, hops = 0, hits = 0, exact = 0;
    uint64_t tests = 0;   // object tests the reference makes (hops x objects)
};

__device__ __forceinline__ void flush_lane_stats(uint64_t *stats, const LaneStats &st) {
    if (!stats) return;
    uint64_t samples = st.samples, hops = st.hops, hits = st.hits, exact = st.exact, tests = st.tests;
    for (int off = 16; off > 0; off >>= 1) {
        samples += __shfl_down_sync(0xffffffffu, samples, off);
        hops += __shfl_down_sync(0xffffffffu, hops, off);
        hits += __shfl_down_sync(0xffffffffu, hits, off);
        exact += __shfl_down_sync(0xffffffffu, exact, off);
        tests += __shfl_down_sync(0xffffffffu, tests, off);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd((unsigned long long *)&stats[HTC_STAT_SAMPLES], (unsigned long long)samples);
        atomicAdd((unsigned long long *)&stats[HTC_STAT_HOPS], (unsigned long long)hops);
        atomicAdd((unsigned long long *)&stats[HTC_STAT_OBJECT_TESTS], (unsigned long long)tests);
        atomicAdd((unsigned long long *)&stats[HTC_STAT_HITS], (unsigned long long)hits);
        atomicAdd((unsigned long long *)&stats[HTC_STAT_EXACT_TESTS], (unsigned long long)exact);
    }
}

// The persistent lane loop of render_persistent: warps take pixel
// indices [first, first + count) from `*counter` (global or shared memory) with one atomic
// per warp; each lane renders its pixel's `passes` samples in order and regenerates a camera
// ray as soon as a path ends. Returns when the warp has no pixel left.
template <int R>
__device__ __forceinline__ void trace_pixels(const StagedScene &s, uint32_t *counter, uint32_t first,
                                             uint32_t count, uint32_t W, uint32_t H, uint32_t hops,
                                             uint32_t passes, uint32_t flags, float4 *__restrict__ canvas,
                                             uint32_t *__restrict__ seeds, LaneStats &st) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t pixel = NO_PIXEL;
    bool done = passes == 0;
    uint32_t pass = 0, rng = 0, prev_hash = HASH_NEVER, hop_i = 0;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float px = 0.f, py = 0.f, size = 0.f;
    typename PathOf<R>::T ray;
    Col intensity = {1.0f, 1.0f, 1.0f};
    Col emission = {0.0f, 0.0f, 0.0f};
    bool in_path = false;

    for (;;) {
        // Lanes without a pixel take the next ones from the counter: one atomic per warp.
        const bool need = !done && pixel == NO_PIXEL;
        const uint32_t mask = __ballot_sync(0xffffffffu, need);
        if (mask) {
            uint32_t base = 0;
            const int leader = __ffs(mask) - 1;
            if (lane == (uint32_t)leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (need) {
                const uint32_t mine = base + __popc(mask & ((1u << lane) - 1u));
                if (mine < count) {
                    pixel = first + mine;
                    const uint32_t x = pixel % W, y = pixel / W;
                    pixel_pos(x, y, W, H, px, py, size);
                    rng = seeds[pixel];
                    acc = canvas[pixel];
                    pass = 0;
                    in_path = false;
                } else {
                    done = true;
                }
            }
        }
        if (__all_sync(0xffffffffu, done)) break;
        if (pixel != NO_PIXEL && !in_path) {
            ray = camera<R>(s, px, py, size, rng, flags);
            intensity.x = intensity.y = intensity.z = 1.0f;
            emission.x = emission.y = emission.z = 0.0f;
            prev_hash = HASH_NEVER;
            hop_i = 0;
            in_path = true;
        }
        if (in_path) {
            bool hit;
            st.hops += 1;
            bool go = hop<R>(s, ray, rng, prev_hash, intensity, emission, hit, st.exact, hop_i + 1 >= hops);
            st.hits += hit ? 1 : 0;
            hop_i += 1;
            if (!go || hop_i >= hops) {
                acc.x += emission.x; acc.y += emission.y; acc.z += emission.z; acc.w += 1.0f;
                st.samples += 1;
                in_path = false;
                pass += 1;
                if (pass >= passes) {
                    canvas[pixel] = acc;
                    seeds[pixel] = rng;
                    pixel = NO_PIXEL;
                }
            }
        }
    }
}

// The last block to finish rewinds the launch's queue words for the next launch.
__device__ __forceinline__ void rewind_queue(uint32_t *queue) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const uint32_t finished = atomicAdd(&queue[1], 1u);
        if (finished == gridDim.x - 1) {
            queue[0] = 0;
            queue[1] = 0;
            __threadfence();
        }
    }
}

template <int R>
__global__ void __launch_bounds__(128, MINB_PERSIST) render_persistent(
    const uint8_t *__restrict__ scene, size_t scene_size, uint32_t max_objects, int address_width,
    uint32_t W, uint32_t H, uint32_t hops, uint32_t passes, uint32_t flags,
    float4 *__restrict__ canvas, uint32_t *__restrict__ seeds, uint64_t *stats, uint32_t *err,
    uint32_t *queue) {
    extern __shared__ float4 smem[];
    __shared__ uint32_t s_hdr[2 + BLOCK_THREADS / 32];
    const SceneSmem sm = carve_scene(smem, max_objects);
    StagedScene s;
    const bool staged = stage_scene<R>(scene, scene_size, max_objects, address_width, err, s, sm, s_hdr);
    LaneStats st;
    if (staged) trace_pixels<R>(s, &queue[0], 0, W * H, W, H, hops, passes, flags, canvas, seeds, st);
    flush_stats(stats, st.samples, st.hops, st.hits, st.exact, staged ? s.n : 0);
    rewind_queue(queue);
}

// ============================================================================ wavefront
// One launch per hop depth. Launch h takes the paths that are still going after h hops
// from a queue, runs one hop on each and appends the survivors to the other queue; paths
// that end add their sample to the canvas right there. Hop 0 starts from the pixels
// (camera ray, no queue read). Warps take 32 queue slots at a time from a counter and
// append survivors with one atomic per warp, order kept within the warp, so a warp's
// lanes stay paths that started at neighbouring pixels and ran the same number of hops:
// no lane idles on a finished path while its warp scans, which is where the one-pass
// kernel loses a third of its lanes. The hop itself is `hop<R>` unchanged, so the result
// is bit-identical to render_plain.
struct WaveQueue {      // ray state, structure of arrays (one float4 load / store each)
    float4 *p;          // ray start
    float4 *v;          // ray direction
    float4 *t;          // intensity xyz, RNG state (bits) in w
    float4 *e;          // emission xyz, pixel index (bits) in w
    uint32_t *h;        // previous hit hash
    const uint32_t *o;  // read order: lane i of a hop takes slot o[i] (NULL: slot i)
};
constexpr size_t WAVE_SLOT_BYTES = 4 * sizeof(float4) + sizeof(uint32_t);

template <int R> __device__ __forceinline__ void path_store(float4 *p, float4 *v, const typename PathOf<R>::T &r) {
    if constexpr (R == RECIPE_HY) {
        *p = make_float4(r.p.x, r.p.y, r.p.z, r.p.w);
        *v = make_float4(r.v.x, r.v.y, r.v.z, r.v.w);
    } else {
        *p = make_float4(r.p.x, r.p.y, r.p.z, 0.0f);
        *v = make_float4(r.v.x, r.v.y, r.v.z, 0.0f);
    }
}
template <int R> __device__ __forceinline__ typename PathOf<R>::T path_load(float4 p, float4 v) {
    typename PathOf<R>::T r;
    if constexpr (R == RECIPE_HY) {
        r.p = q4(p.x, p.y, p.z, p.w);
        r.v = q4(v.x, v.y, v.z, v.w);
    } else {
        r.p = v3(p.x, p.y, p.z);
        r.v = v3(v.x, v.y, v.z);
    }
    return r;
}

__host__ __device__ inline WaveQueue wave_at(const WaveQueue &q, uint64_t off) {
    WaveQueue r;
    r.p = q.p ? q.p + off : nullptr;
    r.v = q.v ? q.v + off : nullptr;
    r.t = q.t ? q.t + off : nullptr;
    r.e = q.e ? q.e + off : nullptr;
    r.h = q.h ? q.h + off : nullptr;
    r.o = q.o ? q.o + off : nullptr;
    return r;
}

// Hop 0's slots are the pixels by tiles of 8 x 4, one warp's: their rays stay closer together than
// those of 32 pixels of a row, so the warp pre-cull keeps fewer objects, and the next queue is
// laid out the same way (24 mixed views batched 36.2 -> 35.7 ms, 800x600 64 passes 18.6 -> 18.4). The
// strips that whole tiles leave at the right and at the bottom follow row by row, so no chunk but the
// last has idle lanes (tiles cut off at the edge cost 637x359 1 %: 1.345 -> 1.357 ms).
__device__ __forceinline__ void first_pixel(uint32_t slot, uint32_t W, uint32_t H, uint32_t &x, uint32_t &y) {
    const uint32_t across = W / 8, tiles = across * (H / 4), rows = H & ~3u;
    const uint32_t tile = slot / 32;
    if (tile < tiles) {
        x = tile % across * 8 + (slot & 7);
        y = tile / across * 4 + (slot >> 3 & 3);
        return;
    }
    slot -= tiles * 32;
    const uint32_t strip = W & 7, right = strip * rows;
    if (slot < right) {
        x = (W & ~7u) + slot % strip;
        y = slot / strip;
    } else {
        x = (slot - right) % W;
        y = rows + (slot - right) / W;
    }
}

// One hop for the 32 queue slots [base, base + 32) of a warp (slots >= n idle): on hop 0 a
// slot stands for a pixel (camera ray from its seed), later for a path read from `in`. Paths that go on
// are appended to `out` with one atomic on `out_count` per warp; paths that end add their
// sample to the canvas (render.cl:20-26). Every lane of the warp calls this together.
// FH: 1 = hop 0 (pixels), 2 = a later hop (queue), known at compile time so that each
// kernel carries only its own half (the kernel is bound by instruction fetch as much as by
// issue).
template <int R, int FH>
__device__ __forceinline__ void wave_chunk(const StagedScene &s, uint32_t base, uint32_t n, bool last_hop,
                                           uint32_t W, uint32_t H, uint32_t flags,
                                           float4 *__restrict__ canvas, uint32_t *__restrict__ seeds,
                                           const WaveQueue &in, const WaveQueue &out, uint32_t *out_count,
                                           LaneStats &st) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t i = base + lane;
    bool cont = false;
    typename PathOf<R>::T ray;
    uint32_t rng = 0, prev_hash = HASH_NEVER, pixel = 0;
    Col intensity = {1.0f, 1.0f, 1.0f};
    Col emission = {0.0f, 0.0f, 0.0f};
    constexpr bool first = FH == 1;
    const bool full_warp = __ballot_sync(0xffffffffu, i < n) == 0xffffffffu;   // every lane has a path
    if (i < n) {
        if (first) {
            uint32_t x, y;
            first_pixel(i, W, H, x, y);
            pixel = y * W + x;
            float px, py, size;
            pixel_pos(x, y, W, H, px, py, size);
            rng = seeds[pixel];
            ray = camera<R>(s, px, py, size, rng, flags);
        } else {
            const uint32_t k = in.o ? in.o[i] : i;
            ray = path_load<R>(in.p[k], in.v[k]);
            const float4 t = in.t[k], e = in.e[k];
            intensity.x = t.x; intensity.y = t.y; intensity.z = t.z;
            rng = __float_as_uint(t.w);
            emission.x = e.x; emission.y = e.y; emission.z = e.z;
            pixel = __float_as_uint(e.w);
            prev_hash = in.h[k];
        }
        bool hit;
        st.hops += 1;
        st.tests += s.n;
        const bool go = hop<R, 1>(s, ray, rng, prev_hash, intensity, emission, hit, st.exact, last_hop, full_warp);
        st.hits += hit ? 1 : 0;
        cont = go;
        if (!cont) {
            st.samples += 1;
            float4 c = canvas[pixel];
            c.x += emission.x; c.y += emission.y; c.z += emission.z; c.w += 1.0f;
            canvas[pixel] = c;
            seeds[pixel] = rng;
        }
    }
    const uint32_t want = __ballot_sync(0xffffffffu, cont);
    if (want) {
        const int leader = __ffs(want) - 1;
        uint32_t obase = 0;
        if (lane == (uint32_t)leader) obase = atomicAdd(out_count, (uint32_t)__popc(want));
        obase = __shfl_sync(0xffffffffu, obase, leader);
        if (cont) {
            const uint32_t j = obase + __popc(want & ((1u << lane) - 1u));
            path_store<R>(&out.p[j], &out.v[j], ray);
            out.t[j] = make_float4(intensity.x, intensity.y, intensity.z, __uint_as_float(rng));
            out.e[j] = make_float4(emission.x, emission.y, emission.z, __uint_as_float(pixel));
            out.h[j] = prev_hash;
        }
    }
}

// ctr[0]: slots taken by warps of this launch; ctr[1]: paths appended to `out`.
// in_count: paths in `in` (NULL for hop 0, which covers the W*H pixels).
// Hop 0 also clears the `n_clear` counters of the next pass.
// `image_ready`: the scene's image was complete before the launch before this one started.
template <int R, int FH>
__global__ void __launch_bounds__(128, minb_wave(R == RECIPE_EU, FH == 1)) render_wave(
    const float4 *image, const uint8_t *__restrict__ scene, uint32_t max_objects, bool image_ready,
    uint32_t W, uint32_t H, uint32_t hops, uint32_t hop_index, uint32_t flags, float4 *__restrict__ canvas,
    uint32_t *__restrict__ seeds, uint64_t *stats, WaveQueue in, const uint32_t *in_count,
    WaveQueue out, uint32_t *ctr, uint32_t *clear, uint32_t n_clear) {
    extern __shared__ float4 smem[];
    // the launch before this one appends to `in`: once it has, there is work to load the scene
    // for; until then (and for queues that stay empty) wait for its end first
    uint32_t n = FH == 1 ? W * H : *reinterpret_cast<const volatile uint32_t *>(in_count);
    const bool early = __syncthreads_or(image_ready && n != 0) != 0;
    if (!early) {
        wait_previous();
        launch_next();
        if (FH != 1) n = *reinterpret_cast<const volatile uint32_t *>(in_count);
        if (blockIdx.x * 128u >= n) return;   // nothing for this block: skip the load
    }
    const SceneSmem sm = carve_scene(smem, max_objects);
    StagedScene s;
    const bool staged = load_scene<R>(image, scene, max_objects, s, sm);
    if (early) {
        wait_previous();
        launch_next();
        if (FH != 1) n = *reinterpret_cast<const volatile uint32_t *>(in_count);
    }
    if (FH == 1 && blockIdx.x == 0)
        for (uint32_t i = threadIdx.x; i < n_clear; i += blockDim.x) clear[i] = 0;
    if (!staged) return;

    const uint32_t lane = threadIdx.x & 31;
    const bool last = hop_index + 1 >= hops;
    if (FH != 1 && n < SORT_MIN) in.o = nullptr;   // too few paths for the sort
    LaneStats st;
    for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&ctr[0], 32u);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (base >= n) break;
        wave_chunk<R, FH>(s, base, n, last, W, H, flags, canvas, seeds, in, out, &ctr[1], st);
    }
    flush_lane_stats(stats, st);
}

// ============================================================================ coherence sort
// Between two hop depths of a hyperbolic pass the new queue gets a read order in which
// neighbouring slots hold rays that leave in similar directions from nearby points: from
// hop depth 2 on, rays start all over the scene, and the lanes of a warp otherwise carry
// unrelated candidate lists through the scan. Each path keeps its own state,
// so the order changes no result, only which paths share a warp.
//
// The order is a counting sort on a key of SORT_BINS values: direction cell (the cube face the
// direction points at, 4 x 4 cells per face: 96 cells), then a 2-bit cell per axis of the ray
// start (x, y, log z) over mean +- 2 sigma of the queue, interleaved (Morton order). Two launches
// per hop depth over windows of the queue, both sized for the largest queue and reading its
// length on the device:
//   k_sort_keys     each block takes mean and sigma of the same SORT_THREADS paths spread over the
//                   queue, keys its window, ranks the paths of each bin with shared-memory atomics
//                   and adds the window's counts to the queue's histogram, one global atomic per
//                   bin in use, whose return value is the window's place within the bin;
//   k_sort_scatter  each block scans the histogram (24 KB, every block for itself), adds its
//                   window's places and writes its slots' numbers to their positions.
// Ties within a key land in the order of the windows' atomics.
constexpr uint32_t SORT_THREADS = 1024;
constexpr uint32_t SORT_PER = 16;                            // slots per thread of the largest window
constexpr uint32_t SORT_WINDOW_MAX = SORT_THREADS * SORT_PER, SORT_WINDOW_MIN = 2048;
constexpr uint32_t SORT_POS_BITS = 2;                        // per axis
constexpr uint32_t SORT_BINS = 96u << (3 * SORT_POS_BITS);   // 6144
static_assert(SORT_BINS % SORT_THREADS == 0, "the scan gives every thread a whole number of bins");
struct SortBuf {
    uint32_t *hist;     // 2 x SORT_BINS: a depth counts into one half while the other is cleared
    uint32_t *place;    // per window: SORT_BINS places of its paths within the bins
    uint32_t *key;      // per slot: bin << 16 | rank among the window's paths of that bin
    uint32_t *perm;     // per sorted position: the slot
};
// Windows of a queue of n paths for `blocks` blocks: as many as blocks, of 2048 to 16384 slots.
__host__ __device__ __forceinline__ uint32_t sort_window(uint32_t n, uint32_t blocks) {
    const uint32_t w = ((n + blocks - 1) / blocks + SORT_THREADS - 1) / SORT_THREADS * SORT_THREADS;
    return w < SORT_WINDOW_MIN ? SORT_WINDOW_MIN : w > SORT_WINDOW_MAX ? SORT_WINDOW_MAX : w;
}
static size_t sort_windows(size_t slots, uint32_t blocks) {   // at most, over every queue length
    return std::max<size_t>(blocks, (slots + SORT_WINDOW_MAX - 1) / SORT_WINDOW_MAX);
}
static size_t sort_bytes(size_t slots, uint32_t blocks) {
    return sizeof(uint32_t) * (2 * (size_t)SORT_BINS + sort_windows(slots, blocks) * SORT_BINS + 2 * slots);
}
static SortBuf sort_buf_at(void *base, size_t slots, uint32_t blocks) {
    SortBuf b;
    b.hist = reinterpret_cast<uint32_t *>(base);
    b.place = b.hist + 2 * SORT_BINS;
    b.key = b.place + sort_windows(slots, blocks) * SORT_BINS;
    b.perm = b.key + slots;
    return b;
}

__device__ __forceinline__ float sort_logz(float z) { return z > 0.0f ? __logf(z) : 0.0f; }
__device__ __forceinline__ uint32_t sort_axis_cell(float u, float lo, float scale) {
    return (uint32_t)fminf(fmaxf((u - lo) * scale, 0.0f), (float)((1u << SORT_POS_BITS) - 1u));   // NaN -> 0
}
__device__ __forceinline__ uint32_t spread3(uint32_t c) {   // bits b2 b1 b0 -> b2 0 0 b1 0 0 b0
    return (c & 1u) | ((c & 2u) << 2) | ((c & 4u) << 4);
}
__device__ __forceinline__ uint32_t sort_dir_cell(float4 v) {
    const float ax = fabsf(v.x), ay = fabsf(v.y), az = fabsf(v.z);
    uint32_t face;
    float m, a, b;
    if (ax >= ay && ax >= az) { face = v.x > 0.0f ? 1u : 0u; m = ax; a = v.y; b = v.z; }
    else if (ay >= az)        { face = v.y > 0.0f ? 3u : 2u; m = ay; a = v.z; b = v.x; }
    else                      { face = v.z > 0.0f ? 5u : 4u; m = az; a = v.x; b = v.y; }
    const float r = m > 0.0f ? rcp_approx(m) : 0.0f;
    const uint32_t ia = (uint32_t)fminf(fmaxf((a * r + 1.0f) * 2.0f, 0.0f), 3.0f);
    const uint32_t ib = (uint32_t)fminf(fmaxf((b * r + 1.0f) * 2.0f, 0.0f), 3.0f);
    return face * 16u + ia * 4u + ib;   // < 96
}
// The cells of a queue's positions: lower bound and cells per unit of x, y, log z, from one path
// per thread of the block (every block of a launch takes the same ones).
struct SortCells { float lo[3], scale[3]; };
__device__ __forceinline__ void sort_cells(const float4 *__restrict__ p, uint32_t n, SortCells *cells) {   // whole block
    __shared__ float part[SORT_THREADS / 32][6];
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const float4 q = p[(uint32_t)((uint64_t)t * n / SORT_THREADS)];
    const float l = sort_logz(q.z);
    float a[6] = {q.x, q.x * q.x, q.y, q.y * q.y, l, l * l};
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        for (int o = 16; o; o >>= 1) a[k] += __shfl_xor_sync(0xffffffffu, a[k], o);
        if (lane == 0) part[warp][k] = a[k];
    }
    __syncthreads();
    if (t < 3) {
        float s0 = 0.0f, s1 = 0.0f;
        for (uint32_t w = 0; w < SORT_THREADS / 32; ++w) {
            s0 += part[w][2 * t];
            s1 += part[w][2 * t + 1];
        }
        const float mean = s0 / SORT_THREADS, sd = sqrtf(fmaxf(s1 / SORT_THREADS - mean * mean, 0.0f));
        cells->lo[t] = mean - 2.0f * sd;
        cells->scale[t] = sd > 0.0f ? (float)(1u << SORT_POS_BITS) / (4.0f * sd) : 0.0f;
    }
    __syncthreads();
}
__device__ __forceinline__ uint32_t sort_key(float4 p, float4 v, const SortCells &c) {   // < SORT_BINS
    const uint32_t cx = sort_axis_cell(p.x, c.lo[0], c.scale[0]);
    const uint32_t cy = sort_axis_cell(p.y, c.lo[1], c.scale[1]);
    const uint32_t cz = sort_axis_cell(sort_logz(p.z), c.lo[2], c.scale[2]);
    return (sort_dir_cell(v) << (3 * SORT_POS_BITS)) | spread3(cx) | (spread3(cy) << 1) | (spread3(cz) << 2);
}

// The m paths of one window: their bins and ranks, and the window's places within the bins of
// the queue's histogram (whole block).
__device__ __forceinline__ void sort_window_keys(const float4 *__restrict__ p, const float4 *__restrict__ v, uint32_t m,
                                                 const SortCells &cells, uint32_t *s_hist, uint32_t *hist,
                                                 uint32_t *__restrict__ place, uint32_t *__restrict__ key) {
    const uint32_t t = threadIdx.x;
    for (uint32_t b = t; b < SORT_BINS; b += SORT_THREADS) s_hist[b] = 0;
    __syncthreads();
    for (uint32_t i = t; i < m; i += SORT_THREADS) {
        const uint32_t k = sort_key(p[i], v[i], cells);
        key[i] = (k << 16) | atomicAdd(&s_hist[k], 1u);
    }
    __syncthreads();
    for (uint32_t b = t; b < SORT_BINS; b += SORT_THREADS) {
        const uint32_t c = s_hist[b];
        if (c) place[b] = atomicAdd(&hist[b], c);
    }
    __syncthreads();
}

__global__ void __launch_bounds__(SORT_THREADS) k_sort_keys(const float4 *__restrict__ p, const float4 *__restrict__ v,
                                                           const uint32_t *count, uint32_t *hist,
                                                           uint32_t *__restrict__ place, uint32_t *__restrict__ key) {
    extern __shared__ uint32_t s_hist[];   // SORT_BINS
    __shared__ SortCells cells;
    wait_previous();
    launch_next();
    const uint32_t n = *reinterpret_cast<const volatile uint32_t *>(count), win = sort_window(n, gridDim.x);
    if (n < SORT_MIN || (uint64_t)blockIdx.x * win >= n) return;
    sort_cells(p, n, &cells);
    for (uint32_t w = blockIdx.x; (uint64_t)w * win < n; w += gridDim.x) {
        const uint32_t base = w * win, m = min(win, n - base);
        sort_window_keys(p + base, v + base, m, cells, s_hist, hist, place + (size_t)w * SORT_BINS, key + base);
    }
}

// Exclusive scan of a histogram of SORT_BINS into shared memory, by the whole block.
__device__ __forceinline__ void sort_scan(const uint32_t *hist, uint32_t *s_base) {
    __shared__ uint32_t s_warp[SORT_THREADS / 32];
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    constexpr uint32_t PER = SORT_BINS / SORT_THREADS;
    uint32_t c[PER], sum = 0;
#pragma unroll
    for (uint32_t k = 0; k < PER; ++k) {
        c[k] = hist[t * PER + k];
        sum += c[k];
    }
    uint32_t x = sum;   // inclusive scan within the warp
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    uint32_t run = x - sum;
    for (uint32_t w = 0; w < warp; ++w) run += s_warp[w];
#pragma unroll
    for (uint32_t k = 0; k < PER; ++k) {
        s_base[t * PER + k] = run;
        run += c[k];
    }
    __syncthreads();
}

__global__ void __launch_bounds__(SORT_THREADS) k_sort_scatter(const uint32_t *key, const uint32_t *count,
                                                              const uint32_t *hist, uint32_t *next_hist,
                                                              const uint32_t *place, uint32_t *__restrict__ perm) {
    extern __shared__ uint32_t s_base[];   // SORT_BINS
    wait_previous();
    launch_next();
    const uint32_t n = *reinterpret_cast<const volatile uint32_t *>(count), t = threadIdx.x, win = sort_window(n, gridDim.x);
    for (uint32_t b = blockIdx.x * SORT_THREADS + t; b < SORT_BINS; b += gridDim.x * SORT_THREADS) next_hist[b] = 0;
    if (n < SORT_MIN || (uint64_t)blockIdx.x * win >= n) return;
    sort_scan(hist, s_base);
    for (uint32_t w = blockIdx.x; (uint64_t)w * win < n; w += gridDim.x) {
        const uint32_t base = w * win, m = min(win, n - base);
        for (uint32_t i = t; i < m; i += SORT_THREADS) {
            const uint32_t k = key[base + i];
            perm[s_base[k >> 16] + place[(size_t)w * SORT_BINS + (k >> 16)] + (k & 0xFFFFu)] = base + i;
        }
    }
}

// ============================================================================ batch
struct BatchView {          // device copy of htc_view plus host-derived fields
    const uint8_t *scene;
    uint64_t scene_size;
    float4 *canvas;
    uint32_t *seeds;
    uint32_t width, height;
    int32_t recipe;
    uint32_t hops, flags;
    int32_t address_width;
    uint32_t passes;
    uint32_t max_objects;   // objects the scene buffer can hold
    uint64_t qoff;          // first slot of the view's region in the wavefront queues
    float4 *image;          // its scene's image
};

// Wavefront form of the batch: one launch per (pass, hop depth) over every view. Each view
// has its own region of the two queues and its own append counter; the launch cuts the
// views' current paths into tiles of `tile_slots` (a block-wide prefix sum over the views'
// counts, expensive views first), blocks take tiles from a counter and stage a view's scene
// only when it changes, and warps take 32 slots of the tile at a time (wave_chunk). A
// view's paths therefore run exactly as in render_wave, and every view's canvas and seeds
// are bit-identical to rendering it alone.
//   cnt[h * n_views + v]: paths of view v appended by hop h of this pass;
//   grab: tiles taken by the blocks of one launch (a word of its own per launch of a pass).
__device__ __forceinline__ uint32_t batch_wave_count(const BatchView &v, uint32_t vi, uint32_t pass, uint32_t h,
                                                     const uint32_t *cnt, uint32_t n_views) {
    if (pass >= v.passes || h >= v.hops) return 0;
    if (h == 0) return v.width * v.height;
    return *reinterpret_cast<const volatile uint32_t *>(&cnt[(h - 1) * n_views + vi]);
}

// The scene images of the views of `order`, one block each.
__global__ void __launch_bounds__(STAGE_THREADS) k_batch_stage(const BatchView *__restrict__ views,
                                                              const uint32_t *__restrict__ order, uint32_t *err) {
    const BatchView &v = views[order[blockIdx.x]];
    if (v.recipe == RECIPE_HY) stage_image<RECIPE_HY>(v.scene, v.scene_size, v.max_objects, v.address_width, err, v.image);
    else stage_image<RECIPE_EU>(v.scene, v.scene_size, v.max_objects, v.address_width, err, v.image);
}

// RF: the recipe of the views in `order`.
template <int RF, int FH>
__global__ void __launch_bounds__(128, minb_batch(RF == RECIPE_EU)) render_batch_wave(
    const BatchView *__restrict__ views, const uint32_t *__restrict__ order, uint32_t n_order, uint32_t n_views,
    uint32_t pass, uint32_t h, uint32_t tile_slots, uint32_t smem_objects, WaveQueue in, WaveQueue out,
    uint32_t *cnt, uint32_t *grab, uint64_t *stats, uint32_t n_sorted, uint32_t *clear, size_t n_clear) {
    extern __shared__ float4 smem[];
    __shared__ uint32_t s_tile, s_next, s_total, s_tsize;
    __shared__ int s_staged_view, s_staged_ok;
    uint32_t *s_pref = reinterpret_cast<uint32_t *>(carve_scene(smem, smem_objects).end);   // n_order + 1 tile offsets
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    wait_previous();
    launch_next();
    if (FH == 1 && blockIdx.x == 0)
        for (size_t i = tid; i < n_clear; i += blockDim.x) clear[i] = 0;

    // tiles of every view at this hop, in `order`, as a prefix sum. The tile size adapts to
    // the launch: about 16 tiles per block when the paths are few (a multiple of 128 slots,
    // so the four warps of a block take equal shares; at least one chunk per warp),
    // `tile_slots` when they are many, so a launch ends with short tiles.
    for (uint32_t i = tid; i < n_order; i += blockDim.x) {
        const uint32_t vi = order[i];
        s_pref[i + 1] = batch_wave_count(views[vi], vi, pass, h, cnt, n_views);
    }
    if (tid == 0) {
        s_pref[0] = 0;
        s_staged_view = -1;
    }
    __syncthreads();
    if (tid < 32) {
        uint64_t paths = 0;
        for (uint32_t i = lane; i < n_order; i += 32) paths += s_pref[i + 1];
        for (int off = 16; off > 0; off >>= 1) paths += __shfl_xor_sync(0xffffffffu, paths, off);
        uint64_t per = (paths / (16ull * gridDim.x) + 127) & ~127ull;
        if (per < 128) per = 128;
        if (per > tile_slots) per = tile_slots;
        if (lane == 0) s_tsize = (uint32_t)per;
    }
    __syncthreads();
    const uint32_t tile = s_tsize;
    for (uint32_t i = tid; i < n_order; i += blockDim.x) s_pref[i + 1] = (s_pref[i + 1] + tile - 1) / tile;
    __syncthreads();
    if (tid < 32) {
        uint32_t carry = 0;
        for (uint32_t b0 = 0; b0 < n_order; b0 += 32) {
            const uint32_t i = b0 + lane;
            uint32_t x = i < n_order ? s_pref[i + 1] : 0;
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
                if (lane >= (uint32_t)off) x += y;
            }
            if (i < n_order) s_pref[i + 1] = x + carry;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) s_total = carry;
    }
    __syncthreads();
    const uint32_t total = s_total;
    StagedScene s;
    s.n = 0;
    LaneStats st;
    for (;;) {
        __syncthreads();
        if (tid == 0) {
            s_tile = total ? atomicAdd(grab, 1u) : 0u;
            s_next = 0;
        }
        __syncthreads();
        const uint32_t t = s_tile;
        if (t >= total) break;
        uint32_t lo = 0, hi = n_order - 1;   // the last view whose first tile is <= t
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) >> 1;
            if (s_pref[mid] <= t) lo = mid;
            else hi = mid - 1;
        }
        const uint32_t vi = order[lo];
        const BatchView &v = views[vi];
        const uint32_t n = batch_wave_count(v, vi, pass, h, cnt, n_views);
        const uint32_t first = (t - s_pref[lo]) * tile;
        const uint32_t count = min(tile, n - first);
        if ((int)vi != s_staged_view) {
            const bool ok = load_scene<RF>(v.image, v.scene, v.max_objects, s, carve_scene(smem, v.max_objects));
            __syncthreads();
            if (tid == 0) {
                s_staged_view = (int)vi;
                s_staged_ok = ok ? 1 : 0;
            }
            __syncthreads();
        }
        if (!s_staged_ok) continue;
        // the first n_sorted views of `order` read a tile's paths through their sorted order
        // (view-relative slots), the others in queue order
        const bool sorted = in.o != nullptr && lo < n_sorted;
        WaveQueue vin = wave_at(in, sorted ? v.qoff : v.qoff + first);
        vin.o = sorted ? in.o + v.qoff + first : nullptr;
        const WaveQueue vout = wave_at(out, v.qoff);
        const bool last_hop = h + 1 >= v.hops;
        uint32_t *out_count = &cnt[h * n_views + vi];
        float4 *canvas = v.canvas;
        uint32_t *seeds = v.seeds;
        for (;;) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&s_next, 32u);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (base >= count) break;
            // slots are the view's on hop 0, tile-relative queue slots later
            const uint32_t b0 = FH == 1 ? first + base : base, n0 = FH == 1 ? first + count : count;
            wave_chunk<RF, FH>(s, b0, n0, last_hop, v.width, v.height, v.flags, canvas, seeds, vin, vout,
                               out_count, st);
        }
    }
    flush_lane_stats(stats, st);
}

// ============================================================================ batch: coherence sort
// The coherence sort of the single-view wavefronts, per view: the first `n_seg` hyperbolic
// views of the launch order (the most expensive ones; at most BATCH_SORT_VIEWS) each get a
// histogram, and their queued paths a read order within their own queue region. The launches'
// windows are cut from the views' queues one view after the other, none over two views.
constexpr uint32_t BATCH_SORT_VIEWS = 128;
struct BatchSortBuf {
    uint32_t *hist;     // 2 x BATCH_SORT_VIEWS x SORT_BINS
    uint32_t *place;    // per window: SORT_BINS
    uint32_t *key;      // per queue slot
    uint32_t *perm;     // per queue slot: view-relative slot in sorted order
};
// Windows of all views: a view's last may be short.
static size_t batch_sort_windows(uint64_t slots, uint32_t blocks) { return sort_windows(slots, blocks) + BATCH_SORT_VIEWS; }
static size_t batch_sort_bytes(uint64_t slots, uint32_t blocks) {
    return sizeof(uint32_t) * (2 * (size_t)BATCH_SORT_VIEWS * SORT_BINS + batch_sort_windows(slots, blocks) * SORT_BINS + 2 * slots);
}
static BatchSortBuf batch_sort_at(void *base, uint64_t slots, uint32_t blocks) {
    BatchSortBuf b;
    b.hist = reinterpret_cast<uint32_t *>(base);
    b.place = b.hist + 2 * (size_t)BATCH_SORT_VIEWS * SORT_BINS;
    b.key = b.place + batch_sort_windows(slots, blocks) * SORT_BINS;
    b.perm = b.key + slots;
    return b;
}

// The windows of the first n_seg views of `order` at queue depth h (whole block): s_count[i] paths
// of view i, s_win[i] windows of the views before it; returns the window size.
__device__ __forceinline__ uint32_t bsort_windows(const BatchView *views, const uint32_t *order, uint32_t n_seg,
                                                  uint32_t n_views, uint32_t pass, uint32_t h, const uint32_t *cnt,
                                                  uint32_t *s_count, uint32_t *s_win) {
    __shared__ uint32_t s_size;
    for (uint32_t i = threadIdx.x; i < n_seg; i += blockDim.x) {
        const uint32_t vi = order[i];
        s_count[i] = batch_wave_count(views[vi], vi, pass, h, cnt, n_views);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint32_t lane = threadIdx.x;
        uint64_t total = 0;
        for (uint32_t i = lane; i < n_seg; i += 32) total += s_count[i];
        for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        const uint32_t win = sort_window((uint32_t)min(total, (uint64_t)0xFFFFFFFFu), gridDim.x);
        uint32_t carry = 0;
        for (uint32_t b0 = 0; b0 < n_seg; b0 += 32) {
            const uint32_t i = b0 + lane, own = i < n_seg ? (s_count[i] + win - 1) / win : 0;
            uint32_t x = own;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= (uint32_t)o) x += y;
            }
            if (i < n_seg) s_win[i] = x + carry - own;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
        if (lane == 0) {
            s_win[n_seg] = carry;
            s_size = win;
        }
    }
    __syncthreads();
    return s_size;
}
__device__ __forceinline__ uint32_t bsort_view(const uint32_t *s_win, uint32_t n_seg, uint32_t w) {
    uint32_t lo = 0, hi = n_seg - 1;   // the last view whose first window is <= w
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (s_win[mid] <= w) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__global__ void __launch_bounds__(SORT_THREADS) k_bsort_keys(const BatchView *__restrict__ views,
                                                            const uint32_t *__restrict__ order, uint32_t n_seg,
                                                            uint32_t n_views, uint32_t pass, uint32_t h,
                                                            const uint32_t *cnt, const float4 *__restrict__ qp,
                                                            const float4 *__restrict__ qv, uint32_t *hist,
                                                            uint32_t *__restrict__ place, uint32_t *__restrict__ key) {
    extern __shared__ uint32_t s_hist[];   // SORT_BINS, then n_seg counts and n_seg + 1 window numbers
    __shared__ SortCells cells;
    uint32_t *s_count = s_hist + SORT_BINS, *s_win = s_count + n_seg;
    wait_previous();
    launch_next();
    const uint32_t win = bsort_windows(views, order, n_seg, n_views, pass, h, cnt, s_count, s_win);
    uint32_t of = 0xFFFFFFFFu;   // the view that `cells` are of
    for (uint32_t w = blockIdx.x; w < s_win[n_seg]; w += gridDim.x) {
        const uint32_t sg = bsort_view(s_win, n_seg, w), n = s_count[sg], base = (w - s_win[sg]) * win;
        const uint64_t qoff = views[order[sg]].qoff;
        if (sg != of) sort_cells(qp + qoff, n, &cells);
        of = sg;
        sort_window_keys(qp + qoff + base, qv + qoff + base, min(win, n - base), cells, s_hist, hist + (size_t)sg * SORT_BINS,
                         place + (size_t)w * SORT_BINS, key + qoff + base);
    }
}

// perm[qoff + position] = view-relative slot; clears the other half of the histograms.
__global__ void __launch_bounds__(SORT_THREADS) k_bsort_scatter(const BatchView *__restrict__ views,
                                                               const uint32_t *__restrict__ order, uint32_t n_seg,
                                                               uint32_t n_views, uint32_t pass, uint32_t h,
                                                               const uint32_t *cnt, const uint32_t *key,
                                                               const uint32_t *hist, uint32_t *next_hist,
                                                               const uint32_t *place,
                                                               uint32_t *__restrict__ perm) {
    extern __shared__ uint32_t s_base[];   // SORT_BINS, then n_seg counts and n_seg + 1 window numbers
    uint32_t *s_count = s_base + SORT_BINS, *s_win = s_count + n_seg;
    wait_previous();
    launch_next();
    const uint32_t win = bsort_windows(views, order, n_seg, n_views, pass, h, cnt, s_count, s_win);
    for (uint32_t b = blockIdx.x * SORT_THREADS + threadIdx.x; b < n_seg * SORT_BINS; b += gridDim.x * SORT_THREADS)
        next_hist[b] = 0;
    uint32_t of = 0xFFFFFFFFu;   // the view whose histogram is scanned
    for (uint32_t w = blockIdx.x; w < s_win[n_seg]; w += gridDim.x) {
        const uint32_t sg = bsort_view(s_win, n_seg, w), base = (w - s_win[sg]) * win, m = min(win, s_count[sg] - base);
        const uint64_t qoff = views[order[sg]].qoff;
        __syncthreads();
        if (sg != of) sort_scan(hist + (size_t)sg * SORT_BINS, s_base);
        of = sg;
        for (uint32_t i = threadIdx.x; i < m; i += SORT_THREADS) {
            const uint32_t k = key[qoff + base + i];
            perm[qoff + s_base[k >> 16] + place[(size_t)w * SORT_BINS + (k >> 16)] + (k & 0xFFFFu)] = base + i;
        }
    }
}

// ============================================================================ double_support
// A scene serialized with double_support (types/src/config.rs:38-43) stores every f64 field
// in 8 bytes, and a primitive vector or matrix of f64 is aligned to its own size
// (types/src/primitive/scalar.rs:186-215, types/src/primitive/matrix.rs:171-209); colors stay
// f32. The reference then builds its kernel with real = double (processing/src/render.rs:50).
// This path narrows such a scene once per render call into the f32 layout the kernels read,
// rounding each f64 to the nearest f32 -- the value the reference's own serializer writes for
// the same scene without double_support (`*self as f32`, scalar.rs:198-207) -- and then
// transports in FP32 as for any other scene: a double_support scene renders bit for bit as
// its f32 serialization does. The field tables follow the layouts hypertrace_b200/types.py
// derives (Moebius 8 reals, Shift3 3 + 1, Rotation3 4, fov and portions 1).
struct NarrowField { uint16_t src, dst; uint8_t kind, n; };   // kind: 0 = n f64 -> f32, 1 = n words, 2 = usize
struct NarrowLayout {
    uint32_t src_objects, src_stride, dst_objects, dst_stride, src_count, dst_count;
    uint32_t n_header, n_object;
    NarrowField header[5], object[8];
};
__constant__ NarrowLayout c_narrow[2] = {
    // HTC_RECIPE_HY: view map, fov, background | map, diffuse color / portion, specular portion,
    // emission, luminous portion, shape index
    {256, 192, 128, 128, 192, 96, 3, 7,
     {{0, 0, 0, 8}, {64, 32, 0, 1}, {128, 64, 1, 3}},
     {{0, 0, 0, 8}, {64, 32, 1, 3}, {80, 48, 0, 1}, {96, 64, 0, 1}, {112, 80, 1, 3}, {128, 96, 0, 1}, {144, 112, 2, 1}}},
    // HTC_RECIPE_EU: view shift, rotation, fov, background | shift, rotation, diffuse color /
    // portion, specular portion, emission, luminous portion, shape index
    {160, 160, 80, 128, 128, 64, 4, 8,
     {{0, 0, 0, 3}, {32, 16, 0, 4}, {64, 32, 0, 1}, {96, 48, 1, 3}},
     {{0, 0, 0, 3}, {32, 16, 0, 4}, {64, 32, 1, 3}, {80, 48, 0, 1}, {96, 64, 0, 1}, {112, 80, 1, 3}, {128, 96, 0, 1},
      {144, 112, 2, 1}}},
};
constexpr uint32_t NARROW_SRC_OBJECTS[2] = {256, 160}, NARROW_SRC_STRIDE[2] = {192, 160};

__device__ __forceinline__ void narrow_fields(const uint8_t *src, uint8_t *dst, const NarrowField *f, uint32_t nf,
                                              int usize_bytes) {
    for (uint32_t i = 0; i < nf; ++i) {
        const NarrowField fd = f[i];
        if (fd.kind == 0) {
            const double *a = reinterpret_cast<const double *>(src + fd.src);
            float *b = reinterpret_cast<float *>(dst + fd.dst);
            for (uint32_t j = 0; j < fd.n; ++j) b[j] = __double2float_rn(a[j]);
        } else {
            const uint32_t words = fd.kind == 1 ? fd.n : (uint32_t)usize_bytes / 4u;
            const uint32_t *a = reinterpret_cast<const uint32_t *>(src + fd.src);
            uint32_t *b = reinterpret_cast<uint32_t *>(dst + fd.dst);
            for (uint32_t j = 0; j < words; ++j) b[j] = a[j];
        }
    }
}
// One thread per record (record 0 = the header, record 1 + i = object i). An object count the
// source buffer cannot hold (or the destination was not sized for) is written as all ones,
// which the render's own staging rejects as a scene error.
__global__ void k_narrow_scene(int li, const uint8_t *__restrict__ src, uint64_t src_size, uint8_t *__restrict__ dst,
                               uint32_t dst_capacity, int usize_bytes) {
    const NarrowLayout &L = c_narrow[li];
    const uint32_t count_lo = *reinterpret_cast<const uint32_t *>(src + L.src_count);
    const uint32_t count_hi = usize_bytes == 8 ? *reinterpret_cast<const uint32_t *>(src + L.src_count + 4) : 0u;
    const uint64_t holds = src_size >= L.src_objects ? (src_size - L.src_objects) / L.src_stride : 0u;
    const bool ok = count_hi == 0 && count_lo <= holds && count_lo <= dst_capacity;
    const uint32_t n = ok ? count_lo : 0u;
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r <= n; r += gridDim.x * blockDim.x) {
        if (r == 0) {
            narrow_fields(src, dst, L.header, L.n_header, usize_bytes);
            uint32_t *c = reinterpret_cast<uint32_t *>(dst + L.dst_count);
            c[0] = ok ? count_lo : 0xFFFFFFFFu;
            if (usize_bytes == 8) c[1] = ok ? 0u : 0xFFFFFFFFu;
        } else {
            narrow_fields(src + L.src_objects + (size_t)(r - 1) * L.src_stride,
                          dst + L.dst_objects + (size_t)(r - 1) * L.dst_stride, L.object, L.n_object, usize_bytes);
        }
    }
}

// ============================================================================ post
// pow(max(x, 0), gamma) is evaluated in FP64 and rounded once (the host libm's powf is
// within a fraction of an ulp of that).
__device__ __forceinline__ float gamma1(float x, float g) {
    float m = fmaxf(x, 0.0f);
    return (float)pow((double)m, (double)g);
}
__device__ __forceinline__ uint8_t pack1(float x) {
    float c = fminf(fmaxf(x, 0.0f), 1.0f);
    return (uint8_t)__float2uint_rz(255.0f * c);
}

__global__ void k_extract(uint32_t n, float passes, const float4 *__restrict__ canvas, float4 *__restrict__ image) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4 c = canvas[i];
        image[i] = make_float4(c.x / passes, c.y / passes, c.z / passes, c.w / passes);
    }
}
__global__ void k_gamma(uint32_t n, float g, const float4 *__restrict__ in, float4 *__restrict__ out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4 c = in[i];
        out[i] = make_float4(gamma1(c.x, g), gamma1(c.y, g), gamma1(c.z, g), gamma1(c.w, g));
    }
}
__global__ void k_pack(uint32_t n, const float4 *__restrict__ in, uchar4 *__restrict__ out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float4 c = in[i];
        out[i] = make_uchar4(pack1(c.x), pack1(c.y), pack1(c.z), pack1(c.w));
    }
}
// Per-pixel initial RNG states: seed_i = fmix32(global_seed ^ fmix32(i + offset)), MurmurHash3's
// 32-bit finaliser (the harness seeds; the reference fills the buffer from a host SmallRng,
// processing/src/canvas.rs:193-195, and its kernel only consumes it).
__device__ __forceinline__ uint32_t fmix32(uint32_t h) {
    h ^= h >> 16;
    h *= 0x85EBCA6Bu;
    h ^= h >> 13;
    h *= 0xC2B2AE35u;
    h ^= h >> 16;
    return h;
}
__global__ void k_fill_seeds(uint32_t n, uint32_t global_seed, uint32_t offset, uint32_t *__restrict__ seeds) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        seeds[i] = fmix32(global_seed ^ fmix32(i + offset));
}

// pack1(gamma1(x, g)) for g > 0 without the FP64 power where an FP32 one decides the byte: y =
// exp2(g log2 x) is within 2.3e-6 relative of x^g while 255 y >= 1 (|g log2 x| <= 8; log2f is good to
// 1 ulp, exp2f to 2), so the byte is that of y unless 255 y lies within 3e-6 (255 y) + 1e-6 of a
// whole number (about one value in 1000). The power of x >= 1 clamps to 1. The fused kernel was
// bound by the four FP64 powers a pixel: 1920x1080 71 us, now 27 (its instructions; the 41 MB that
// it reads and writes take 6.4).
static __device__ __noinline__ uint8_t gamma_pack_exact(float x, float g) { return pack1(gamma1(x, g)); }
__device__ __forceinline__ uint8_t gamma_pack(float x, float g) {
    if (x >= 1.0f) return 255;
    if (!(x > 0.0f)) return 0;   // max(x, 0) = 0, NaN too
    const float v = 255.0f * exp2f(g * log2f(x));
    if (!(fabsf(v - rintf(v)) > fmaf(v, 3e-6f, 1e-6f))) return gamma_pack_exact(x, g);
    return (uint8_t)__float2uint_rz(v);
}
__global__ void k_extract_gamma_pack(uint32_t n, float passes, float g, const float4 *__restrict__ canvas,
                                     uchar4 *__restrict__ out) {
    const bool usual = g > 0.0f && g < 16.0f;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 c = canvas[i];
        const float x = c.x / passes, y = c.y / passes, z = c.z / passes, w = c.w / passes;
        out[i] = usual ? make_uchar4(gamma_pack(x, g), gamma_pack(y, g), gamma_pack(z, g), gamma_pack(w, g))
                       : make_uchar4(gamma_pack_exact(x, g), gamma_pack_exact(y, g), gamma_pack_exact(z, g), gamma_pack_exact(w, g));
    }
}

// ============================================================================ calibration
// FP32 FMA throughput probe: independent FMA chains per thread, enough warps to fill every
// scheduler. 2 flops per FMA; the result is written so nothing is dead code.
__global__ void __launch_bounds__(256) k_fma_probe(float *out, int iters) {
    float a0 = threadIdx.x * 1e-7f, a1 = a0 + 1e-7f, a2 = a0 + 2e-7f, a3 = a0 + 3e-7f;
    float a4 = a0 + 4e-7f, a5 = a0 + 5e-7f, a6 = a0 + 6e-7f, a7 = a0 + 7e-7f;
    const float m = 0.999999f, c = 1e-7f;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            a0 = fmaf(a0, m, c); a1 = fmaf(a1, m, c); a2 = fmaf(a2, m, c); a3 = fmaf(a3, m, c);
            a4 = fmaf(a4, m, c); a5 = fmaf(a5, m, c); a6 = fmaf(a6, m, c); a7 = fmaf(a7, m, c);
        }
    }
    out[blockIdx.x * blockDim.x + threadIdx.x] = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
}

// ============================================================================ workspace pools
// One memory pool per device for the workspaces that calls take and give back in stream order
// (render_wave_pooled), shared by the device's programs so that a new program finds memory that
// an earlier one's calls have mapped (a pool per program made its first call 2 to 15 ms long). Made
// by the first call that needs it, destroyed with the last program; between calls it keeps up to two
// workspaces of the largest size taken so far and 64 MB (its reservations are larger than what
// is taken from them, and what is over the limit goes back to the system at every
// synchronisation: 200 us a call). What it keeps is not lost to others: an allocation that needs it
// gets it (cudaMalloc of the device's free memory and half of what the pool kept succeeds).
namespace {
constexpr int MAX_DEVICES = 64;
struct DevicePool {
    std::mutex mutex;
    cudaMemPool_t pool = nullptr;
    uint32_t programs = 0;
    size_t largest = 0;    // workspace taken so far
    uint32_t without = 0;  // passes that asked for a larger one since
} g_pools[MAX_DEVICES];
int pool_enter(int dev) {
    if (dev < 0 || dev >= MAX_DEVICES) return -1;
    std::lock_guard<std::mutex> lock(g_pools[dev].mutex);
    ++g_pools[dev].programs;
    return dev;
}
void pool_leave(int dev) {
    if (dev < 0) return;
    DevicePool &d = g_pools[dev];
    std::lock_guard<std::mutex> lock(d.mutex);
    if (--d.programs == 0 && d.pool) {
        cudaMemPoolDestroy(d.pool);   // blocks still in use are freed with their last use
        d.pool = nullptr;
        d.largest = 0;
    }
    if (d.programs == 0) d.without = 0;
}
// While another stream captures in the global mode, calls that are not stream-ordered on every thread
// would break its capture, and so do those of a pool. They do not touch that stream, so the thread
// leaves the mode for as long as it works with the pool.
struct RelaxedCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};
// A block of `bytes` for `passes` passes on `st`, or NULL. A workspace larger than any before has to be
// mapped, which takes 1.2 ms at 800x600 and 3 at 1080p, more than wavefronts save on a few passes. So
// the first POOL_WITHOUT passes that ask for one go without, in calls of up to POOL_LONG passes: a program
// that is made for a frame or two and destroyed maps nothing (made, one frame, destroyed: 18 objects at
// 800x600 2.1 -> 1.1 ms, 200 at 1080p 6.0 -> 3.7; two frames 2.6 -> 1.5 and 7.3 -> 6.5; 8 passes in one call
// of 18 and of 77 objects 5.3 -> 4.1 and 3.6 -> 3.4, 16 passes 9.1 with either).
constexpr uint32_t POOL_WITHOUT = 4, POOL_LONG = 8;
void *pool_take(int dev, size_t bytes, uint32_t passes, cudaStream_t st) {
    if (dev < 0) return nullptr;
    const RelaxedCapture relaxed;
    DevicePool &d = g_pools[dev];
    std::lock_guard<std::mutex> lock(d.mutex);
    if (bytes > d.largest && d.without < POOL_WITHOUT && passes <= POOL_LONG) {
        d.without += passes;
        return nullptr;
    }
    cudaError_t e = cudaSuccess;
    if (!d.pool) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        e = cudaMemPoolCreate(&d.pool, &props);
        if (e != cudaSuccess) d.pool = nullptr;
    }
    if (e == cudaSuccess && bytes > d.largest) {
        uint64_t keep = 2 * (uint64_t)bytes + (64u << 20);
        e = cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep);
        if (e == cudaSuccess) {
            d.largest = bytes;
            d.without = 0;
        }
    }
    void *block = nullptr;
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(&block, bytes, d.pool, st);
    if (e != cudaSuccess) {
        cudaGetLastError();   // the caller renders without
        return nullptr;
    }
    return block;
}
// Gives the block back when the work enqueued on `st` so far is done.
cudaError_t pool_give(void *block, cudaStream_t st) {
    const RelaxedCapture relaxed;
    return cudaFreeAsync(block, st);
}
}  // namespace

// ============================================================================ C ABI
static int check_program(const htc_program *p) {
    if (!p) return fail(HTC_ERR_INVALID, "program is NULL");
    return HTC_OK;
}
static size_t smem_bytes(uint32_t max_objects) {   // carve_scene's layout
    return scene_win_offset(max_objects) + 2u * 16u * BLOCK_THREADS;
}
static uint32_t objects_capacity(int recipe, size_t scene_size) {
    const size_t hdr = recipe == HTC_RECIPE_HY ? Layout<RECIPE_HY>::OBJECTS : Layout<RECIPE_EU>::OBJECTS;
    if (scene_size < hdr) return 0;
    size_t n = (scene_size - hdr) / OBJ_STRIDE;
    return n > 0xFFFFFFu ? 0xFFFFFFu : (uint32_t)n;
}

template <int R>
static int set_smem_attr(size_t smem) {
    HTC_CUDA(cudaFuncSetAttribute(render_plain<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    HTC_CUDA(cudaFuncSetAttribute(render_persistent<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    HTC_CUDA(cudaFuncSetAttribute(render_wave<R, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    HTC_CUDA(cudaFuncSetAttribute(render_wave<R, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return HTC_OK;
}

static int validate_render_args(htc_program *p, uint32_t W, uint32_t H, const void *scene, size_t scene_size,
                                const float *canvas, const uint32_t *seeds, uint32_t *max_objects, size_t *smem) {
    int rc = check_program(p);
    if (rc) return rc;
    if (W == 0 || H == 0) return fail(HTC_ERR_INVALID, "canvas width and height must be positive");
    if ((uint64_t)W * (uint64_t)H >= 0xFFFFFFFFull) return fail(HTC_ERR_INVALID, "canvas too large (W*H must fit in 32 bits)");
    if (!scene || !canvas || !seeds) return fail(HTC_ERR_INVALID, "scene, canvas and seeds must be device pointers");
    if ((reinterpret_cast<uintptr_t>(scene) & 15u) != 0 || (reinterpret_cast<uintptr_t>(canvas) & 15u) != 0)
        return fail(HTC_ERR_INVALID, "scene and canvas must be 16-byte aligned");
    *max_objects = objects_capacity(p->recipe, scene_size);
    if (scene_size < (p->recipe == HTC_RECIPE_HY ? 128u : 80u))
        return fail(HTC_ERR_SCENE, "scene buffer is smaller than the scene header");
    *smem = smem_bytes(*max_objects);
    if (*smem > (size_t)p->max_smem)
        return fail(HTC_ERR_UNSUPPORTED, "scene has more objects than shared memory can stage");
    return HTC_OK;
}

// A program around a generic scene kernel: error word only (no staging, no queue).
static int wrap_generic(GenericProgram *g, int recipe, uint32_t light_hops, int address_width, uint32_t flags,
                        htc_program **out) {
    htc_program *p = new htc_program();
    p->recipe = recipe;
    p->hops = light_hops;
    p->address_width = address_width;
    p->flags = flags;
    p->generic = g;
    p->device = -1;
    cudaError_t e = cudaMalloc(&p->d_err, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMemset(p->d_err, 0, sizeof(uint32_t));
    if (e != cudaSuccess) {
        if (p->d_err) cudaFree(p->d_err);
        generic_program_destroy(g);
        delete p;
        return cuda_fail(e, "htc_program_create");
    }
    *out = p;
    return HTC_OK;
}

extern "C" {

const char *htc_last_error(void) { return g_last_error.c_str(); }
int htc_version(void) { return 10000; }

int htc_device_count(int *count) {
    if (!count) return fail(HTC_ERR_INVALID, "count is NULL");
    HTC_CUDA(cudaGetDeviceCount(count));
    return HTC_OK;
}
int htc_set_device(int device) {
    HTC_CUDA(cudaSetDevice(device));
    return HTC_OK;
}

int htc_program_create(int recipe, uint32_t light_hops, int address_width, int double_support,
                       uint32_t flags, htc_program **out) {
    if (!out) return fail(HTC_ERR_INVALID, "out is NULL");
    *out = nullptr;
    if (recipe != HTC_RECIPE_HY && recipe != HTC_RECIPE_EU && recipe != HTC_RECIPE_HY_TILED &&
        recipe != HTC_RECIPE_EU_GRADIENT)
        return fail(HTC_ERR_UNSUPPORTED, "unknown scene recipe");
    if (light_hops == 0) return fail(HTC_ERR_INVALID, "light_hops must be positive");
    if (address_width != 32 && address_width != 64) return fail(HTC_ERR_INVALID, "address_width must be 32 or 64");
    if (flags & ~(HTC_FLAG_JITTER_YX | HTC_FLAG_NO_SORT)) return fail(HTC_ERR_INVALID, "unknown program flags");
    if (double_support && recipe != HTC_RECIPE_HY && recipe != HTC_RECIPE_EU)
        return fail(HTC_ERR_UNSUPPORTED, "double_support scenes are served for HTC_RECIPE_HY and HTC_RECIPE_EU only");
    if (recipe == HTC_RECIPE_HY_TILED || recipe == HTC_RECIPE_EU_GRADIENT) {
        GenericProgram *g = nullptr;
        int rc = generic_program_create(recipe, address_width, &g);
        if (rc) return rc;
        return wrap_generic(g, recipe, light_hops, address_width, flags, out);
    }
    int dev = 0;
    HTC_CUDA(cudaGetDevice(&dev));
    htc_program *p = new htc_program();
    p->recipe = recipe;
    p->hops = light_hops;
    p->address_width = address_width;
    p->flags = flags;
    p->double_support = double_support ? 1 : 0;
    cudaError_t e = cudaDeviceGetAttribute(&p->num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&p->max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaMalloc(&p->d_err, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMemset(p->d_err, 0, sizeof(uint32_t));
    if (e == cudaSuccess && double_support) e = cudaEventCreateWithFlags(&p->narrow_done, cudaEventDisableTiming);
    if (e != cudaSuccess) {
        if (p->d_err) cudaFree(p->d_err);
        delete p;
        return cuda_fail(e, "htc_program_create");
    }
    p->max_smem -= 1024;   // static shared memory of the kernels
    int rc = recipe == HTC_RECIPE_HY ? set_smem_attr<RECIPE_HY>(p->max_smem) : set_smem_attr<RECIPE_EU>(p->max_smem);
    if (rc) {
        cudaFree(p->d_err);
        if (p->narrow_done) cudaEventDestroy(p->narrow_done);
        delete p;
        return rc;
    }
    p->device = pool_enter(dev);
    *out = p;
    return HTC_OK;
}

void htc_program_destroy(htc_program *p) {
    if (!p) return;
    cudaFree(p->d_err);
    if (p->wave_buf) cudaFree(p->wave_buf);
    if (p->d_wave_ctr) cudaFree(p->d_wave_ctr);
    if (p->sort_buf) cudaFree(p->sort_buf);
    if (p->image) cudaFree(p->image);
    pool_leave(p->device);
    if (p->narrow_buf) cudaFree(p->narrow_buf);
    if (p->narrow_done) cudaEventDestroy(p->narrow_done);
    if (p->generic) generic_program_destroy(p->generic);
    delete p;
}

int htc_program_build(const char *scene_type, uint32_t light_hops, int address_width, uint32_t flags, char *log,
                      size_t log_len, htc_program **out) {
    if (!out) return fail(HTC_ERR_INVALID, "out is NULL");
    *out = nullptr;
    if (!scene_type || !scene_type[0]) return fail(HTC_ERR_INVALID, "scene_type is empty");
    if (light_hops == 0) return fail(HTC_ERR_INVALID, "light_hops must be positive");
    if (address_width != 32 && address_width != 64) return fail(HTC_ERR_INVALID, "address_width must be 32 or 64");
    if (flags & ~HTC_FLAG_JITTER_YX) return fail(HTC_ERR_INVALID, "unknown program flags");
    GenericProgram *g = nullptr;
    int rc = generic_program_build(scene_type, address_width, log, log_len, &g);
    if (rc) return rc;
    return wrap_generic(g, HTC_RECIPE_CUSTOM, light_hops, address_width, flags, out);
}

int htc_program_static_size(const htc_program *p, uint64_t *bytes) {
    int rc = check_program(p);
    if (rc) return rc;
    if (!bytes) return fail(HTC_ERR_INVALID, "bytes is NULL");
    if (p->generic) *bytes = generic_min_size(p->generic);
    else if (p->double_support) *bytes = NARROW_SRC_OBJECTS[p->recipe == HTC_RECIPE_HY ? 0 : 1];
    else *bytes = p->recipe == HTC_RECIPE_HY ? Layout<RECIPE_HY>::OBJECTS : Layout<RECIPE_EU>::OBJECTS;
    return HTC_OK;
}

int htc_program_check(htc_program *p, void *stream) {
    int rc = check_program(p);
    if (rc) return rc;
    uint32_t err = 0;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    HTC_CUDA(cudaMemcpyAsync(&err, p->d_err, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    HTC_CUDA(cudaStreamSynchronize(st));
    if (err) {
        HTC_CUDA(cudaMemsetAsync(p->d_err, 0, sizeof(uint32_t), st));
        HTC_CUDA(cudaStreamSynchronize(st));
        if (err & ERR_SCENE) return fail(HTC_ERR_SCENE, "scene bytes failed validation (object count or shape index out of range)");
        return fail(HTC_ERR_SCENE, "device error word set");
    }
    return HTC_OK;
}

int htc_malloc(void **dptr, size_t bytes) {
    if (!dptr) return fail(HTC_ERR_INVALID, "dptr is NULL");
    HTC_CUDA(cudaMalloc(dptr, bytes ? bytes : 1));
    return HTC_OK;
}
int htc_free(void *dptr) {
    HTC_CUDA(cudaFree(dptr));
    return HTC_OK;
}
int htc_memcpy_htod(void *dst, const void *src, size_t bytes, void *stream) {
    HTC_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, reinterpret_cast<cudaStream_t>(stream)));
    return HTC_OK;
}
int htc_memcpy_dtoh(void *dst, const void *src, size_t bytes, void *stream) {
    HTC_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, reinterpret_cast<cudaStream_t>(stream)));
    return HTC_OK;
}
int htc_memset(void *dst, int value, size_t bytes, void *stream) {
    HTC_CUDA(cudaMemsetAsync(dst, value, bytes, reinterpret_cast<cudaStream_t>(stream)));
    return HTC_OK;
}
int htc_stream_sync(void *stream) {
    HTC_CUDA(cudaStreamSynchronize(reinterpret_cast<cudaStream_t>(stream)));
    return HTC_OK;
}

// Argument checks and launch of a generic scene program (passes samples per pixel).
static int render_generic_program(htc_program *p, uint32_t W, uint32_t H, const void *scene, size_t scene_size,
                                  float *canvas, uint32_t *seeds, uint32_t passes, uint64_t *stats, void *stream) {
    if (W == 0 || H == 0) return fail(HTC_ERR_INVALID, "canvas width and height must be positive");
    if ((uint64_t)W * (uint64_t)H >= 0xFFFFFFFFull) return fail(HTC_ERR_INVALID, "canvas too large (W*H must fit in 32 bits)");
    if (!scene || !canvas || !seeds) return fail(HTC_ERR_INVALID, "scene, canvas and seeds must be device pointers");
    if ((reinterpret_cast<uintptr_t>(scene) & 31u) != 0 || (reinterpret_cast<uintptr_t>(canvas) & 15u) != 0)
        return fail(HTC_ERR_INVALID, "scene must be 32-byte and canvas 16-byte aligned");
    if (passes == 0) return HTC_OK;
    return generic_render(p->generic, W, H, p->hops, p->flags, scene, scene_size, canvas, seeds, passes, stats,
                          p->d_err, stream);
}

}  // extern "C"

// A call's use of the program's narrowed scene. Its launches read that one buffer to the end, so the
// uses of several streams and threads follow one another: the next call's stream waits for the event
// that ends this one. (On a capturing stream there is no event outside the capture to wait for: such a
// call, and the replays of its graph, are the caller's to keep apart, as the header says.)
struct NarrowUse {
    htc_program *p = nullptr;
    cudaStream_t st = nullptr;
    std::unique_lock<std::mutex> lock;
    ~NarrowUse() {
        if (p) cudaEventRecord(p->narrow_done, st);
    }
};
static bool capturing(cudaStream_t st) {   // or cannot be told
    cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &s) == cudaSuccess) return s != cudaStreamCaptureStatusNone;
    cudaGetLastError();
    return true;
}

// A double_support program's scene, narrowed on `stream` into the program's f32-layout buffer
// (k_narrow_scene); *scene / *scene_size then name that buffer, which is the call's until `use` ends.
// Other programs: unchanged.
static int narrow_scene(htc_program *p, const void **scene, size_t *scene_size, void *stream, NarrowUse &use) {
    if (!p || !p->double_support) return HTC_OK;
    const int li = p->recipe == HTC_RECIPE_HY ? 0 : 1;
    if (!*scene) return fail(HTC_ERR_INVALID, "scene must be a device pointer");
    if ((reinterpret_cast<uintptr_t>(*scene) & 15u) != 0) return fail(HTC_ERR_INVALID, "scene must be 16-byte aligned");
    if (*scene_size < NARROW_SRC_OBJECTS[li])
        return fail(HTC_ERR_SCENE, "scene buffer is smaller than the scene header (double_support layout)");
    uint64_t cap = (*scene_size - NARROW_SRC_OBJECTS[li]) / NARROW_SRC_STRIDE[li];
    if (cap > 0xFFFFFFull) cap = 0xFFFFFFull;
    const size_t dst_objects = li == 0 ? Layout<RECIPE_HY>::OBJECTS : Layout<RECIPE_EU>::OBJECTS;
    const size_t bytes = dst_objects + (size_t)cap * OBJ_STRIDE;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    use.lock = std::unique_lock<std::mutex>(p->narrow_mutex);
    if (!capturing(st)) {
        HTC_CUDA(cudaStreamWaitEvent(st, p->narrow_done, 0));
        use.p = p;
        use.st = st;
    }
    if (p->narrow_bytes < bytes) {
        if (p->narrow_buf) HTC_CUDA(cudaFree(p->narrow_buf));
        p->narrow_buf = nullptr;
        p->narrow_bytes = 0;
        HTC_CUDA(cudaMalloc(&p->narrow_buf, bytes));
        HTC_CUDA(cudaMemsetAsync(p->narrow_buf, 0, bytes, st));   // the layout's padding
        p->narrow_bytes = bytes;
    }
    const uint32_t records = (uint32_t)cap + 1u;
    const unsigned blocks = std::min<unsigned>((records + 127u) / 128u, 148u * 8u);
    k_narrow_scene<<<blocks, 128, 0, st>>>(li, reinterpret_cast<const uint8_t *>(*scene), *scene_size, p->narrow_buf,
                                           (uint32_t)cap, p->address_width / 8);
    HTC_CUDA(cudaGetLastError());
    *scene = p->narrow_buf;
    *scene_size = bytes;
    return HTC_OK;
}

// One pass with the one-pass kernel (checked arguments).
constexpr uint32_t PLAIN_ROWS = 4u * 65535u;   // 4 rows a block, 65535 blocks
static int render_plain_pass(htc_program *p, uint32_t W, uint32_t H, const void *scene, size_t scene_size, uint32_t max_objects,
                             size_t smem, float *canvas, uint32_t *seeds, uint64_t *stats, void *stream) {
    dim3 grid((W + 31) / 32, (H + 3) / 4);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const uint8_t *sc = reinterpret_cast<const uint8_t *>(scene);
    float4 *cv = reinterpret_cast<float4 *>(canvas);
    if (p->recipe == HTC_RECIPE_HY)
        render_plain<RECIPE_HY><<<grid, 128, smem, st>>>(sc, scene_size, max_objects, p->address_width, W, H,
                                                         p->hops, p->flags, cv, seeds, stats, p->d_err);
    else
        render_plain<RECIPE_EU><<<grid, 128, smem, st>>>(sc, scene_size, max_objects, p->address_width, W, H,
                                                         p->hops, p->flags, cv, seeds, stats, p->d_err);
    HTC_CUDA(cudaGetLastError());
    return HTC_OK;
}


// Whether a call's hyperbolic wavefronts are sorted between hop depths. The two sort launches
// cost 15 us per depth on small queues and 50 us on 2 M paths; below 2^19 pixels or 100 objects
// coherence saves less. Measured, sorted / in queue order, us per pass: 1080p / 200 objects (4.7 hops
// a path) 2764 / 3029, (2.0 hops) 1232 / 1245, 720p / 120 objects 1483 / 1542, 720p / 77 objects 721 / 708,
// 1080p / 18 objects 1082 / 1070, 640x480 / 200 objects 471 / 396.
static bool wave_sorted(const htc_program *p, uint64_t pixels, uint32_t max_objects) {
    return p->recipe == HTC_RECIPE_HY && !(p->flags & HTC_FLAG_NO_SORT) && pixels >= (1u << 19) && max_objects >= 100;
}
// Queues of W*H slots each (a hop never has more paths than pixels), the hop counters and the scene's
// image; allocated on the first call that needs more and kept with the program. They go by the canvas
// alone, whatever the scene, and the sort's buffer, which comes with the first call that sorts, by the
// queues: a call on a canvas no larger than an earlier one's frees nothing that a captured call's graph
// works in, and can be captured itself (if none sorted before it, it takes its paths in queue order).
static bool wave_reserved(const htc_program *p, size_t slots) { return p->image && p->d_wave_ctr && p->wave_slots >= slots; }
static int wave_reserve(htc_program *p, size_t slots, bool sorted) {
    if (!p->image) HTC_CUDA(cudaMalloc(&p->image, sizeof(float4) * (1 + (size_t)p->max_smem / 16)));   // image_words of the largest scene
    if (!p->d_wave_ctr) {
        // 2 words per hop depth, two sets
        HTC_CUDA(cudaMalloc(&p->d_wave_ctr, 4 * sizeof(uint32_t) * (size_t)p->hops));
    }
    slots = (slots + 63) & ~(size_t)63;   // keeps the second queue and every array 16-byte aligned
    if (p->wave_slots < slots) {
        if (p->sort_buf) HTC_CUDA(cudaFree(p->sort_buf));
        p->sort_buf = nullptr;
        if (p->wave_buf) HTC_CUDA(cudaFree(p->wave_buf));
        p->wave_buf = nullptr;
        p->wave_slots = 0;
        HTC_CUDA(cudaMalloc(&p->wave_buf, 2 * WAVE_SLOT_BYTES * slots));
        p->wave_slots = slots;
    }
    if (sorted && !p->sort_buf) HTC_CUDA(cudaMalloc(&p->sort_buf, sort_bytes(p->wave_slots, (uint32_t)p->num_sms)));
    return HTC_OK;
}
// What one call's launches work in: the program's own buffers, or a block of the device's pool.
struct WaveWork {
    float4 *image;
    uint32_t *ctr;      // 4 words per hop depth
    void *sort;         // NULL: the paths stay in queue order
    void *queues;
    size_t slots;       // per queue, and of the sort's buffer
};
static WaveWork wave_work_owned(const htc_program *p, bool sorted) {
    return WaveWork{p->image, p->d_wave_ctr, sorted ? p->sort_buf : nullptr, p->wave_buf, p->wave_slots};
}
// The same laid out in one block at `base`; returns its size.
static size_t wave_work_block(const htc_program *p, uint64_t pixels, uint32_t max_objects, uint8_t *base, WaveWork *w) {
    const size_t slots = (size_t)((pixels + 63) & ~(uint64_t)63);
    size_t at = 0;
    const auto take = [&](size_t bytes) {
        uint8_t *r = base + at;
        at += (bytes + 255) & ~(size_t)255;
        return r;
    };
    w->image = reinterpret_cast<float4 *>(take(sizeof(float4) * image_words(max_objects)));
    w->ctr = reinterpret_cast<uint32_t *>(take(4 * sizeof(uint32_t) * (size_t)p->hops));
    w->sort = wave_sorted(p, pixels, max_objects) ? take(sort_bytes(slots, (uint32_t)p->num_sms)) : nullptr;
    w->queues = take(2 * WAVE_SLOT_BYTES * slots);
    w->slots = slots;
    return at;
}
static WaveQueue wave_queue(const WaveWork &w, int which) {
    const size_t n = w.slots;
    uint8_t *b = reinterpret_cast<uint8_t *>(w.queues) + (size_t)which * WAVE_SLOT_BYTES * n;
    WaveQueue q;
    q.p = reinterpret_cast<float4 *>(b);
    q.v = q.p + n;
    q.t = q.v + n;
    q.e = q.t + n;
    q.h = reinterpret_cast<uint32_t *>(q.e + n);
    q.o = nullptr;
    return q;
}
template <int R>
static int launch_wave(const htc_program *p, const WaveWork &w, uint32_t W, uint32_t H, const uint8_t *sc, size_t scene_size,
                       uint32_t max_objects, size_t smem, float4 *cv, uint32_t *seeds, uint32_t passes,
                       uint64_t *stats, cudaStream_t st) {
    int per_sm = 0;
    // a grid per kernel: the hop-0 and later-hop kernels have register caps of their own
    int per_sm0 = 0;
    HTC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, render_wave<R, 2>, 128, smem));
    HTC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm0, render_wave<R, 1>, 128, smem));
    if (per_sm < 1) per_sm = 1;
    if (per_sm0 < 1) per_sm0 = 1;
    const uint64_t needed = ((uint64_t)W * H + 127) / 128;
    const uint64_t blocks = std::min<uint64_t>((uint64_t)per_sm * (uint64_t)p->num_sms, needed);
    const uint64_t blocks0 = std::min<uint64_t>((uint64_t)per_sm0 * (uint64_t)p->num_sms, needed);
    const WaveQueue q[2] = {wave_queue(w, 0), wave_queue(w, 1)};
    const WaveQueue none = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    const bool sorted = w.sort != nullptr;
    const unsigned sort_blocks = (unsigned)p->num_sms;
    const SortBuf sb = sorted ? sort_buf_at(w.sort, w.slots, sort_blocks) : SortBuf{};
    const size_t sort_smem = sizeof(uint32_t) * SORT_BINS;
    uint32_t sorts = 0;   // both histograms start cleared; k_sort_scatter clears the one its depth did not use
    if (sorted) HTC_CUDA(cudaMemsetAsync(sb.hist, 0, 2 * sizeof(uint32_t) * SORT_BINS, st));
    // two sets of counters in turn: a pass's hop 0 clears the next one's
    const uint32_t n_ctr = 2 * p->hops;
    HTC_CUDA(cudaMemsetAsync(w.ctr, 0, 2 * sizeof(uint32_t) * (size_t)n_ctr, st));
    k_stage<R><<<1, STAGE_THREADS, 0, st>>>(sc, scene_size, max_objects, p->address_width, p->d_err, w.image);
    HTC_CUDA(cudaGetLastError());
    for (uint32_t pass = 0; pass < passes; ++pass) {
        uint32_t *ctr = w.ctr + (size_t)(pass & 1u) * n_ctr, *next = w.ctr + (size_t)(~pass & 1u) * n_ctr;
        for (uint32_t h = 0; h < p->hops; ++h) {
            WaveQueue in = h == 0 ? none : q[(h - 1) & 1];
            const uint32_t *in_count = h == 0 ? nullptr : ctr + 2 * (h - 1) + 1;
            if (sorted && h > 0) {
                uint32_t *hist = sb.hist + (sorts & 1u) * SORT_BINS, *other = sb.hist + (~sorts & 1u) * SORT_BINS;
                ++sorts;
                HTC_CUDA(launch(false, k_sort_keys, sort_blocks, SORT_THREADS, sort_smem, st, in.p, in.v, in_count, hist, sb.place, sb.key));
                HTC_CUDA(launch(true, k_sort_scatter, sort_blocks, SORT_THREADS, sort_smem, st, sb.key, in_count, hist, other, sb.place, sb.perm));
                in.o = sb.perm;
            }
            HTC_CUDA(launch(true, h == 0 ? render_wave<R, 1> : render_wave<R, 2>, (unsigned)(h == 0 ? blocks0 : blocks),
                            BLOCK_THREADS, smem, st, w.image, sc, max_objects, pass + h > 0, W, H, p->hops, h, p->flags, cv, seeds,
                            stats, in, in_count, q[h & 1], ctr + 2 * h, next, n_ctr));
        }
    }
    return HTC_OK;
}

static int launch_wave_any(const htc_program *p, const WaveWork &w, uint32_t W, uint32_t H, const void *scene, size_t scene_size,
                           uint32_t max_objects, size_t smem, float *canvas, uint32_t *seeds, uint32_t passes, uint64_t *stats,
                           cudaStream_t st) {
    const uint8_t *sc = reinterpret_cast<const uint8_t *>(scene);
    float4 *cv = reinterpret_cast<float4 *>(canvas);
    return p->recipe == HTC_RECIPE_HY
        ? launch_wave<RECIPE_HY>(p, w, W, H, sc, scene_size, max_objects, smem, cv, seeds, passes, stats, st)
        : launch_wave<RECIPE_EU>(p, w, W, H, sc, scene_size, max_objects, smem, cv, seeds, passes, stats, st);
}

// Whether one pass is faster as wavefronts than with the one-pass kernel. Small canvases leave the
// deeper hop launches most of the GPU idle; a hop count beyond the workloads' would add launches
// for queues that are empty. Measured, one call of one pass, one-pass kernel / wavefronts in us:
// hyperbolic scenes of 18, 77, 200 objects at 400x300 126/139, 217/245, 268/300, at 512x384 176/166,
// 333/297, 402/337, at 800x600 346/297, 646/467, 821/456, of 2, 4 and 8 objects at 512x384 26/46, 67/104,
// 218/193, at 800x600 47/56, 129/140, 454/360, at 1280x720 88/84, 228/204, 791/594; Euclidean scenes of 9,
// 17, 25, 33 objects at 800x600 62/86, 118/130, 121/138, 190/217, at 1024x768 89/105, 177/163, 179/172,
// 281/255.
constexpr uint32_t WAVE_MAX_HOPS = 16, EU_WAVE_OBJECTS = 16, WAVE_PIXELS = 9u << 14;
static bool wave_pays(const htc_program *p, uint64_t pixels, uint32_t max_objects) {
    if (p->hops > WAVE_MAX_HOPS) return false;
    return p->recipe == HTC_RECIPE_HY ? pixels >= (max_objects < 6 ? 3u << 18 : WAVE_PIXELS) : pixels >= (3u << 18) && max_objects >= EU_WAVE_OBJECTS;
}

// Wavefronts in a workspace taken from the device's pool and given back in stream order, so that
// calls of one program on several streams or threads do not meet (in the scene of a double_support
// program they would: NarrowUse). *done = false: none was to be
// had (no memory, a capturing stream); nothing was launched.
static int render_wave_pooled(htc_program *p, uint32_t W, uint32_t H, const void *scene, size_t scene_size, uint32_t max_objects,
                              size_t smem, float *canvas, uint32_t *seeds, uint32_t passes, uint64_t *stats, cudaStream_t st,
                              bool *done) {
    *done = false;
    if (capturing(st)) return HTC_OK;
    WaveWork w;
    const size_t bytes = wave_work_block(p, (uint64_t)W * H, max_objects, nullptr, &w);
    void *block = pool_take(p->device, bytes, H > PLAIN_ROWS ? 0xFFFFFFFFu : passes, st);   // the one-pass kernel ends there
    if (!block) return HTC_OK;
    *done = true;
    wave_work_block(p, (uint64_t)W * H, max_objects, reinterpret_cast<uint8_t *>(block), &w);
    const int rc = launch_wave_any(p, w, W, H, scene, scene_size, max_objects, smem, canvas, seeds, passes, stats, st);
    const cudaError_t e = pool_give(block, st);
    return rc ? rc : e != cudaSuccess ? cuda_fail(e, "cudaFreeAsync") : HTC_OK;
}

static int render_wavefront_impl(htc_program *p, uint32_t W, uint32_t H, const void *scene, size_t scene_size,
                                 float *canvas, uint32_t *seeds, uint32_t passes, uint64_t *stats, void *stream) {
    if (p && p->generic) return fail(HTC_ERR_UNSUPPORTED, "the wavefront form serves the built-in recipes only");
    uint32_t max_objects = 0;
    size_t smem = 0;
    int rc = validate_render_args(p, W, H, scene, scene_size, canvas, seeds, &max_objects, &smem);
    if (rc) return rc;
    if (passes == 0) return HTC_OK;
    const bool sorted = wave_sorted(p, (uint64_t)W * H, max_objects);
    rc = wave_reserve(p, (size_t)W * H, sorted && !(wave_reserved(p, (size_t)W * H) && capturing(reinterpret_cast<cudaStream_t>(stream))));
    if (rc) return rc;
    return launch_wave_any(p, wave_work_owned(p, sorted), W, H, scene, scene_size, max_objects, smem, canvas, seeds, passes, stats,
                           reinterpret_cast<cudaStream_t>(stream));
}

extern "C" {

int htc_render_ex(htc_program *p, uint32_t W, uint32_t H, const void *scene, size_t scene_size,
                  float *canvas, uint32_t *seeds, uint64_t *stats, void *stream) {
    if (p && p->generic) return render_generic_program(p, W, H, scene, scene_size, canvas, seeds, 1, stats, stream);
    NarrowUse narrow;
    if (p && canvas && seeds && W && H) {   // argument errors are reported by the render checks
        int rc = narrow_scene(p, &scene, &scene_size, stream, narrow);
        if (rc) return rc;
    }
    uint32_t max_objects = 0;
    size_t smem = 0;
    int rc = validate_render_args(p, W, H, scene, scene_size, canvas, seeds, &max_objects, &smem);
    if (rc) return rc;
    if (wave_pays(p, (uint64_t)W * H, max_objects)) {
        bool done = false;
        rc = render_wave_pooled(p, W, H, scene, scene_size, max_objects, smem, canvas, seeds, 1, stats,
                                reinterpret_cast<cudaStream_t>(stream), &done);
        if (rc || done) return rc;
    }
    return render_plain_pass(p, W, H, scene, scene_size, max_objects, smem, canvas, seeds, stats, stream);
}

int htc_render(htc_program *p, uint32_t W, uint32_t H, const void *scene, size_t scene_size, float *canvas,
               uint32_t *seeds, void *stream) {
    return htc_render_ex(p, W, H, scene, scene_size, canvas, seeds, nullptr, stream);
}

int htc_render_wavefront(htc_program *p, uint32_t W, uint32_t H, const void *scene, size_t scene_size,
                         float *canvas, uint32_t *seeds, uint32_t passes, uint64_t *stats, void *stream) {
    NarrowUse narrow;
    if (p && canvas && seeds && W && H && passes) {
        int rc = narrow_scene(p, &scene, &scene_size, stream, narrow);
        if (rc) return rc;
    }
    return render_wavefront_impl(p, W, H, scene, scene_size, canvas, seeds, passes, stats, stream);
}

int htc_render_passes(htc_program *p, uint32_t W, uint32_t H, const void *scene, size_t scene_size,
                      float *canvas, uint32_t *seeds, uint32_t passes, uint64_t *stats, void *stream) {
    if (p && p->generic) return render_generic_program(p, W, H, scene, scene_size, canvas, seeds, passes, stats, stream);
    NarrowUse narrow;
    if (p && canvas && seeds && W && H && passes) {
        int rc = narrow_scene(p, &scene, &scene_size, stream, narrow);
        if (rc) return rc;
    }
    uint32_t max_objects = 0;
    size_t smem = 0;
    int rc = validate_render_args(p, W, H, scene, scene_size, canvas, seeds, &max_objects, &smem);
    if (rc) return rc;
    if (passes == 0) return HTC_OK;
    // The program keeps queues of its own for large canvases and, where wavefronts pay at all, for
    // hyperbolic scenes of 100 objects on (200 objects, us per pass, one-pass kernel / wavefronts: 320x240
    // 190/252, 400x300 260/280); the other calls may run on several streams at once and work in the pool.
    const uint64_t pixels = (uint64_t)W * H;
    // Several passes pay for wavefronts on smaller canvases than one does, since the staging is shared and the
    // launches overlap: 2^19 pixels for hyperbolic scenes of any size and Euclidean ones of 16 objects on
    // (1024x520 and 1024x700, us of 8 passes, one-pass kernel / wavefronts: hyperbolic 1, 2, 4, 5 objects
    // 343/291, 2210/2519, 1370/1280, 2958/2680 and 440/341, 2930/3301, 1722/1539, 4277/3808; Euclidean 16, 25, 33
    // 731/843, 1217/1166, 1388/1314 and 970/988, 1592/1358, 1942/1619). Euclidean scenes of fewer objects need
    // more pixels (us per pass, 3 and 9 objects: 1024x768 80/91 and 83/93, 1440x900 122/123 and 125/124).
    // The one-pass kernel's grid ends at PLAIN_ROWS rows.
    const bool few = p->recipe == HTC_RECIPE_EU && max_objects < EU_WAVE_OBJECTS && H <= PLAIN_ROWS;
    const bool own = pixels >= (few ? 5u << 18 : 1u << 19) || (p->recipe == HTC_RECIPE_HY && max_objects >= 100 && pixels >= WAVE_PIXELS);
    if (own && (wave_reserved(p, pixels) || !capturing(reinterpret_cast<cudaStream_t>(stream))))
        return render_wavefront_impl(p, W, H, scene, scene_size, canvas, seeds, passes, stats, stream);
    if (wave_pays(p, pixels, max_objects)) {
        bool done = false;
        rc = render_wave_pooled(p, W, H, scene, scene_size, max_objects, smem, canvas, seeds, passes, stats,
                                reinterpret_cast<cudaStream_t>(stream), &done);
        if (rc || done) return rc;
    }
    for (uint32_t k = 0; k < passes; ++k) {
        rc = render_plain_pass(p, W, H, scene, scene_size, max_objects, smem, canvas, seeds, stats, stream);
        if (rc) return rc;
    }
    return HTC_OK;
}

static unsigned post_blocks(uint32_t n) {
    uint32_t b = (n + 255) / 256;
    return b > 148u * 16u ? 148u * 16u : (b ? b : 1u);
}

int htc_extract(uint32_t W, uint32_t H, uint32_t passes, const float *canvas, float *image, void *stream) {
    if (!canvas || !image || passes == 0) return fail(HTC_ERR_INVALID, "bad extract arguments");
    uint32_t n = W * H;
    k_extract<<<post_blocks(n), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        n, (float)passes, reinterpret_cast<const float4 *>(canvas), reinterpret_cast<float4 *>(image));
    HTC_CUDA(cudaGetLastError());
    return HTC_OK;
}
int htc_gamma(uint32_t W, uint32_t H, float gamma, const float *input, float *output, void *stream) {
    if (!input || !output) return fail(HTC_ERR_INVALID, "bad gamma arguments");
    uint32_t n = W * H;
    k_gamma<<<post_blocks(n), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        n, gamma, reinterpret_cast<const float4 *>(input), reinterpret_cast<float4 *>(output));
    HTC_CUDA(cudaGetLastError());
    return HTC_OK;
}
int htc_pack(uint32_t W, uint32_t H, const float *image, uint8_t *packed, void *stream) {
    if (!image || !packed) return fail(HTC_ERR_INVALID, "bad pack arguments");
    uint32_t n = W * H;
    k_pack<<<post_blocks(n), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        n, reinterpret_cast<const float4 *>(image), reinterpret_cast<uchar4 *>(packed));
    HTC_CUDA(cudaGetLastError());
    return HTC_OK;
}
int htc_extract_gamma_pack(uint32_t W, uint32_t H, uint32_t passes, float gamma, const float *canvas,
                           uint8_t *packed, void *stream) {
    if (!canvas || !packed || passes == 0) return fail(HTC_ERR_INVALID, "bad extract_gamma_pack arguments");
    uint32_t n = W * H;
    k_extract_gamma_pack<<<post_blocks(n), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        n, (float)passes, gamma, reinterpret_cast<const float4 *>(canvas), reinterpret_cast<uchar4 *>(packed));
    HTC_CUDA(cudaGetLastError());
    return HTC_OK;
}

int htc_fill_seeds(uint32_t *seeds, uint32_t n, uint32_t global_seed, uint32_t offset, void *stream) {
    if (!seeds && n) return fail(HTC_ERR_INVALID, "seeds is NULL");
    if (n == 0) return HTC_OK;
    k_fill_seeds<<<post_blocks(n), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(n, global_seed, offset, seeds);
    HTC_CUDA(cudaGetLastError());
    return HTC_OK;
}

// ---------------------------------------------------------------- batches
}  // extern "C"

struct htc_batch {
    uint32_t max_views;
    BatchView *d_views;
    uint32_t *d_err;
    uint32_t smem_objects;
    uint32_t blocks_per_sm;
    uint32_t tile_pixels;
    int num_sms, max_smem;
    cudaGraph_t graph;
    cudaGraphExec_t graph_exec;
    uint64_t *graph_stats;   // the stats buffer the graph's launches write
    std::vector<BatchView> h_views;
    // Two pinned staging slots for the asynchronous descriptor upload; slot i may be
    // rewritten once its last copy (event staged[i]) has run.
    BatchView *p_views[2];
    cudaEvent_t staged[2];
    int slot;
    // wavefront form: view order (expensive first), queues, counters
    uint32_t *d_order;
    uint32_t *p_order[2];
    uint32_t n_views, n_order, n_hy, n_eu, hops_max, passes_max;
    void *wave_buf;
    uint64_t wave_slots;     // slots per queue
    uint32_t *d_wcnt;
    size_t wcnt_words;
    float4 *images;          // the views' scene images
    size_t image_words;
    std::vector<float4 *> old_images;   // smaller ones, which launches and graphs may still read
    void *sort_buf;          // coherence sort of the hyperbolic views (BatchSortBuf)
    uint64_t sort_slots;     // = wave_slots when allocated
    uint32_t hops_of[2], passes_of[2];   // the most of the hyperbolic, of the Euclidean views
    cudaStream_t side;       // where the Euclidean launches run beside the hyperbolic ones
    cudaEvent_t forked, joined;
};
// Counters of one recipe and pass: every view's paths by hop, then the tiles taken by hop.
constexpr size_t batch_counters(uint32_t n_views, uint32_t hops) { return ((size_t)n_views + 1) * hops; }
static_assert(batch_counters(4096, 0xFFFFFFFFu) == 4097ull * 0xFFFFFFFFull && batch_counters(0xFFFFFFFFu, 1) == 1ull << 32, "counted in 64 bits");

static void batch_free(htc_batch *b) {
    if (!b) return;
    for (int i = 0; i < 2; ++i) {
        if (b->staged[i]) {
            cudaEventSynchronize(b->staged[i]);
            cudaEventDestroy(b->staged[i]);
        }
        if (b->p_views[i]) cudaFreeHost(b->p_views[i]);
        if (b->p_order[i]) cudaFreeHost(b->p_order[i]);
    }
    if (b->forked) cudaEventDestroy(b->forked);
    if (b->joined) cudaEventDestroy(b->joined);
    if (b->side) cudaStreamDestroy(b->side);
    if (b->d_order) cudaFree(b->d_order);
    if (b->wave_buf) cudaFree(b->wave_buf);
    if (b->d_wcnt) cudaFree(b->d_wcnt);
    if (b->sort_buf) cudaFree(b->sort_buf);
    if (b->images) cudaFree(b->images);
    for (float4 *old : b->old_images) cudaFree(old);
    if (b->graph_exec) cudaGraphExecDestroy(b->graph_exec);
    if (b->graph) cudaGraphDestroy(b->graph);
    cudaFree(b->d_views);
    cudaFree(b->d_err);
    delete b;
}

template <int RF>
static cudaError_t batch_wave_smem_attr(int smem) {
    cudaError_t e = cudaFuncSetAttribute(render_batch_wave<RF, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(render_batch_wave<RF, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    return e;
}

template <int RF>
static int batch_wave_blocks(htc_batch *b, size_t smem, unsigned *blocks) {
    int per_sm = 0;
    HTC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, render_batch_wave<RF, 2>, 128, smem));
    if (b->blocks_per_sm && (int)b->blocks_per_sm < per_sm) per_sm = (int)b->blocks_per_sm;
    if (per_sm < 1) per_sm = 1;
    *blocks = (unsigned)per_sm * (unsigned)b->num_sms;
    return HTC_OK;
}

// The launches of a batch. The two geometries share nothing but the stage before them, so the
// Euclidean ones run on a stream of their own beside the hyperbolic ones (`st_eu`), and fill
// what those leave of the chip at the end of every launch and while few paths are left; within a
// stream the launches overlap at their edges, except with the sort's first kernel: its 148
// large blocks would crowd on the multiprocessors that are free first. 24 mixed views: 35.34 ms one
// after another, 34.54 on two streams, 34.65 with the overlap as well; a server's steps of 1 to 4
// views (12 requests) 52.7, 50.7 and 49.95; the sort's first kernel overlapping too 34.8 and 50.4.
static int batch_passes(htc_batch *b, const WaveQueue (&q)[2], unsigned blocks_hy, unsigned blocks_eu, size_t smem, uint32_t n_seg,
                        uint64_t *stats, cudaStream_t st, cudaStream_t st_eu) {
    // each geometry has counters of its own, in two sets: a pass's hop 0 clears the next one's
    const size_t words = batch_counters(b->n_views, b->hops_max);
    const uint32_t *order_hy = b->d_order + b->n_order, *order_eu = order_hy + b->n_hy;
    const unsigned sort_blocks = (unsigned)b->num_sms;
    const BatchSortBuf sb = n_seg ? batch_sort_at(b->sort_buf, b->sort_slots, sort_blocks) : BatchSortBuf{};
    const size_t sort_smem = sizeof(uint32_t) * (SORT_BINS + 2 * n_seg + 1);
    uint32_t sorts = 0;   // both sets of histograms start cleared; k_bsort_scatter clears the one its depth did not use
    for (uint32_t pass = 0; pass < b->passes_max; ++pass) {
        uint32_t *set = b->d_wcnt + (pass & 1u) * words, *next = b->d_wcnt + (~pass & 1u) * words;
        for (uint32_t h = 0; h < b->hops_max; ++h) {
            const WaveQueue &in = q[(h + 1) & 1], &out = q[h & 1];
            uint32_t *cnt = set, *grab = cnt + (size_t)b->n_views * b->hops_max + h;
            if (pass < b->passes_of[0] && h < b->hops_of[0]) {
                WaveQueue in_hy = in;
                if (n_seg && h > 0) {
                    uint32_t *hist = sb.hist + (size_t)(sorts & 1u) * BATCH_SORT_VIEWS * SORT_BINS;
                    uint32_t *other = sb.hist + (size_t)(~sorts & 1u) * BATCH_SORT_VIEWS * SORT_BINS;
                    ++sorts;
                    HTC_CUDA(launch(false, k_bsort_keys, sort_blocks, SORT_THREADS, sort_smem, st, b->d_views, order_hy, n_seg, b->n_views, pass, h,
                                    cnt, in.p, in.v, hist, sb.place, sb.key));
                    HTC_CUDA(launch(true, k_bsort_scatter, sort_blocks, SORT_THREADS, sort_smem, st, b->d_views, order_hy, n_seg, b->n_views, pass, h,
                                    cnt, sb.key, hist, other, sb.place, sb.perm));
                    in_hy.o = sb.perm;
                }
                HTC_CUDA(launch(true, h == 0 ? render_batch_wave<RECIPE_HY, 1> : render_batch_wave<RECIPE_HY, 2>, blocks_hy, 128, smem, st,
                                b->d_views, order_hy, b->n_hy, b->n_views, pass, h, b->tile_pixels, b->smem_objects, in_hy, out, cnt, grab,
                                stats, n_seg, next, words));
            }
            if (pass < b->passes_of[1] && h < b->hops_of[1]) {
                cnt += 2 * words;
                HTC_CUDA(launch(true, h == 0 ? render_batch_wave<RECIPE_EU, 1> : render_batch_wave<RECIPE_EU, 2>, blocks_eu, 128, smem, st_eu,
                                b->d_views, order_eu, b->n_eu, b->n_views, pass, h, b->tile_pixels, b->smem_objects, in, out, cnt, grab + 2 * words,
                                stats, 0u, next + 2 * words, words));
            }
        }
    }
    return HTC_OK;
}

static int batch_launch_wave(htc_batch *b, uint64_t *stats, cudaStream_t st) {
    if (b->n_order == 0) return HTC_OK;
    const size_t smem = smem_bytes(b->smem_objects) + sizeof(uint32_t) * ((size_t)b->n_views + 1);
    WaveQueue q[2];
    for (int k = 0; k < 2; ++k) {
        uint8_t *base = reinterpret_cast<uint8_t *>(b->wave_buf) + (size_t)k * WAVE_SLOT_BYTES * b->wave_slots;
        const uint64_t n = b->wave_slots;
        q[k].p = reinterpret_cast<float4 *>(base);
        q[k].v = q[k].p + n;
        q[k].t = q[k].v + n;
        q[k].e = q[k].t + n;
        q[k].h = reinterpret_cast<uint32_t *>(q[k].e + n);
        q[k].o = nullptr;
    }
    unsigned blocks_hy = 0, blocks_eu = 0;
    int rc = batch_wave_blocks<RECIPE_HY>(b, smem, &blocks_hy);
    if (!rc) rc = batch_wave_blocks<RECIPE_EU>(b, smem, &blocks_eu);
    if (rc) return rc;
    // coherence sort of the first n_seg hyperbolic views in launch order (the expensive ones)
    const uint32_t n_seg = b->sort_buf ? std::min(b->n_hy, BATCH_SORT_VIEWS) : 0u;
    if (n_seg) HTC_CUDA(cudaMemsetAsync(batch_sort_at(b->sort_buf, b->sort_slots, (unsigned)b->num_sms).hist, 0,
                                        2 * sizeof(uint32_t) * (size_t)BATCH_SORT_VIEWS * SORT_BINS, st));
    HTC_CUDA(cudaMemsetAsync(b->d_wcnt, 0, 4 * sizeof(uint32_t) * batch_counters(b->n_views, b->hops_max), st));
    k_batch_stage<<<b->n_order, STAGE_THREADS, 0, st>>>(b->d_views, b->d_order, b->d_err);
    HTC_CUDA(cudaGetLastError());
    if (!b->n_hy || !b->n_eu) return batch_passes(b, q, blocks_hy, blocks_eu, smem, n_seg, stats, st, st);
    HTC_CUDA(cudaEventRecord(b->forked, st));
    HTC_CUDA(cudaStreamWaitEvent(b->side, b->forked, 0));
    rc = batch_passes(b, q, blocks_hy, blocks_eu, smem, n_seg, stats, st, b->side);
    HTC_CUDA(cudaEventRecord(b->joined, b->side));
    HTC_CUDA(cudaStreamWaitEvent(st, b->joined, 0));
    return rc;
}

extern "C" {

int htc_batch_create(uint32_t max_views, htc_batch **out) {
    if (!out) return fail(HTC_ERR_INVALID, "out is NULL");
    *out = nullptr;
    if (max_views == 0) return fail(HTC_ERR_INVALID, "max_views must be positive");
    int dev = 0;
    HTC_CUDA(cudaGetDevice(&dev));
    htc_batch *b = new htc_batch();
    b->max_views = max_views;
    cudaError_t e = cudaDeviceGetAttribute(&b->num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&b->max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess) e = cudaMalloc(&b->d_views, sizeof(BatchView) * max_views);
    if (e == cudaSuccess) e = cudaMalloc(&b->d_order, 2 * sizeof(uint32_t) * max_views);   // all, then by recipe
    if (e == cudaSuccess) e = cudaMalloc(&b->d_err, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaMemset(b->d_err, 0, sizeof(uint32_t));
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&b->side, cudaStreamNonBlocking);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->forked, cudaEventDisableTiming);
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->joined, cudaEventDisableTiming);
    for (int i = 0; i < 2 && e == cudaSuccess; ++i) {
        e = cudaHostAlloc(reinterpret_cast<void **>(&b->p_views[i]), sizeof(BatchView) * max_views, cudaHostAllocDefault);
        if (e == cudaSuccess) e = cudaHostAlloc(reinterpret_cast<void **>(&b->p_order[i]), 2 * sizeof(uint32_t) * max_views, cudaHostAllocDefault);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->staged[i], cudaEventDisableTiming);
    }
    if (e == cudaSuccess) {
        b->max_smem -= 1024;
        e = batch_wave_smem_attr<RECIPE_HY>(b->max_smem);
        if (e == cudaSuccess) e = batch_wave_smem_attr<RECIPE_EU>(b->max_smem);
    }
    if (e != cudaSuccess) {
        batch_free(b);
        return cuda_fail(e, "htc_batch_create");
    }
    *out = b;
    return HTC_OK;
}

void htc_batch_destroy(htc_batch *b) { batch_free(b); }

}  // extern "C"

// Grows the wavefront queues (slots per queue) and counters (words) when a view set needs
// more; launches already enqueued on `st` may still use the old ones, so they finish first.
static int batch_grow(htc_batch *b, uint64_t slots, size_t words, cudaStream_t st) {
    if (slots <= b->wave_slots && words <= b->wcnt_words && b->sort_slots >= b->wave_slots) return HTC_OK;
    HTC_CUDA(cudaStreamSynchronize(st));
    // a captured graph holds the old buffers' addresses: the next graph launch captures anew
    if (b->graph_exec) { cudaGraphExecDestroy(b->graph_exec); b->graph_exec = nullptr; }
    if (b->graph) { cudaGraphDestroy(b->graph); b->graph = nullptr; }
    if (slots > b->wave_slots) {
        if (b->wave_buf) HTC_CUDA(cudaFree(b->wave_buf));
        b->wave_buf = nullptr;
        b->wave_slots = 0;
        const uint64_t cap = (slots + slots / 4 + 63) & ~(uint64_t)63;
        HTC_CUDA(cudaMalloc(&b->wave_buf, 2 * WAVE_SLOT_BYTES * cap));
        b->wave_slots = cap;
    }
    if (words > b->wcnt_words) {
        if (b->d_wcnt) HTC_CUDA(cudaFree(b->d_wcnt));
        b->d_wcnt = nullptr;
        b->wcnt_words = 0;
        HTC_CUDA(cudaMalloc(&b->d_wcnt, sizeof(uint32_t) * words));
        b->wcnt_words = words;
    }
    if (b->sort_slots < b->wave_slots) {
        if (b->sort_buf) HTC_CUDA(cudaFree(b->sort_buf));
        b->sort_buf = nullptr;
        b->sort_slots = 0;
        HTC_CUDA(cudaMalloc(&b->sort_buf, batch_sort_bytes(b->wave_slots, (uint32_t)b->num_sms)));
        b->sort_slots = b->wave_slots;
    }
    return HTC_OK;
}
// Room for the views' scene images. Nothing waits: the view table of the launches enqueued so far
// points into the buffer that was, which is kept until the batch is destroyed (the new one is at least
// twice as large, so all of them together are less than it).
static int batch_grow_images(htc_batch *b, size_t words) {
    if (words <= b->image_words) return HTC_OK;
    words = std::max(words, 2 * b->image_words);
    float4 *images = nullptr;
    const RelaxedCapture relaxed;
    HTC_CUDA(cudaMalloc(&images, sizeof(float4) * words));
    if (b->images) b->old_images.push_back(b->images);
    b->images = images;
    b->image_words = words;
    return HTC_OK;
}

extern "C" {

int htc_batch_reserve(htc_batch *b, uint64_t pixels, uint32_t max_hops, void *stream) {
    if (!b) return fail(HTC_ERR_INVALID, "batch is NULL");
    if (max_hops == 0) return fail(HTC_ERR_INVALID, "max_hops must be positive");
    // images of the largest scenes for as many views as 64 MB hold (287; more by demand, batch_grow_images)
    const size_t largest = 1 + (size_t)b->max_smem / 16;
    int rc = batch_grow_images(b, std::min(b->max_views * largest, (size_t)(64u << 20) / sizeof(float4)));
    if (rc) return rc;
    // each view's region is rounded up to 64 slots
    return batch_grow(b, pixels + 64ull * b->max_views, 4 * batch_counters(b->max_views, max_hops),
                      reinterpret_cast<cudaStream_t>(stream));
}

int htc_batch_set_views(htc_batch *b, const htc_view *views, uint32_t n_views, uint32_t tile_pixels,
                        uint32_t blocks_per_sm, void *stream) {
    if (!b) return fail(HTC_ERR_INVALID, "batch is NULL");
    if (n_views > b->max_views) return fail(HTC_ERR_INVALID, "more views than the batch was created for");
    if (n_views && !views) return fail(HTC_ERR_INVALID, "views is NULL");
    if (tile_pixels == 0) return fail(HTC_ERR_INVALID, "tile_pixels must be positive");
    b->h_views.assign(n_views, BatchView());
    uint32_t smem_objects = 0;
    std::vector<std::pair<double, uint32_t>> order;
    for (uint32_t i = 0; i < n_views; ++i) {
        const htc_view &v = views[i];
        if (v.recipe != HTC_RECIPE_HY && v.recipe != HTC_RECIPE_EU) return fail(HTC_ERR_UNSUPPORTED, "unknown scene recipe in a view");
        if (v.light_hops == 0) return fail(HTC_ERR_INVALID, "light_hops must be positive");
        if (v.address_width != 32 && v.address_width != 64) return fail(HTC_ERR_INVALID, "address_width must be 32 or 64");
        if (v.flags & ~HTC_FLAG_JITTER_YX) return fail(HTC_ERR_INVALID, "unknown view flags");
        if (v.width == 0 || v.height == 0 || (uint64_t)v.width * v.height >= 0xFFFFFFFFull)
            return fail(HTC_ERR_INVALID, "view size must be positive and fit 32 bits");
        if (!v.scene || !v.canvas || !v.seeds) return fail(HTC_ERR_INVALID, "view buffers must be device pointers");
        if ((reinterpret_cast<uintptr_t>(v.scene) & 15u) || (reinterpret_cast<uintptr_t>(v.canvas) & 15u))
            return fail(HTC_ERR_INVALID, "scene and canvas must be 16-byte aligned");
        if (v.scene_size < (v.recipe == HTC_RECIPE_HY ? 128u : 80u)) return fail(HTC_ERR_SCENE, "view scene smaller than its header");
        BatchView &d = b->h_views[i];
        d.scene = reinterpret_cast<const uint8_t *>(v.scene);
        d.scene_size = v.scene_size;
        d.canvas = reinterpret_cast<float4 *>(v.canvas);
        d.seeds = v.seeds;
        d.width = v.width;
        d.height = v.height;
        d.recipe = v.recipe;
        d.hops = v.light_hops;
        d.flags = v.flags;
        d.address_width = v.address_width;
        d.passes = v.passes;
        d.max_objects = objects_capacity(v.recipe, v.scene_size);
        if (v.passes == 0) continue;
        if (d.max_objects > smem_objects) smem_objects = d.max_objects;
        // cost per pixel ~ passes x hops x objects: expensive views first (longest-first order
        // shortens the tail of the persistent launch)
        order.push_back({(double)v.passes * v.light_hops * (1.0 + d.max_objects), i});
    }
    if (smem_bytes(smem_objects) + sizeof(uint32_t) * ((size_t)n_views + 1) > (size_t)b->max_smem)
        return fail(HTC_ERR_UNSUPPORTED, "a view has more objects than shared memory can stage");
    std::stable_sort(order.begin(), order.end(), [](const std::pair<double, uint32_t> &a, const std::pair<double, uint32_t> &c) { return a.first > c.first; });
    // wavefront queues: one region of W*H slots (rounded to 64: 16-byte aligned arrays) per view
    uint64_t slots = 0;
    size_t images = 0;
    uint32_t hops_max = 0, passes_max = 0, hops_of[2] = {0, 0}, passes_of[2] = {0, 0};
    for (const auto &o : order) {
        BatchView &d = b->h_views[o.second];
        d.qoff = slots;
        slots += ((uint64_t)d.width * d.height + 63) & ~(uint64_t)63;
        images += image_words(d.max_objects);
        hops_max = std::max(hops_max, d.hops);
        passes_max = std::max(passes_max, d.passes);
        const int k = d.recipe == RECIPE_HY ? 0 : 1;
        hops_of[k] = std::max(hops_of[k], d.hops);
        passes_of[k] = std::max(passes_of[k], d.passes);
    }
    b->smem_objects = smem_objects;
    b->blocks_per_sm = blocks_per_sm;
    b->tile_pixels = tile_pixels;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    {
        int rc = batch_grow(b, slots, 4 * batch_counters(n_views, hops_max), st);
        if (!rc) rc = batch_grow_images(b, images);
        if (rc) return rc;
    }
    images = 0;
    for (const auto &o : order) {   // their places, now that the buffer is there
        b->h_views[o.second].image = b->images + images;
        images += image_words(b->h_views[o.second].max_objects);
    }
    b->n_views = n_views;
    b->n_order = (uint32_t)order.size();
    b->hops_max = hops_max;
    b->passes_max = passes_max;
    for (int k = 0; k < 2; ++k) {
        b->hops_of[k] = hops_of[k];
        b->passes_of[k] = passes_of[k];
    }
    // Asynchronous upload through the next pinned slot: wait only for that slot's previous
    // copy, then copy on `stream` (ordered after any launch still reading the device arrays).
    const int k = b->slot;
    b->slot ^= 1;
    HTC_CUDA(cudaEventSynchronize(b->staged[k]));
    if (n_views) std::memcpy(b->p_views[k], b->h_views.data(), sizeof(BatchView) * n_views);
    // the cost order of every view, then the same order split by recipe
    uint32_t *po = b->p_order[k];
    b->n_hy = b->n_eu = 0;
    for (uint32_t i = 0; i < b->n_order; ++i) po[i] = order[i].second;
    for (uint32_t i = 0; i < b->n_order; ++i)
        if (b->h_views[order[i].second].recipe == RECIPE_HY) po[b->n_order + b->n_hy++] = order[i].second;
    for (uint32_t i = 0; i < b->n_order; ++i)
        if (b->h_views[order[i].second].recipe != RECIPE_HY) po[b->n_order + b->n_hy + b->n_eu++] = order[i].second;
    if (b->n_order) HTC_CUDA(cudaMemcpyAsync(b->d_order, po, 2 * sizeof(uint32_t) * b->n_order, cudaMemcpyHostToDevice, st));
    if (n_views) HTC_CUDA(cudaMemcpyAsync(b->d_views, b->p_views[k], sizeof(BatchView) * n_views, cudaMemcpyHostToDevice, st));
    HTC_CUDA(cudaEventRecord(b->staged[k], st));
    if (b->graph_exec) { cudaGraphExecDestroy(b->graph_exec); b->graph_exec = nullptr; }
    if (b->graph) { cudaGraphDestroy(b->graph); b->graph = nullptr; }
    return HTC_OK;
}

int htc_batch_render(htc_batch *b, uint64_t *stats, void *stream) {
    if (!b) return fail(HTC_ERR_INVALID, "batch is NULL");
    return batch_launch_wave(b, stats, reinterpret_cast<cudaStream_t>(stream));
}

int htc_batch_graph_launch(htc_batch *b, uint64_t *stats, void *stream) {
    if (!b) return fail(HTC_ERR_INVALID, "batch is NULL");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (b->graph_exec && b->graph_stats != stats) {   // the graph's kernels hold the stats pointer
        cudaGraphExecDestroy(b->graph_exec);
        b->graph_exec = nullptr;
        cudaGraphDestroy(b->graph);
        b->graph = nullptr;
    }
    if (!b->graph_exec) {
        cudaStream_t cap;
        HTC_CUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
        cudaError_t e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
        int rc = HTC_OK;
        if (e == cudaSuccess) rc = batch_launch_wave(b, stats, cap);
        cudaGraph_t g = nullptr;
        cudaError_t e2 = cudaStreamEndCapture(cap, &g);
        cudaStreamDestroy(cap);
        if (e != cudaSuccess) return cuda_fail(e, "cudaStreamBeginCapture");
        if (rc) { if (g) cudaGraphDestroy(g); return rc; }
        if (e2 != cudaSuccess) return cuda_fail(e2, "cudaStreamEndCapture");
        e = cudaGraphInstantiate(&b->graph_exec, g, 0);
        if (e != cudaSuccess) { cudaGraphDestroy(g); return cuda_fail(e, "cudaGraphInstantiate"); }
        b->graph = g;
        b->graph_stats = stats;
    }
    HTC_CUDA(cudaGraphLaunch(b->graph_exec, st));
    return HTC_OK;
}

int htc_batch_check(htc_batch *b, void *stream) {
    if (!b) return fail(HTC_ERR_INVALID, "batch is NULL");
    uint32_t err = 0;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    HTC_CUDA(cudaMemcpyAsync(&err, b->d_err, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    HTC_CUDA(cudaStreamSynchronize(st));
    if (err) {
        HTC_CUDA(cudaMemsetAsync(b->d_err, 0, sizeof(uint32_t), st));
        HTC_CUDA(cudaStreamSynchronize(st));
        return fail(HTC_ERR_SCENE, "a view's scene bytes failed validation");
    }
    return HTC_OK;
}


// ---------------------------------------------------------------- allocation-free entry
// Scratch of htc_render_passes_noalloc: the persistent kernel's work-queue words
// ([0] next pixel, [1] finished blocks) and the error word the kernel writes when the caller
// passes no `status` ([2]; nothing reads it, so such a caller gets no error report, as the
// header says). A file-scope device array, so the entry point never allocates; it lives on
// every device that loads this library until the process exits. In host code
// `g_noalloc_scratch` is only a stand-in for the symbol: its device address comes from
// cudaGetSymbolAddress.
constexpr uint32_t NOALLOC_SCRATCH_WORDS = 64;   // 256 bytes
constexpr uint64_t NOALLOC_MAX_PIXELS = 1ull << 31;   // the queue word counts pixels
static __device__ __align__(256) uint32_t g_noalloc_scratch[NOALLOC_SCRATCH_WORDS];

namespace {
constexpr int NOALLOC_MAX_DEVICES = 64;
std::mutex g_noalloc_mutex;
uint32_t *g_noalloc_ptr[NOALLOC_MAX_DEVICES];
int g_noalloc_sms[NOALLOC_MAX_DEVICES];
int g_noalloc_smem[NOALLOC_MAX_DEVICES];

// Once per device, with that device current: resolve the scratch address and the launch
// limits. Allocates nothing. The cached address and kernel attributes outlive a device reset,
// which the header therefore excludes after the first call.
int noalloc_setup(int dev, uint32_t **scratch, int *num_sms, int *max_smem) {
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) return fail(HTC_ERR_UNSUPPORTED, "device index beyond the supported range");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (!g_noalloc_ptr[dev]) {
        uint32_t *ptr = nullptr;
        HTC_CUDA(cudaGetSymbolAddress(reinterpret_cast<void **>(&ptr), g_noalloc_scratch));
        int sms = 0, smem = 0;
        HTC_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        HTC_CUDA(cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
        smem -= 1024;
        int rc = set_smem_attr<RECIPE_HY>(smem);
        if (rc) return rc;
        rc = set_smem_attr<RECIPE_EU>(smem);
        if (rc) return rc;
        g_noalloc_sms[dev] = sms;
        g_noalloc_smem[dev] = smem;
        g_noalloc_ptr[dev] = ptr;
    }
    *scratch = g_noalloc_ptr[dev];
    *num_sms = g_noalloc_sms[dev];
    *max_smem = g_noalloc_smem[dev];
    return HTC_OK;
}
}  // namespace

int htc_render_passes_noalloc(int recipe, uint32_t light_hops, int address_width, uint32_t flags, uint32_t W,
                              uint32_t H, const void *scene, size_t scene_size, float *canvas, uint32_t *seeds,
                              uint32_t passes, uint64_t *stats, uint32_t *status, void *stream) {
    if (recipe != HTC_RECIPE_HY && recipe != HTC_RECIPE_EU) return fail(HTC_ERR_UNSUPPORTED, "unknown scene recipe");
    if (light_hops == 0) return fail(HTC_ERR_INVALID, "light_hops must be positive");
    if (address_width != 32 && address_width != 64) return fail(HTC_ERR_INVALID, "address_width must be 32 or 64");
    if (flags & ~HTC_FLAG_JITTER_YX) return fail(HTC_ERR_INVALID, "unknown program flags");
    if (W == 0 || H == 0) return fail(HTC_ERR_INVALID, "canvas width and height must be positive");
    if ((uint64_t)W * (uint64_t)H > NOALLOC_MAX_PIXELS)
        return fail(HTC_ERR_UNSUPPORTED, "htc_render_passes_noalloc serves at most 2^31 pixels per call (width*height)");
    if (!scene || !canvas || !seeds) return fail(HTC_ERR_INVALID, "scene, canvas and seeds must be device pointers");
    if ((reinterpret_cast<uintptr_t>(scene) & 15u) != 0 || (reinterpret_cast<uintptr_t>(canvas) & 15u) != 0)
        return fail(HTC_ERR_INVALID, "scene and canvas must be 16-byte aligned");
    if (scene_size < (recipe == HTC_RECIPE_HY ? 128u : 80u))
        return fail(HTC_ERR_SCENE, "scene buffer is smaller than the scene header");
    int dev = 0;
    HTC_CUDA(cudaGetDevice(&dev));
    uint32_t *scratch = nullptr;
    int num_sms = 0, max_smem = 0;
    int rc = noalloc_setup(dev, &scratch, &num_sms, &max_smem);
    if (rc) return rc;
    const uint32_t max_objects = objects_capacity(recipe, scene_size);
    const size_t smem = smem_bytes(max_objects);
    if (smem > (size_t)max_smem) return fail(HTC_ERR_UNSUPPORTED, "scene has more objects than shared memory can stage");
    if (passes == 0) return HTC_OK;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    // The queue words must start at zero; the array keeps whatever the last call left.
    HTC_CUDA(cudaMemsetAsync(scratch, 0, 3 * sizeof(uint32_t), st));
    int per_sm = 0;
    cudaError_t e = recipe == HTC_RECIPE_HY
        ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, render_persistent<RECIPE_HY>, 128, smem)
        : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, render_persistent<RECIPE_EU>, 128, smem);
    if (e != cudaSuccess) return cuda_fail(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor");
    if (per_sm < 1) per_sm = 1;
    uint64_t blocks = (uint64_t)per_sm * (uint64_t)num_sms;
    const uint64_t needed = ((uint64_t)W * H + 127) / 128;
    if (blocks > needed) blocks = needed;
    uint32_t *err = status ? status : scratch + 2;
    const uint8_t *sc = reinterpret_cast<const uint8_t *>(scene);
    float4 *cv = reinterpret_cast<float4 *>(canvas);
    if (recipe == HTC_RECIPE_HY)
        render_persistent<RECIPE_HY><<<(unsigned)blocks, 128, smem, st>>>(sc, scene_size, max_objects, address_width, W, H,
                                                                          light_hops, passes, flags, cv, seeds, stats, err,
                                                                          scratch);
    else
        render_persistent<RECIPE_EU><<<(unsigned)blocks, 128, smem, st>>>(sc, scene_size, max_objects, address_width, W, H,
                                                                          light_hops, passes, flags, cv, seeds, stats, err,
                                                                          scratch);
    HTC_CUDA(cudaGetLastError());
    return HTC_OK;
}

int htc_fp32_probe(float *scratch, uint32_t blocks, int iters, double *flops, void *stream) {
    if (!scratch || !flops || blocks == 0 || iters <= 0) return fail(HTC_ERR_INVALID, "bad probe arguments");
    k_fma_probe<<<blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(scratch, iters);
    HTC_CUDA(cudaGetLastError());
    *flops = 2.0 * 8.0 * 16.0 * (double)iters * 256.0 * (double)blocks;
    return HTC_OK;
}

}  // extern "C"
