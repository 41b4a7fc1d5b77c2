// Wavefront path tracer reproducing azimuth's estimator (TraceRay,
// src/azimuth_main.cpp:966-1133) on the GPU.
//
// A camera sample in azimuth is a recursive tree: every non-emitting hit adds
// its direct light and ambient term and recurses into a diffuse scatter ray,
// a mirror ray and the dielectric refraction and reflection rays.  Here every
// tree node is one queue entry carrying the product of the weights above it
// ("throughput"); levels are processed breadth-first over a wave of samples:
//
//   camera  -> queue[1]                    (GetSampleCoord + GetRayForPixel)
//   per level L = 1 .. MaxRecursionDepth+1:
//     extend  queue[L]  -> hits            (RayEntityIntersection)
//     shade   hits      -> queue[L+1], shadow queue, per-sample sums
//     shadow  shadow queue -> per-sample sums (the visibility tests of CalculateLighting)
//   splat   per-sample sums -> film        (ComputeSampleWeight, box or Gaussian)
//
// The counter RNG is keyed by the tree node, so the order in which the GPU
// visits nodes does not change any random number: the result equals azimuth's
// own tree up to float summation order.  Child nodes whose weight is exactly
// zero (e.g. the scatter ray of a pure mirror) are not traced; azimuth traces
// them and multiplies their radiance by zero.
#include <cub/cub.cuh>

#include <algorithm>
#include <cfloat>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "az_internal.h"
#include "az_phase.cuh"
#include "az_pool.h"
#include "az_render.h"
#include "az_shade.cuh"
#include "az_wave.cuh"

namespace az {
namespace {

using namespace azd;

// GetSampleCoord + GetRayForPixel (src/azimuth_main.cpp:1135-1178) of camera
// sample s into wave slot i.
__device__ __forceinline__ void camera_node(const CameraParams &cam, const WaveQueues &Q, uint64_t s, uint64_t seed,
                                            uint32_t i) {
    uint32_t row, col, sx, sy;
    sample_of(cam, s, row, col, sx, sy);
    NodeRng rng;
    rng.init(seed, (row << 16) | col, (sy << 16) | sx, 0u, 0u);
    float cx = (float)col + (0.5f * cam.inv_sqrt + (float)sx * cam.inv_sqrt);
    float cy = (float)row + (0.5f * cam.inv_sqrt + (float)sy * cam.inv_sqrt);
    // the lens pair is drawn y first: GCC evaluates the two Random01()
    // arguments of Vec2(...) right to left in the oracle build
    float ly = rng.next() - 0.5f;
    float lx = rng.next() - 0.5f;
    lx *= cam.aperture;
    ly *= cam.aperture;
    f3 offx = cam.axx * lx, offy = cam.axy * ly;
    f3 dir = normalize(cam.base + cx * cam.stepx - cy * cam.stepy - offx - offy);
    f3 o = cam.pos + offx + offy;
    float time = rng.next();
    Q.o[1][i] = make_float4(o.x, o.y, o.z, time);
    Q.d[1][i] = make_float4(dir.x, dir.y, dir.z, __uint_as_float(cam.scene << PF_SCENE_SHIFT));
    Q.tp[1][i] = make_float4(1.0f, 1.0f, 1.0f, __uint_as_float(i));
    Q.digits[1][i] = 0u;
    Q.accum[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

__global__ void k_camera(CameraParams cam, WaveQueues Q, uint64_t wave_start, uint32_t n) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t seed = cam.seed;
    if (Q.wave) {
        wave_start = Q.wave[0];
        n = (uint32_t)Q.wave[1];
        seed = Q.wave[2];
        if (i == 0) Q.counts[1] = n;   // the level-1 queue is the wave itself
    }
    if (i >= n) return;
    camera_node(cam, Q, wave_start + i, seed, i);
}

// Camera samples of a tile wave: each block takes the next tile of the wave's
// work queue (`next`, zeroed before the launch) until the queue is empty.
__global__ void k_camera_tiles(const Tile *tiles, uint32_t ntiles, uint32_t *next, WaveQueues Q, uint2 *slot_map) {
    __shared__ uint32_t taken;
    for (;;) {
        if (threadIdx.x == 0) taken = atomicAdd(next, 1u);
        __syncthreads();
        const uint32_t t = taken;
        __syncthreads();   // every thread has read `taken` before it is overwritten
        if (t >= ntiles) return;
        const Tile T = tiles[t];
        const CameraParams &cam = Q.job_cams[T.job];
        for (uint32_t k = threadIdx.x; k < T.count; k += blockDim.x) {
            camera_node(cam, Q, (uint64_t)T.first + k, cam.seed, T.slot + k);
            slot_map[T.slot + k] = make_uint2(T.job, T.first + k);
        }
    }
}

// Sort keys that group a level's queue by where its rays start: a 15-bit
// Morton code of the origin's cell in a 32^3 grid over the scene bounds, for
// extension rays the top 13 bits of it and the direction octant.  Entries past
// the queue's size get the largest key, so after a stable sort the first
// `size` indices are the queue's own.
__global__ void k_order_keys(DevScene S, WaveQueues Q, uint32_t level, int shadow, uint32_t cap, uint32_t *keys,
                             uint32_t *vals) {
    const uint32_t n = shadow ? min(Q.counts[AZ_COUNT_SHADOW + level], Q.cap_s) : min(Q.counts[level], Q.cap_q);
    const int buf = level & 1;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += gridDim.x * blockDim.x) {
        uint32_t key = 0xFFFFu;
        if (i < n) {
            const float4 o = shadow ? Q.so[i] : Q.o[buf][i];
            uint32_t c[3];
            const float p[3] = {o.x, o.y, o.z};
            for (int a = 0; a < 3; a++) {
                const float u = (p[a] - S.box_lo[a]) * S.box_scale[a] * 32.0f;
                c[a] = u > 0.0f ? min((uint32_t)u, 31u) : 0u;   // NaN and below the box: cell 0
            }
            uint32_t m = 0;
            for (int b = 4; b >= 0; b--)
                m = (m << 3) | (((c[0] >> b) & 1u) << 2) | (((c[1] >> b) & 1u) << 1) | ((c[2] >> b) & 1u);
            if (shadow) {
                key = m;
            } else {
                const float4 d = Q.d[buf][i];
                const uint32_t oct = (d.x < 0.0f ? 4u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 1u : 0u);
                key = ((m >> 2) << 3) | oct;
            }
        }
        keys[i] = key;
        vals[i] = i;
    }
}

// When a warp of the traversal kernels does what (az_phase.cuh): finished lanes
// wait until `refill` of them can write their results and take new queries
// together (LaunchParams); primitives are tested once kPrimLanes lanes hold
// some, or at least as many as could visit a node, and for as long as
// kPrimStay do.  Measured on full frames of the dense mesh, the interior and the
// moving spheres (one B200): kPrimLanes 10: 211 / 296 / 169 ms, 12: 210 / 292 /
// 170, 16: 208 / 287 / 172.
constexpr uint32_t kPrimLanes = 16, kPrimStay = 8;
constexpr uint32_t kFetchBatch = 64;   // queries a warp takes from the queue at once
constexpr uint32_t kNoQuery = 0xFFFFFFFFu;
constexpr int kTraceBlock = 128;       // threads a block of the traversal kernels

// The loop of a phase-scheduled kernel: called by all 32 lanes of a warp.
//   load(q)          the world ray of queue entry q
//   begin(q)         starts its query; false when this kernel leaves it out
//   end(q)           writes the result of a finished query; false: it goes on
//   size             the queue's length (in device memory), at most cap
//   order            the queue's visiting order or null
template <bool COUNT, typename TRACER, typename LOAD, typename BEGIN, typename END, typename SCENE>
__device__ __forceinline__ void phase_run(TRACER &T, const uint32_t *size, uint32_t cap, const uint32_t *order,
                                          uint32_t *fetch, uint32_t refill, bool cull, float eps, LOAD load,
                                          BEGIN begin, END end, SCENE scene, uint32_t *err,
                                          uint32_t *counts) {
    constexpr uint32_t kAll = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t qi = kNoQuery;            // this lane's queue entry
    bool done = false;                 // its query has finished
    uint32_t next = 0, last = 0;       // the warp's batch of work items; kNoQuery: the queue is exhausted
    uint32_t nodes_seen = 0, prims_seen = 0;
    auto ray = [&]() { return load(qi); };
    for (;;) {
        if (done) {
            done = false;
            if (end(qi)) qi = kNoQuery;
        }
        uint32_t idle = __ballot_sync(kAll, qi == kNoQuery);
        while (idle && last != kNoQuery) {
            if (next == last) {
                // batches small enough that the launch's warps share a short queue evenly
                const uint32_t n = min(*size, cap);
                const uint32_t batch = min(kFetchBatch, max(32u, n / (gridDim.x * (blockDim.x >> 5) * 2u)));
                if (lane == 0) next = atomicAdd(fetch, batch);
                next = __shfl_sync(kAll, next, 0);
                last = min(next + batch, n);
                if (next >= n) {
                    next = last = kNoQuery;
                    break;
                }
            }
            const uint32_t k = next + __popc(idle & ((1u << lane) - 1u));
            if ((idle >> lane) & 1u && k < last) {
                const uint32_t q = order ? order[k] : k;
                if (begin(q)) qi = q;
            }
            next = min(last, next + (uint32_t)__popc(idle));
            idle = __ballot_sync(kAll, qi == kNoQuery);
        }
        // rounds until enough lanes wait (all of the idle ones are idle for good)
        const uint32_t spare = __popc(idle);
        if (spare == 32u) break;
        for (uint32_t rounds = 0;; rounds++) {
            if (rounds > AZD_MAX_STEPS) {
                // far more than a valid hierarchy needs: give up on these queries and on the rest
                if (qi != kNoQuery && !done) {
                    atomicOr(err, 1u);
                    T.abandon();
                }
                next = last = kNoQuery;
            }
            bool live = qi != kNoQuery && !done;
            if (live && T.refill(scene(), ray, eps)) {
                done = true;
                live = false;
            }
            const uint32_t nodes = __ballot_sync(kAll, live && T.wants_node());
            uint32_t prims = __ballot_sync(kAll, live && T.has_prims());
            const uint32_t busy = __popc(nodes | prims);
            if (!busy || 32u - busy - spare >= refill) break;
            const uint32_t np = __popc(prims);
            if (np >= kPrimLanes || (np && np >= __popc(nodes))) {
                do {
                    if (COUNT) prims_seen += __popc(prims);
                    if (live && T.has_prims() && T.prim(scene(), ray, cull, eps, err)) {
                        done = true;
                        live = false;
                    }
                    prims = __ballot_sync(kAll, live && T.has_prims());
                } while (__popc(prims) >= kPrimStay);
            } else {
                if (COUNT) nodes_seen += __popc(nodes);
                if (live && T.wants_node()) T.node(scene(), err);
            }
        }
    }
    if (COUNT && lane == 0) {
        atomicAdd(counts + 0, nodes_seen);
        atomicAdd(counts + 1, prims_seen);
    }
}

// Closest hits of the level's queue.
// WT: triangles by the watertight test (AZ_FLAG_WATERTIGHT) instead of azimuth's.
// MULTI: a tile wave of several scenes: each query is traced in the scene its
// entry names (WaveQueues.scenes).
// SPH: the scene has spheres at the top level (DevScene.top_spheres).
// COUNT: visit counters (AZ_FLAG_COUNT_TRAVERSAL).
// Bound by the issue of divergent instructions (profiles/): 128 threads of at
// most 64 registers, 32 warps a multiprocessor, no spills.
//
// MINB == 0: one query per thread in a grid-stride loop, for scenes whose whole
// hierarchy is a few nodes: all lanes then take nearly the same steps, and the
// votes and the shared stack cost more than they give (Cornell box, 1 M samples:
// closest hits 0.48 ms a frame against 0.65).
template <int MINB, bool WT, bool MULTI, bool SPH, bool COUNT>
__global__ void __launch_bounds__(kTraceBlock, MINB ? MINB : 8)
    k_extend(DevScene S, CameraParams cam, WaveQueues Q, uint32_t level) {
    if constexpr (MINB == 0) {
        const uint32_t n = min(Q.counts[level], Q.cap_q);
        for (uint32_t k = blockIdx.x * kTraceBlock + threadIdx.x; k < n; k += gridDim.x * kTraceBlock) {
            const uint32_t i = Q.eorder ? Q.eorder[k] : k;
            const float4 o = Q.o[level & 1][i], d = Q.d[level & 1][i];
            Ray r;
            r.o = mk(o.x, o.y, o.z);
            r.d = mk(d.x, d.y, d.z);
            r.time = o.w;
            Hit h;
            trace<Q_CLOSEST, WT>(S, r, cam.cull != 0, cam.eps_isect, FLT_MAX, h,
                                 COUNT ? Q.counts + AZ_COUNT_NODES : nullptr, Q.counts + AZ_COUNT_ERROR);
            Q.hit[i] = make_uint4(__float_as_uint(h.t), __float_as_uint(h.tl), h.prim, h.ent);
        }
        return;
    }
    __shared__ PhaseShared<kTraceBlock> shared;
    uint2 deep[AZD_WSTACK - kSharedStack];
    PhaseTracer<Q_CLOSEST, WT, SPH, kTraceBlock, MULTI> T(shared, deep);
    const int buf = level & 1;
    uint32_t si = 0;   // MULTI: the entry's scene
    auto load = [&](uint32_t q) {
        const float4 o = Q.o[buf][q], d = Q.d[buf][q];
        Ray r;
        r.o = mk(o.x, o.y, o.z);
        r.d = mk(d.x, d.y, d.z);
        r.time = o.w;
        if (MULTI) si = (__float_as_uint(d.w) & PF_SCENE) >> PF_SCENE_SHIFT;
        return r;
    };
    auto scene = [&]() -> const DevScene & { return MULTI ? Q.scenes[si] : S; };
    auto begin = [&](uint32_t q) {
        const Ray r = load(q);
        T.init(scene(), r, FLT_MAX, 0xFFFFFFFFu);
        return true;
    };
    auto end = [&](uint32_t q) {
        if (T.in_blas) T.take_group_hit(scene(), load(q), cam.eps_isect);
        Q.hit[q] = T.hit();
        return true;
    };
    phase_run<COUNT>(T, Q.counts + level, Q.cap_q, Q.eorder, Q.counts + AZ_COUNT_FETCH + level, cam.refill,
                     cam.cull != 0, cam.eps_isect, load, begin, end, scene, Q.counts + AZ_COUNT_ERROR,
                     Q.counts + AZ_COUNT_NODES);
}

// Entity lights: a light sample is occluded unless the nearest hit is the
// light's entity, so the light's own nearest hit is found first and the
// visibility query looks for anything else before it.  This kernel replaces the
// limit of the level's SHADOW_ENTITY queries by that distance (FLT_MAX: the ray
// misses the light).  Inside k_shadow the light's test ran with the few lanes
// that took a new query at a time and its call spilled the traversal's
// registers: C1's visibility queries take 66 ms a frame after this pass (of
// 2-3 ms, bound by the 36 bytes it reads per query) against 80 ms.
template <bool MULTI>
__global__ void __launch_bounds__(256) k_light_limits(DevScene S0, WaveQueues Q, uint32_t level) {
    const uint32_t n = min(Q.counts[AZ_COUNT_SHADOW + level], Q.cap_s);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t meta = Q.smeta[i];
        if (shadow_kind(meta) != SHADOW_ENTITY) continue;
        const DevScene &S = MULTI ? Q.scenes[shadow_scene(meta)] : S0;
        const float4 o = Q.so[i], d = Q.sd[i];
        Ray r;
        r.o = mk(o.x, o.y, o.z);
        r.d = mk(d.x, d.y, d.z);
        r.time = o.w;
        float t = FLT_MAX;
        light_entity_hit(S.ents, S.light_tris, S.lights[shadow_light(meta)], r, t);
        Q.sd[i].w = t;
    }
}

// Visibility of the SHADOW_ENTITY_FULL queries of the shadow queue (entity
// lights too large for the two-phase test): one full nearest-hit query each,
// visible when the nearest hit is the light's entity (src/azimuth_main.cpp:694-712).
// Launched only for scenes that have such a light.
template <bool WT, bool MULTI = false>
__global__ void __launch_bounds__(128) k_shadow_full(DevScene S0, CameraParams cam, WaveQueues Q, uint32_t level) {
    const uint32_t n = min(Q.counts[AZ_COUNT_SHADOW + level], Q.cap_s);
    uint32_t *cnt = cam.count_traversal ? Q.counts + AZ_COUNT_SNODES : nullptr;
    uint32_t *err = Q.counts + AZ_COUNT_ERROR;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t meta = Q.smeta[i];
        if (shadow_kind(meta) != SHADOW_ENTITY_FULL) continue;
        const DevScene &S = MULTI ? Q.scenes[shadow_scene(meta)] : S0;
        const float4 o = Q.so[i], d = Q.sd[i], c = Q.sc[i];
        const DevLight &L = S.lights[shadow_light(meta)];
        Ray r;
        r.o = mk(o.x, o.y, o.z);
        r.d = mk(d.x, d.y, d.z);
        r.time = o.w;
        Hit h;
        const bool any = trace<Q_CLOSEST, WT>(S, r, false, 0.0f, FLT_MAX, h, cnt, err);
        if (!any || S.ents[h.ent].uid == L.uid) add_accum(Q.accum, __float_as_uint(c.w), mk(c.x, c.y, c.z));
    }
}

// Visibility of the queued light samples; unoccluded ones are added to their
// sample.  Template arguments as k_extend.
template <int MINB, bool WT, bool MULTI, bool SPH, bool COUNT>
__global__ void __launch_bounds__(kTraceBlock, MINB ? MINB : 8)
    k_shadow(DevScene S, CameraParams cam, WaveQueues Q, uint32_t level) {
    if constexpr (MINB == 0) {
        const uint32_t n = min(Q.counts[AZ_COUNT_SHADOW + level], Q.cap_s);
        for (uint32_t k = blockIdx.x * kTraceBlock + threadIdx.x; k < n; k += gridDim.x * kTraceBlock) {
            const uint32_t i = Q.sorder ? Q.sorder[k] : k;
            const float4 o = Q.so[i], d = Q.sd[i], c = Q.sc[i];
            const uint32_t meta = Q.smeta[i];
            const uint32_t kind = shadow_kind(meta);
            if (kind == SHADOW_ENTITY_FULL) continue;   // k_shadow_full
            Ray r;
            r.o = mk(o.x, o.y, o.z);
            r.d = mk(d.x, d.y, d.z);
            r.time = o.w;
            Hit h;
            if (!trace<Q_ANY, WT>(S, r, false, 0.0f, kind == SHADOW_ANY ? FLT_MAX : d.w, h,
                                  COUNT ? Q.counts + AZ_COUNT_SNODES : nullptr, Q.counts + AZ_COUNT_ERROR,
                                  kind == SHADOW_ENTITY ? S.lights[shadow_light(meta)].ent_index : 0xFFFFFFFFu))
                add_accum(Q.accum, __float_as_uint(c.w), mk(c.x, c.y, c.z));
        }
        return;
    }
    __shared__ PhaseShared<kTraceBlock> shared;
    uint2 deep[AZD_WSTACK - kSharedStack];
    PhaseTracer<Q_ANY, WT, SPH, kTraceBlock, MULTI> T(shared, deep);
    uint32_t si = 0;   // MULTI: the entry's scene
    auto load = [&](uint32_t q) {
        const float4 o = Q.so[q], d = Q.sd[q];
        Ray r;
        r.o = mk(o.x, o.y, o.z);
        r.d = mk(d.x, d.y, d.z);
        r.time = o.w;
        return r;
    };
    auto scene = [&]() -> const DevScene & { return MULTI ? Q.scenes[si] : S; };
    auto begin = [&](uint32_t q) {
        const uint32_t meta = Q.smeta[q];
        const uint32_t kind = shadow_kind(meta);
        if (MULTI) si = shadow_scene(meta);
        if (kind == SHADOW_ENTITY_FULL) return false;   // k_shadow_full
        const Ray r = load(q);
        T.init(scene(), r, kind == SHADOW_ANY ? FLT_MAX : Q.sd[q].w,   // an entity light's: k_light_limits
               kind == SHADOW_ENTITY ? scene().lights[shadow_light(meta)].ent_index : 0xFFFFFFFFu);
        return true;
    };
    auto end = [&](uint32_t q) {
        if (!T.confirm(scene(), load(q), 0.0f)) return false;
        if (!T.occluded) {
            const float4 c = Q.sc[q];
            add_accum(Q.accum, __float_as_uint(c.w), mk(c.x, c.y, c.z));
        }
        return true;
    };
    phase_run<COUNT>(T, Q.counts + AZ_COUNT_SHADOW + level, Q.cap_s, Q.sorder,
                     Q.counts + AZ_COUNT_FETCH + AZ_MAX_LEVELS + level, cam.shadow_refill, false, 0.0f, load, begin, end,
                     scene, Q.counts + AZ_COUNT_ERROR, Q.counts + AZ_COUNT_SNODES);
}

// ComputeSampleWeight (src/azimuth_main.cpp:1209-1254) for every sample of the wave.
// ComputeSampleWeight (src/azimuth_main.cpp:1209-1254): sample s's sum `a`
// into the film, box or Gaussian footprint.
__device__ __forceinline__ void splat_sample(const CameraParams &cam, az_pixel *film, uint64_t s, float4 a) {
    uint32_t row, col, sx, sy;
    sample_of(cam, s, row, col, sx, sy);
    float4 *f = reinterpret_cast<float4 *>(film);
    if (cam.filter == AZ_Filter_Box) {
        atomicAdd(&f[(size_t)row * cam.width + col], make_float4(a.x, a.y, a.z, 1.0f));
        return;
    }
    float cx = (float)col + (0.5f * cam.inv_sqrt + (float)sx * cam.inv_sqrt);
    float cy = (float)row + (0.5f * cam.inv_sqrt + (float)sy * cam.inv_sqrt);
    int32_t w1 = (int32_t)cam.width - 1, h1 = (int32_t)cam.height - 1;
    int32_t x0 = max((int32_t)col - cam.gk, 0), x1 = min((int32_t)col + cam.gk, w1);
    int32_t y0 = max((int32_t)row - cam.gk, 0), y1 = min((int32_t)row + cam.gk, h1);
    for (int32_t gy = y0; gy <= y1; gy++)
        for (int32_t gx = x0; gx <= x1; gx++) {
            float dx = cx - ((float)gx + 0.5f), dy = cy - ((float)gy + 0.5f);
            float d2 = dx * dx + dy * dy;
            float g = cam.g_norm * expf(cam.g_neg * d2);
            atomicAdd(&f[(size_t)gy * cam.width + gx], make_float4(a.x * g, a.y * g, a.z * g, g));
        }
}

__global__ void k_splat(CameraParams cam, WaveQueues Q, uint64_t wave_start, uint32_t n, az_pixel *film) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (Q.wave) {
        wave_start = Q.wave[0];
        n = (uint32_t)Q.wave[1];
    }
    if (i >= n) return;
    if (Q.counts[AZ_COUNT_OVERFLOW]) return;   // the wave is re-run
    if (cam.sample_out) {
        cam.sample_out[wave_start + i] = Q.accum[i];
        return;
    }
    splat_sample(cam, film, wave_start + i, Q.accum[i]);
}

// The samples of a tile wave, each into its own job's film.
__global__ void k_splat_tiles(WaveQueues Q, uint32_t n, az_pixel *const *films) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (Q.counts[AZ_COUNT_OVERFLOW]) return;   // the wave is re-run
    const uint2 js = Q.slot_map[i];
    splat_sample(Q.job_cams[js.x], films[js.x], js.y, Q.accum[i]);
}

// Launch configurations of the two traversal kernels, chosen per scene by
// az_gpu_autotune: resident blocks per multiprocessor (which caps registers:
// 7 blocks of 128 threads 72, 8 blocks 64) and the lanes that wait for each
// other before a warp writes results and takes new queries (32: a warp's
// queries begin and end together); or one query per thread (0 blocks).
struct Variant {
    int minb;
    uint32_t refill;
};
constexpr Variant kVariants[] = {{8, 4},  {8, 6},  {8, 10}, {8, 12}, {8, 14}, {8, 16}, {8, 20},
                                 {8, 8},  {8, 24}, {8, 32}, {0, 32}, {7, 4},  {7, 6},  {7, 8},
                                 {7, 10}, {7, 12}, {7, 14}, {7, 16}, {7, 24}, {7, 32}};
constexpr uint32_t kVariantCount = sizeof(kVariants) / sizeof(kVariants[0]);
static_assert(kVariantCount == AZ_LAUNCH_VARIANTS, "variant table and header disagree");

template <int MINB, bool WT, bool MULTI, bool SPH, bool COUNT>
void LaunchTraversal(bool shadow, int sms, const DevScene &S, const CameraParams &cam, const WaveQueues &Q,
                     uint32_t L, cudaStream_t st) {
    const int grid = sms * (2048 / kTraceBlock);
    if (shadow) k_shadow<MINB, WT, MULTI, SPH, COUNT><<<grid, kTraceBlock, 0, st>>>(S, cam, Q, L);
    else k_extend<MINB, WT, MULTI, SPH, COUNT><<<grid, kTraceBlock, 0, st>>>(S, cam, Q, L);
}

template <int MINB, bool WT, bool MULTI>
void LaunchTraversal(bool shadow, int sms, const DevScene &S, const CameraParams &cam, const WaveQueues &Q,
                     uint32_t L, cudaStream_t st) {
    if (S.top_spheres) {
        if (cam.count_traversal) LaunchTraversal<MINB, WT, MULTI, true, true>(shadow, sms, S, cam, Q, L, st);
        else LaunchTraversal<MINB, WT, MULTI, true, false>(shadow, sms, S, cam, Q, L, st);
    } else {
        if (cam.count_traversal) LaunchTraversal<MINB, WT, MULTI, false, true>(shadow, sms, S, cam, Q, L, st);
        else LaunchTraversal<MINB, WT, MULTI, false, false>(shadow, sms, S, cam, Q, L, st);
    }
}

// The closest-hit stage of level L, or its visibility stage, in launch
// configuration v (its blocks per multiprocessor; the lanes are in `cam`).
void LaunchTraversalVariant(uint32_t v, bool shadow, int sms, const DevScene &S, const CameraParams &cam,
                            const WaveQueues &Q, uint32_t L, cudaStream_t st) {
    const int grid = sms * 16;
    const bool loop = kVariants[v].minb == 0 && !Q.scenes && !cam.watertight;
    if (shadow && S.entity_lights) {
        if (Q.scenes) k_light_limits<true><<<sms * 8, 256, 0, st>>>(S, Q, L);
        else k_light_limits<false><<<sms * 8, 256, 0, st>>>(S, Q, L);
    }
    if (shadow && S.full_light_queries) {
        if (Q.scenes && cam.watertight) k_shadow_full<true, true><<<grid, 128, 0, st>>>(S, cam, Q, L);
        else if (Q.scenes) k_shadow_full<false, true><<<grid, 128, 0, st>>>(S, cam, Q, L);
        else if (cam.watertight) k_shadow_full<true><<<grid, 128, 0, st>>>(S, cam, Q, L);
        else k_shadow_full<false><<<grid, 128, 0, st>>>(S, cam, Q, L);
    }
    // A tile wave of several scenes and the watertight test have one block count:
    // their lanes keep more state (24 jobs of three scenes: 28.1 ms with 7 blocks,
    // 29.2 with 8, whose kernels spill)
    if (Q.scenes && cam.watertight) LaunchTraversal<7, true, true>(shadow, sms, S, cam, Q, L, st);
    else if (Q.scenes) LaunchTraversal<7, false, true>(shadow, sms, S, cam, Q, L, st);
    else if (cam.watertight) LaunchTraversal<7, true, false>(shadow, sms, S, cam, Q, L, st);
    else if (loop) LaunchTraversal<0, false, false>(shadow, sms, S, cam, Q, L, st);
    else if (kVariants[v].minb == 7) LaunchTraversal<7, false, false>(shadow, sms, S, cam, Q, L, st);
    else LaunchTraversal<8, false, false>(shadow, sms, S, cam, Q, L, st);
}

}  // namespace

// Camera basis and pixel steps of ProduceImageInLinearSpace
// (src/azimuth_main.cpp:1265-1347), evaluated on the host in float.
int SetupCamera(const az_camera *c, az_scissor sc, int32_t filter, uint32_t cull, const az_epsilon_values *eps,
                uint64_t seed, CameraParams &cam) {
    using azd::f3;
    auto v = [](const az_vec3 &a) { return azd::mk(a.x, a.y, a.z); };
    if (c->Resolution.x == 0 || c->Resolution.y == 0 || c->Resolution.x > 65535 || c->Resolution.y > 65535)
        return SetError(AZ_ERR_INVALID_ARGUMENT, "camera resolution must be 1..65535 per axis");
    f3 gaze = v(c->Gaze);
    if (c->GazeIsPoint) gaze = v(c->Gaze) - v(c->Position);
    f3 gn = azd::normalize(gaze);
    f3 az = -gn, ax, ay;
    if (c->IsLeftHanded) {
        ax = azd::normalize(azd::cross(azd::normalize(v(c->Up)), gn));
        ay = azd::cross(ax, az);
    } else {
        ax = azd::normalize(azd::cross(gn, azd::normalize(v(c->Up))));
        ay = azd::cross(az, ax);
    }
    float fdn = 1.0f;
    if (c->FocusDistance != 0.0f) fdn = c->FocusDistance / c->NearDistance;
    memset(&cam, 0, sizeof(cam));
    cam.width = c->Resolution.x;
    cam.height = c->Resolution.y;
    az_vec4 np = c->NearPlane;   // r, l, b, t
    if (c->Type == AZ_Camera_Simple) {
        float hh = c->NearDistance * tanf((c->FovY / 2.0f / 180.0f) * (float)3.14159265359);
        float ar = (float)cam.width / (float)cam.height;
        float wh = ar * hh;
        np.w = +hh;
        np.z = -hh;
        np.x = +wh;
        np.y = -wh;
    }
    float psx = (np.x - np.y) / (float)cam.width, psy = (np.w - np.z) / (float)cam.height;
    cam.stepx = ax * psx * fdn;
    cam.stepy = ay * psy * fdn;
    f3 tl = v(c->Position) + c->NearDistance * gn + np.y * ax + np.w * ay;
    cam.base = (tl - v(c->Position)) * fdn;
    cam.pos = v(c->Position);
    cam.axx = ax;
    cam.axy = ay;
    cam.aperture = c->ApertureSize;
    cam.sqrt_spp = (uint32_t)sqrtf((float)c->SampleCount);
    cam.inv_sqrt = 1.0f / cam.sqrt_spp;
    float gr = 1.5f, sigma = gr / 3.0f, two = 2.0f * (sigma * sigma);
    cam.g_neg = -1.0f / two;
    cam.g_norm = 1.0f / (two * (float)3.14159265359);
    cam.gk = (int32_t)ceilf(gr - 0.5f);
    uint32_t r1 = std::min(sc.Max.y, cam.height), c1 = std::min(sc.Max.x, cam.width);
    cam.r0 = sc.Min.y;
    cam.c0 = sc.Min.x;
    cam.hsc = r1 > cam.r0 ? r1 - cam.r0 : 0;
    cam.wsc = c1 > cam.c0 ? c1 - cam.c0 : 0;
    cam.npix = (uint64_t)cam.hsc * cam.wsc;
    cam.by_npix.set((uint32_t)cam.npix);   // at most 65535^2
    cam.by_wsc.set(cam.wsc);
    cam.by_sqrt.set(cam.sqrt_spp);
    if (filter != AZ_Filter_Box && filter != AZ_Filter_Gaussian) return SetError(AZ_ERR_INVALID_ARGUMENT, "unknown filter");
    cam.filter = filter;
    cam.seed = seed;
    cam.eps_isect = eps ? eps->Intersection : 0.0f;
    cam.eps_shadow = eps ? eps->ShadowRay : 0.000275f;
    cam.cull = cull;
    return AZ_OK;
}

WaveBuffers::~WaveBuffers() {
    DropGraph();
    // every render waits for its waves, so nothing uses the buffers any more
    for (void *p : ptrs) PoolFree(p, nullptr);
    PoolFree(guide_lobes, nullptr);
    PoolFree(guide_rec, nullptr);
    for (void *p : {(void *)okey[0], (void *)okey[1], (void *)oval, (void *)oidx_e, (void *)oidx_s, otemp})
        PoolFree(p, nullptr);
    if (side) ReleaseSide(SideStream{side, ev_fork, ev_join});
}

int WaveBuffers::EnsureSide() {
    if (side) return AZ_OK;
    SideStream s;
    const cudaError_t e = AcquireSide(&s);
    if (e != cudaSuccess) return CudaError(e, "creating the wave's side stream");
    side = s.stream;
    ev_fork = s.fork;
    ev_join = s.join;
    return AZ_OK;
}

int WaveBuffers::EnsureOrder(uint32_t cap, cudaStream_t st) {
    if (cap <= ocap && otemp) return AZ_OK;
    DropGraph();   // it refers to the buffers replaced below
    for (uint32_t **p : {&okey[0], &okey[1], &oval, &oidx_e, &oidx_s}) {
        PoolFree(*p, st);
        *p = nullptr;
    }
    PoolFree(otemp, st);
    otemp = nullptr;
    ocap = 0;
    for (uint32_t **p : {&okey[0], &okey[1], &oval, &oidx_e, &oidx_s})
        if (PoolAlloc((void **)p, (size_t)cap * sizeof(uint32_t), st) != cudaSuccess)
            return SetError(AZ_ERR_OUT_OF_MEMORY, "queue ordering buffers");
    size_t bytes = 0;
    AZ_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, bytes, okey[0], okey[1], oval, oidx_e, (int)cap, 0, 16));
    if (PoolAlloc(&otemp, bytes, st) != cudaSuccess) return SetError(AZ_ERR_OUT_OF_MEMORY, "queue ordering scratch");
    otemp_bytes = bytes;
    ocap = cap;
    return AZ_OK;
}

void WaveBuffers::DropGraph() {
    if (graph) cudaGraphExecDestroy(graph);
    graph = nullptr;
    graph_key.clear();
}

int WaveBuffers::Ensure(uint32_t chunk, uint32_t cap_q, uint32_t cap_s, cudaStream_t st) {
    if (chunk <= this->chunk && cap_q <= q.cap_q && cap_s <= q.cap_s && !ptrs.empty()) return AZ_OK;
    DropGraph();   // it refers to the buffers freed below
    for (void *p : ptrs) PoolFree(p, st);
    ptrs.clear();
    memset(&q, 0, sizeof(q));
    auto alloc = [&](size_t bytes) -> void * {
        void *p = nullptr;
        if (PoolAlloc(&p, bytes, st) != cudaSuccess) return nullptr;
        ptrs.push_back(p);
        return p;
    };
    for (int b = 0; b < 2; b++) {
        q.o[b] = (float4 *)alloc((size_t)cap_q * sizeof(float4));
        q.d[b] = (float4 *)alloc((size_t)cap_q * sizeof(float4));
        q.tp[b] = (float4 *)alloc((size_t)cap_q * sizeof(float4));
        q.att[b] = (float4 *)alloc((size_t)cap_q * sizeof(float4));
        q.digits[b] = (uint32_t *)alloc((size_t)cap_q * sizeof(uint32_t));
        if (!q.o[b] || !q.d[b] || !q.tp[b] || !q.att[b] || !q.digits[b]) return SetError(AZ_ERR_OUT_OF_MEMORY, "wave queues");
    }
    q.hit = (uint4 *)alloc((size_t)cap_q * sizeof(uint4));
    q.so = (float4 *)alloc((size_t)cap_s * sizeof(float4));
    q.sd = (float4 *)alloc((size_t)cap_s * sizeof(float4));
    q.sc = (float4 *)alloc((size_t)cap_s * sizeof(float4));
    q.smeta = (uint32_t *)alloc((size_t)cap_s * sizeof(uint32_t));
    q.accum = (float4 *)alloc((size_t)chunk * sizeof(float4));
    q.counts = (uint32_t *)alloc(AZ_COUNT_TOTAL * sizeof(uint32_t));
    wave_dev = (uint64_t *)alloc(4 * sizeof(uint64_t));
    if (!q.hit || !q.so || !q.sd || !q.sc || !q.smeta || !q.accum || !q.counts || !wave_dev)
        return SetError(AZ_ERR_OUT_OF_MEMORY, "wave queues");
    q.cap_q = cap_q;
    q.cap_s = cap_s;
    this->chunk = chunk;
    return AZ_OK;
}

// CUDA events between the stages of every level; summed per stage.
struct StageTimer {
    std::vector<cudaEvent_t> ev;
    std::vector<int> kind;   // event k ends stage kind[k]-1 when kind[k] > 0
    float ms[3] = {0, 0, 0};
    void Mark(cudaStream_t st, int k) {
        cudaEvent_t e;
        cudaEventCreate(&e);
        cudaEventRecord(e, st);
        ev.push_back(e);
        kind.push_back(k);
    }
    void Collect() {   // after a stream synchronize
        for (size_t i = 1; i < ev.size(); i++) {
            if (kind[i] >= 1 && kind[i - 1] == kind[i] - 1) {
                float t = 0.0f;
                cudaEventElapsedTime(&t, ev[i - 1], ev[i]);
                ms[kind[i] - 1] += t;
            }
        }
        for (cudaEvent_t e : ev) cudaEventDestroy(e);
        ev.clear();
        kind.clear();
    }
    ~StageTimer() {
        for (cudaEvent_t e : ev) cudaEventDestroy(e);
    }
};

// Renders samples [start, start+n) of the scissor into `film`; returns the
// per-wave counters (path and shadow queue sizes per level, overflow flag).
// Launches of one wave.  With `capture`, the launches read the wave's first
// sample, size and seed from W.wave_dev (set before every replay of the
// captured graph) and size their grids for `n` = the largest wave.
// Sorts the extension (shadow = 0) or shadow queue of `level` by origin cell
// into its visiting order (k_order_keys + a 16-bit radix sort).
static int OrderQueue(const GpuScene &G, const WaveQueues &Q, WaveBuffers &W, uint32_t level, int shadow, int sms,
                      cudaStream_t st, RenderCounters &rc) {
    const uint32_t cap = shadow ? Q.cap_s : Q.cap_q;
    k_order_keys<<<sms * 8, 256, 0, st>>>(G.dev, Q, level, shadow, cap, W.okey[0], W.oval);
    rc.launches++;
    AZ_CUDA_TRY(cub::DeviceRadixSort::SortPairs(W.otemp, W.otemp_bytes, W.okey[0], W.okey[1], W.oval,
                                                shadow ? W.oidx_s : W.oidx_e, (int)cap, 0, 16, st));
    return AZ_OK;
}

// The device side of a tile wave (az_gpu_render_tiles): the wave's tiles, the
// counter its camera kernel pulls them with, and the jobs' cameras and films.
struct TileWave {
    const Tile *tiles;
    uint32_t ntiles;
    uint32_t *next;
    uint2 *slot_map;
    const CameraParams *cams;
    az_pixel *const *films;
    const DevScene *scenes;   // jobs of several scenes: their device records (null: one scene)
    const DevScene *dev;      // and the host record the launches are chosen for (null: the scene's own)
};

static int RenderWave(const GpuScene &G, const CameraParams &cam, WaveBuffers &W, uint64_t start, uint32_t n,
                      az_pixel *film, cudaStream_t st, int sms, RenderCounters &rc, StageTimer *timer,
                      GuideState *guide, bool train, bool capture = false, const TileWave *tw = nullptr) {
    WaveQueues Q = W.q;
    if (tw) {
        Q.slot_map = tw->slot_map;
        Q.job_cams = tw->cams;
        Q.scenes = tw->scenes;
    }
    // the scene the launches are chosen for: a tile wave of several scenes
    // passes one whose features, depth and light kinds cover all of them
    const DevScene &D = tw && tw->dev ? *tw->dev : G.dev;
    if (capture) Q.wave = W.wave_dev;
    if (cam.order & kOrderExtend) Q.eorder = W.oidx_e;
    if (cam.order & kOrderShadow) Q.sorder = W.oidx_s;
    // While the guide trains, its early proposals can be far from the light
    // field; capping the chance of sampling them at one half keeps every
    // sample's weight within twice cosine sampling's (the estimate stays
    // unbiased for any cap).  Inference-only renders use the learned value.
    Q.guide_alpha_max = train ? 0.5f : 1.0f;
    const uint32_t levels = std::min<uint32_t>(D.max_depth + 1, AZ_MAX_LEVELS - 2);
    if (guide) {
        // proposals for every queue entry this wave can hold (the queue is capped to match)
        int grc = GuidePrepareWave(*guide, W, Q, std::min<uint32_t>(Q.cap_q, n + n / 2 + 1024), train ? levels : 0u, st);
        if (grc != AZ_OK) return grc;
    }
    AZ_CUDA_TRY(cudaMemsetAsync(Q.counts, 0, AZ_COUNT_TOTAL * sizeof(uint32_t), st));
    if (!capture) {
        uint32_t first = n;
        AZ_CUDA_TRY(cudaMemcpyAsync(Q.counts + 1, &first, sizeof(uint32_t), cudaMemcpyHostToDevice, st));
    }
    if (tw) {
        AZ_CUDA_TRY(cudaMemsetAsync(tw->next, 0, sizeof(uint32_t), st));
        k_camera_tiles<<<std::min<uint32_t>(tw->ntiles, (uint32_t)sms * 8), 256, 0, st>>>(tw->tiles, tw->ntiles,
                                                                                          tw->next, Q, tw->slot_map);
    } else {
        k_camera<<<(n + 255) / 256, 256, 0, st>>>(cam, Q, start, n);
    }
    rc.launches++;
    const int grid = sms * 16;
    const uint32_t v = cam.variant;
    // Level L's visibility queries need only its shading; level L+1's
    // closest-hit queries need the same.  Run them side by side (visibility
    // on the side stream) so that the tail of one fills with the other's work;
    // the next shading waits for both.  Not with stage timing, nor with queue
    // ordering (both orderings share one sort scratch).
    const bool overlap = W.side && !timer && !cam.order && !cam.serial_levels;
    if (overlap) {
        LaunchTraversalVariant(v, false, sms, D, cam, Q, 1, st);
        for (uint32_t L = 1; L <= levels; L++) {
            if (guide && L + 1 <= D.max_depth + 1) {   // the deepest level spawns nothing to guide
                int grc = GuideInfer(*guide, G, Q, L, st);
                if (grc != AZ_OK) return grc;
                rc.launches++;
            }
            LaunchShade(grid, D, cam, Q, start, L, st);
            AZ_CUDA_TRY(cudaEventRecord(W.ev_fork, st));
            AZ_CUDA_TRY(cudaStreamWaitEvent(W.side, W.ev_fork, 0));
            LaunchTraversalVariant(cam.shadow_variant, true, sms, D, cam, Q, L, W.side);
            AZ_CUDA_TRY(cudaEventRecord(W.ev_join, W.side));
            if (L < levels) LaunchTraversalVariant(v, false, sms, D, cam, Q, L + 1, st);
            AZ_CUDA_TRY(cudaStreamWaitEvent(st, W.ev_join, 0));
            rc.launches += 3 + D.full_light_queries + D.entity_lights;
            rc.extend_launches++;
        }
    }
    for (uint32_t L = 1; L <= levels && !overlap; L++) {
        if (timer) timer->Mark(st, 0);
        if (cam.order & kOrderExtend) {
            int orc = OrderQueue(G, Q, W, L, 0, sms, st, rc);
            if (orc != AZ_OK) return orc;
        }
        LaunchTraversalVariant(v, false, sms, D, cam, Q, L, st);
        if (guide && L + 1 <= D.max_depth + 1) {   // the deepest level spawns nothing to guide
            int grc = GuideInfer(*guide, G, Q, L, st);
            if (grc != AZ_OK) return grc;
            rc.launches++;
        }
        if (timer) timer->Mark(st, 1);
        LaunchShade(grid, D, cam, Q, start, L, st);
        if (timer) timer->Mark(st, 2);
        if (cam.order & kOrderShadow) {
            int orc = OrderQueue(G, Q, W, L, 1, sms, st, rc);
            if (orc != AZ_OK) return orc;
        }
        LaunchTraversalVariant(cam.shadow_variant, true, sms, D, cam, Q, L, st);
        if (timer) timer->Mark(st, 3);
        rc.launches += 3 + D.full_light_queries + D.entity_lights;
        rc.extend_launches++;
    }
    if (guide && train) {
        int grc = GuideTrainWave(*guide, Q, st);
        if (grc != AZ_OK) return grc;
        rc.launches += 7;
    }
    if (tw) k_splat_tiles<<<(n + 255) / 256, 256, 0, st>>>(Q, n, tw->films);
    else k_splat<<<(n + 255) / 256, 256, 0, st>>>(cam, Q, start, n, film);
    rc.launches++;
    AZ_CUDA_TRY(cudaGetLastError());
    return AZ_OK;
}

// The descriptor that a replayed wave reads (no pinned memory to keep, and no
// wait for a copy from pageable memory).
__global__ void k_set_wave(uint64_t *wave, uint64_t start, uint64_t n, uint64_t seed) {
    wave[0] = start;
    wave[1] = n;
    wave[2] = seed;
}

// One wave through the captured graph of W (captured on the second wave of the
// same scene, camera, film, launch configuration and largest wave).
static int ReplayWave(const GpuScene &G, const CameraParams &cam, WaveBuffers &W, uint64_t start, uint32_t n,
                      uint32_t n_max, az_pixel *film, cudaStream_t st, int sms, RenderCounters &rc) {
    struct Key {
        const GpuScene *g;
        az_pixel *film;
        CameraParams cam;
        uint32_t n_max, cap_q, cap_s;
        int sms;
        const void *q0;
    } key;
    memset(&key, 0, sizeof(key));
    key.g = &G;
    key.film = film;
    key.cam = cam;
    key.cam.seed = 0;   // read from the descriptor
    key.n_max = n_max;
    key.cap_q = W.q.cap_q;
    key.cap_s = W.q.cap_s;
    key.sms = sms;
    key.q0 = W.q.o[0];
    const unsigned char *kb = reinterpret_cast<const unsigned char *>(&key);
    RenderCounters launches{};
    const auto same = [&](const std::vector<unsigned char> &k) {
        return k.size() == sizeof(key) && memcmp(k.data(), kb, sizeof(key)) == 0;
    };
    if (!W.graph || !same(W.graph_key)) {
        // The first wave of a kind is launched directly: capturing and
        // instantiating its graph takes as long as several waves of a small
        // render, and a one-shot image has no second one.
        if (!same(W.direct_key)) {
            W.direct_key.assign(kb, kb + sizeof(key));
            return RenderWave(G, cam, W, start, n, film, st, sms, rc, nullptr, nullptr, false);
        }
        W.DropGraph();
        AZ_CUDA_TRY(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        int crc = RenderWave(G, cam, W, 0, n_max, film, st, sms, launches, nullptr, nullptr, false, true);
        cudaGraph_t graph = nullptr;
        cudaError_t e = cudaStreamEndCapture(st, &graph);
        if (crc != AZ_OK) {
            if (graph) cudaGraphDestroy(graph);
            return crc;
        }
        if (e != cudaSuccess) return CudaError(e, "capturing the wave launches");
        e = cudaGraphInstantiate(&W.graph, graph, 0);
        cudaGraphDestroy(graph);
        if (e != cudaSuccess) {
            W.graph = nullptr;
            return CudaError(e, "instantiating the wave graph");
        }
        W.graph_key.assign(kb, kb + sizeof(key));
        W.graph_launches = launches.launches;
        W.graph_extend_launches = launches.extend_launches;
    }
    k_set_wave<<<1, 1, 0, st>>>(W.wave_dev, start, n, cam.seed);
    AZ_CUDA_TRY(cudaGraphLaunch(W.graph, st));
    rc.launches += W.graph_launches;
    rc.extend_launches += W.graph_extend_launches;
    return AZ_OK;
}

// in kVariants: {0, 32}, {8, 32}, {8, 8}, {8, 12}
constexpr uint32_t kLoop = 10, kTogether = 9, kEight = 7, kTwelve = 3;
void ChooseDefaultVariants(GpuScene &G) {
    // Scenes of a few nodes (Cornell box 1 + 1, 1 M samples: 1.61 ms a frame
    // with one query per thread, 1.82 by phases).  The visibility queries of
    // several kinds of light take different paths in a warp all the same (the
    // features scene, six lights: 6.2 ms one per thread, 3.9 by phases).
    if (G.node_count <= 64) {
        G.variant = kLoop;
        G.shadow_variant = G.dev.light_count + (G.dev.use_env_map ? 1u : 0u) <= 2 ? kLoop : kTogether;
        return;
    }
    // Larger hierarchies (dense mesh / interior / moving spheres, full frames,
    // with 6, 8, 10 and 14 waiting lanes): closest hits 91 / 170 / 114,
    // 89 / 170 / 115, 88 / 171 / 117, 89 / 178 / 120 ms; visibility with 6, 10
    // and 14: 69 / 65 / 19.6, 66 / 67 / 20.2, 64 / 69 / 21.1 ms.
    G.variant = kEight;
    G.shadow_variant = kTwelve;
}

// The launch configurations of a render: the one the caller names (for both
// traversal kernels), else the scene's.  A wave of several scenes has no form
// with one query per thread, so it takes the default lanes for a scene's that
// is meant for it: with all 32 lanes waiting for each other, 24 jobs of three
// scenes take 25.6 ms, with 8 and 12 18.8.
static int ChooseVariants(const GpuScene &G, const az_render_opts *opts, CameraParams &cam, bool several = false) {
    cam.variant = opts && opts->variant ? opts->variant - 1 : G.variant;
    if (cam.variant >= kVariantCount) return SetError(AZ_ERR_INVALID_ARGUMENT, "unknown launch variant");
    cam.shadow_variant = (opts && opts->variant) || G.shadow_variant >= kVariantCount ? cam.variant : G.shadow_variant;
    if (several && kVariants[cam.variant].minb == 0) cam.variant = kEight;
    if (several && kVariants[cam.shadow_variant].minb == 0) cam.shadow_variant = kTwelve;
    cam.refill = kVariants[cam.variant].refill;
    cam.shadow_refill = kVariants[cam.shadow_variant].refill;
    return AZ_OK;
}

// The queue ordering of a render: the flags', else the scene's choice.
static uint32_t QueueOrder(const GpuScene &G, const az_render_opts *opts) {
    const uint32_t f = opts ? opts->flags : 0u;
    if (f & AZ_FLAG_ORDER_NONE) return 0u;
    if (f & (AZ_FLAG_ORDER_SHADOW | AZ_FLAG_ORDER_EXTEND))
        return ((f & AZ_FLAG_ORDER_SHADOW) ? kOrderShadow : 0u) | ((f & AZ_FLAG_ORDER_EXTEND) ? kOrderExtend : 0u);
    return G.order;
}

// The default wave of a render: as many camera samples as a quarter of the
// free device memory holds in wave queues, a power of two from 2^22 to 2^26.
// Bigger waves keep the launches of the deep tree levels, where most paths
// have ended, full (C1: 427 ms per frame at 2^22, 393 at 2^24, 383 at 2^26).
// The queues `W` already holds and what the pool keeps unused count as free, so
// that repeated renders of a scene keep their wave size.
static uint32_t DefaultWave(uint32_t per_node_shadow, const WaveBuffers &W, uint64_t total) {
    uint64_t n = 1u << 22;
    if (total <= n) return (uint32_t)n;   // one wave of the smallest size holds the render
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) {
        cudaGetLastError();
        return (uint32_t)n;
    }
    // per sample: 1.5 queue entries of 168 bytes (two ping-pong sets of four
    // float4, digits, hit), shadow entries of 52 bytes, one float4 sum
    const double shadow_entries = std::min(1.5 * std::max(per_node_shadow, 1u), 4.0);
    const double per_sample = 1.5 * 168.0 + shadow_entries * 52.0 + 16.0;
    const double held = W.ptrs.empty() ? 0.0
                                       : (double)W.q.cap_q * 168.0 + (double)W.q.cap_s * 52.0 + (double)W.chunk * 16.0;
    const uint64_t fit = (uint64_t)(((double)free_b + (double)PoolUnused() + held) / 4.0 / per_sample);
    while (n * 2 <= fit && n < (1u << 26)) n *= 2;
    return (uint32_t)n;
}

int Render(GpuScene &G, az_pixel *film, const az_camera *camera, const az_epsilon_values *eps, az_scissor sc,
           int32_t filter, uint32_t cull, const az_render_opts *opts, cudaStream_t st, az_render_stats *stats,
           GuideState *guide, bool train, WaveBuffers *wave_buffers, float4 *sample_out) {
    CameraParams cam;
    int rc = SetupCamera(camera, sc, filter, cull, eps, opts ? opts->seed : 0, cam);
    if (rc != AZ_OK) return rc;
    cam.sample_out = sample_out;
    cam.count_traversal = opts && (opts->flags & AZ_FLAG_COUNT_TRAVERSAL) ? 1u : 0u;
    cam.env_importance = opts && (opts->flags & AZ_FLAG_ENV_IMPORTANCE) && G.dev.env_rows ? 1u : 0u;
    if ((rc = ChooseVariants(G, opts, cam)) != AZ_OK) return rc;
    cam.order = QueueOrder(G, opts);
    cam.serial_levels = opts && (opts->flags & AZ_FLAG_SERIAL_LEVELS) ? 1u : 0u;
    cam.watertight = opts && (opts->flags & AZ_FLAG_WATERTIGHT) ? 1u : 0u;
    if (G.dev.max_depth + 1 > AZ_MAX_LEVELS - 2) return SetError(AZ_ERR_UNSUPPORTED, "MaxRecursionDepth above 61");
    const uint64_t all = cam.npix * (uint64_t)cam.sqrt_spp * cam.sqrt_spp;
    // a part of the camera-sample sequence (one GPU's share of a frame)
    uint64_t begin = 0, end = all;
    if (opts && opts->sample_parts > 1) {
        if (opts->sample_part >= opts->sample_parts)
            return SetError(AZ_ERR_INVALID_ARGUMENT, "sample_part must be below sample_parts");
        begin = all / opts->sample_parts * opts->sample_part +
                std::min<uint64_t>(opts->sample_part, all % opts->sample_parts);
        end = begin + all / opts->sample_parts + (opts->sample_part < all % opts->sample_parts ? 1 : 0);
    }
    const uint64_t total = end - begin;
    if (stats) memset(stats, 0, sizeof(*stats));
    if (total == 0) return AZ_OK;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, G.device);
    uint32_t per_node_shadow = G.dev.light_count + (G.dev.use_env_map ? 1u : 0u);
    WaveBuffers &W = wave_buffers ? *wave_buffers : G.waves;
    uint32_t chunk = opts && opts->chunk_samples ? opts->chunk_samples : DefaultWave(per_node_shadow, W, total);
    // a training render updates the guide after every wave: smaller waves, more updates
    if (guide && train && !(opts && opts->chunk_samples)) chunk = 1u << 20;
    // the visit counters are 32-bit per wave: counting renders keep 2^22-sample waves
    if (cam.count_traversal && !(opts && opts->chunk_samples)) chunk = std::min(chunk, 1u << 22);
    chunk = (uint32_t)std::min<uint64_t>(chunk, total);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    if (stats) {
        AZ_CUDA_TRY(cudaEventCreate(&e0));
        AZ_CUDA_TRY(cudaEventCreate(&e1));
        AZ_CUDA_TRY(cudaEventRecord(e0, st));
    }
    RenderCounters counters{};
    std::vector<uint32_t> host_counts(AZ_COUNT_TOTAL);
    std::unique_ptr<StageTimer> timer;
    if (stats && opts && (opts->flags & AZ_FLAG_TIME_STAGES)) timer.reset(new StageTimer());
    // The launches of a wave run as one CUDA graph from the second wave of a
    // scene, camera, film and launch configuration on (ReplayWave), with each
    // wave's first sample, size and seed in a 24-byte descriptor.  Not for stage
    // timing, guided renders, or a legacy default stream (which cannot be
    // captured).
    const bool use_graph = !(opts && (opts->flags & AZ_FLAG_NO_GRAPH)) && !timer && !guide && st != nullptr &&
                           st != cudaStreamLegacy && st != cudaStreamPerThread;
    uint64_t pos = begin;
    while (pos < end) {
        uint32_t n = (uint32_t)std::min<uint64_t>(chunk, end - pos);
        uint32_t cap_q = std::max<uint32_t>(n + n / 2, 1024);
        uint32_t cap_s = std::max<uint32_t>((uint32_t)std::min<uint64_t>((uint64_t)cap_q * std::max(per_node_shadow, 1u),
                                                                         (uint64_t)n * 4), 1024);
        rc = W.Ensure(n, cap_q, cap_s, st);
        if (rc != AZ_OK) return rc;
        if (cam.order && (rc = W.EnsureOrder(std::max(W.q.cap_q, W.q.cap_s), st)) != AZ_OK) return rc;
        if (!cam.serial_levels && (rc = W.EnsureSide()) != AZ_OK) return rc;
        if (use_graph) {
            rc = ReplayWave(G, cam, W, pos, n, chunk, film, st, sms, counters);
        } else {
            rc = RenderWave(G, cam, W, pos, n, film, st, sms, counters, timer.get(), guide, train);
        }
        if (rc != AZ_OK) return rc;
        AZ_CUDA_TRY(cudaMemcpyAsync(host_counts.data(), W.q.counts, AZ_COUNT_TOTAL * sizeof(uint32_t),
                                    cudaMemcpyDeviceToHost, st));
        AZ_CUDA_TRY(cudaStreamSynchronize(st));
        if (timer) timer->Collect();
        if (host_counts[AZ_COUNT_ERROR])
            return SetError(AZ_ERR_CUDA, "BVH traversal exceeded its step limit (corrupt hierarchy)");
        if (host_counts[AZ_COUNT_OVERFLOW]) {
            // a queue overflowed: this wave wrote nothing; retry it with half the samples
            if (n <= 1024) return SetError(AZ_ERR_OUT_OF_MEMORY, "wave queue overflow with 1024 samples");
            chunk = std::max<uint32_t>(n / 2, 1024);
            counters.retries++;
            continue;
        }
        for (uint32_t L = 1; L < AZ_MAX_LEVELS; L++) {
            counters.extend += host_counts[L];
            counters.shadow += host_counts[AZ_COUNT_SHADOW + L];
        }
        counters.nodes += host_counts[AZ_COUNT_NODES];
        counters.prims += host_counts[AZ_COUNT_NODES + 1];
        counters.snodes += host_counts[AZ_COUNT_SNODES];
        counters.sprims += host_counts[AZ_COUNT_SNODES + 1];
        counters.chunks++;
        pos += n;
    }
    if (stats) {
        AZ_CUDA_TRY(cudaEventRecord(e1, st));
        AZ_CUDA_TRY(cudaEventSynchronize(e1));
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, e0, e1);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        stats->samples = total;
        stats->extend_rays = counters.extend;
        stats->shadow_rays = counters.shadow;
        stats->chunks = counters.chunks;
        stats->retries = counters.retries;
        stats->kernel_launches = counters.launches;
        stats->gpu_ms = ms;
        stats->node_visits = counters.nodes;
        stats->prim_visits = counters.prims;
        stats->shadow_node_visits = counters.snodes;
        stats->shadow_prim_visits = counters.sprims;
        stats->extend_launches = (uint32_t)counters.extend_launches;
        if (timer) {
            stats->extend_ms = timer->ms[0];
            stats->shade_ms = timer->ms[1];
            stats->shadow_ms = timer->ms[2];
        }
    }
    return AZ_OK;
}

int RenderTiles(GpuScene &G, std::vector<TileJob> &jobs, const az_render_opts *opts, cudaStream_t st,
                az_render_stats *stats, cudaEvent_t origin) {
    if (stats) memset(stats, 0, sizeof(*stats));
    if (jobs.empty()) return AZ_OK;
    const uint32_t nj = (uint32_t)jobs.size();
    // the jobs' scenes: one, or a table the kernels index per queue entry
    std::vector<GpuScene *> scenes;
    std::vector<uint32_t> scene_of(nj, 0);
    for (uint32_t j = 0; j < nj; j++) {
        GpuScene *sg = jobs[j].scene ? jobs[j].scene : &G;
        if (sg->device != G.device) return SetError(AZ_ERR_INVALID_ARGUMENT, "tile jobs on different devices");
        auto it = std::find(scenes.begin(), scenes.end(), sg);
        if (it == scenes.end()) {
            if (scenes.size() == kMaxWaveScenes)
                return SetError(AZ_ERR_UNSUPPORTED, "a tile render of more than 256 scenes");
            scenes.push_back(sg);
            it = scenes.end() - 1;
        }
        scene_of[j] = (uint32_t)(it - scenes.begin());
    }
    const bool multi = scenes.size() > 1;
    // the record the launches are chosen for: the first scene's, with the
    // features, light kinds and depth of all of them; the launch configuration
    // is that of the scene with the most nodes, whose queries take the time
    DevScene wave_dev = scenes[0]->dev;
    const GpuScene *largest = scenes[0];
    uint32_t per_node_shadow = 0;
    for (GpuScene *sg : scenes) {
        const DevScene &d = sg->dev;
        if (sg->node_count > largest->node_count) largest = sg;
        if (d.max_depth + 1 > AZ_MAX_LEVELS - 2) return SetError(AZ_ERR_UNSUPPORTED, "MaxRecursionDepth above 61");
        wave_dev.features |= d.features;
        wave_dev.full_light_queries |= d.full_light_queries;
        wave_dev.entity_lights |= d.entity_lights;
        wave_dev.top_spheres += d.top_spheres;
        wave_dev.max_depth = std::max(wave_dev.max_depth, d.max_depth);
        per_node_shadow = std::max(per_node_shadow, d.light_count + (d.use_env_map ? 1u : 0u));
    }
    std::vector<CameraParams> cams(nj);
    uint64_t total = 0;
    for (uint32_t j = 0; j < nj; j++) {
        const TileJob &J = jobs[j];
        const GpuScene &Gj = *scenes[scene_of[j]];
        if (!J.film || !J.camera) return SetError(AZ_ERR_INVALID_ARGUMENT, "tile job without film or camera");
        CameraParams &c = cams[j];
        int rc = SetupCamera(J.camera, J.scissor, J.filter, J.cull, J.eps, J.seed, c);
        if (rc != AZ_OK) return rc;
        c.scene = scene_of[j];
        c.count_traversal = opts && (opts->flags & AZ_FLAG_COUNT_TRAVERSAL) ? 1u : 0u;
        c.env_importance = opts && (opts->flags & AZ_FLAG_ENV_IMPORTANCE) && Gj.dev.env_rows ? 1u : 0u;
        if ((rc = ChooseVariants(*largest, opts, c, multi)) != AZ_OK) return rc;
        // several scenes: no queue ordering (its keys use one scene's bounds)
        c.order = multi ? 0u : QueueOrder(G, opts);
        c.serial_levels = opts && (opts->flags & AZ_FLAG_SERIAL_LEVELS) ? 1u : 0u;
        c.watertight = opts && (opts->flags & AZ_FLAG_WATERTIGHT) ? 1u : 0u;
        // the traversal and shading kernels take these from the wave's first job
        if (c.eps_isect != cams[0].eps_isect || c.eps_shadow != cams[0].eps_shadow || c.cull != cams[0].cull)
            return SetError(AZ_ERR_INVALID_ARGUMENT, "the jobs of a tile render need the same epsilons and culling");
        const uint64_t samples = c.npix * (uint64_t)c.sqrt_spp * c.sqrt_spp;
        if (samples >= (1ull << 32)) return SetError(AZ_ERR_UNSUPPORTED, "a tile job with 2^32 samples or more");
        jobs[j].samples = samples;
        jobs[j].done_ms = 0.0f;
        total += samples;
    }
    if (total == 0) return AZ_OK;
    // every job's samples in runs of kTile consecutive sample indices (one
    // sample number over a run of pixels: coherent camera rays), jobs of one
    // scene after another: a warp's lanes then mostly read one scene
    constexpr uint32_t kTile = 4096;
    std::vector<Tile> tiles;
    std::vector<size_t> last_tile(nj, 0);
    std::vector<uint32_t> by_scene(nj);
    for (uint32_t j = 0; j < nj; j++) by_scene[j] = j;
    std::stable_sort(by_scene.begin(), by_scene.end(),
                     [&](uint32_t a, uint32_t b) { return scene_of[a] < scene_of[b]; });
    for (uint32_t j : by_scene) {
        for (uint64_t first = 0; first < jobs[j].samples; first += kTile)
            tiles.push_back(Tile{j, (uint32_t)first, (uint32_t)std::min<uint64_t>(kTile, jobs[j].samples - first), 0u});
        last_tile[j] = tiles.size();   // one past the job's last tile
    }
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, G.device);
    uint32_t chunk = opts && opts->chunk_samples ? opts->chunk_samples : DefaultWave(per_node_shadow, G.waves, total);
    chunk = std::max<uint32_t>((uint32_t)std::min<uint64_t>(chunk, total), kTile);
    WaveBuffers &W = G.waves;
    // device tables: cameras, films, this wave's tiles, the work-queue counter, slot -> (job, sample)
    PoolBuf<CameraParams> d_cams;
    PoolBuf<az_pixel *> d_films;
    PoolBuf<Tile> d_tiles;
    PoolBuf<uint32_t> d_next;
    PoolBuf<uint2> d_slots;
    PoolBuf<DevScene> d_scenes;
    std::vector<az_pixel *> films(nj);
    for (uint32_t j = 0; j < nj; j++) films[j] = jobs[j].film;
    AZ_CUDA_TRY(d_cams.alloc(nj, st));
    AZ_CUDA_TRY(d_films.alloc(nj, st));
    AZ_CUDA_TRY(d_tiles.alloc(chunk / kTile + 2 + nj, st));
    AZ_CUDA_TRY(d_next.alloc(1, st));
    AZ_CUDA_TRY(d_slots.alloc(chunk, st));
    AZ_CUDA_TRY(cudaMemcpyAsync(d_cams.p, cams.data(), nj * sizeof(CameraParams), cudaMemcpyHostToDevice, st));
    AZ_CUDA_TRY(cudaMemcpyAsync(d_films.p, films.data(), nj * sizeof(az_pixel *), cudaMemcpyHostToDevice, st));
    std::vector<DevScene> scene_recs;
    if (multi) {
        for (GpuScene *sg : scenes) scene_recs.push_back(sg->dev);
        AZ_CUDA_TRY(d_scenes.alloc(scene_recs.size(), st));
        AZ_CUDA_TRY(cudaMemcpyAsync(d_scenes.p, scene_recs.data(), scene_recs.size() * sizeof(DevScene),
                                    cudaMemcpyHostToDevice, st));
    }
    struct Events {
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        ~Events() {
            if (e0) cudaEventDestroy(e0);
            if (e1) cudaEventDestroy(e1);
        }
    } ev;
    AZ_CUDA_TRY(cudaEventCreate(&ev.e0));
    AZ_CUDA_TRY(cudaEventCreate(&ev.e1));
    AZ_CUDA_TRY(cudaEventRecord(ev.e0, st));
    RenderCounters counters{};
    std::vector<uint32_t> host_counts(AZ_COUNT_TOTAL);
    size_t ti = 0;
    while (ti < tiles.size()) {
        // the wave: the next tiles while they fit in `chunk` samples (the
        // tile table holds at most chunk / kTile + 2 + nj of them)
        uint32_t n = 0;
        size_t te = ti;
        while (te < tiles.size() && n + tiles[te].count <= chunk) {
            tiles[te].slot = n;
            n += tiles[te].count;
            te++;
        }
        const uint32_t ntiles = (uint32_t)(te - ti);
        const uint32_t cap_q = std::max<uint32_t>(n + n / 2, 1024);
        const uint32_t cap_s = std::max<uint32_t>(
            (uint32_t)std::min<uint64_t>((uint64_t)cap_q * std::max(per_node_shadow, 1u), (uint64_t)n * 4), 1024);
        int rc = W.Ensure(n, cap_q, cap_s, st);
        if (rc != AZ_OK) return rc;
        if (cams[0].order && (rc = W.EnsureOrder(std::max(W.q.cap_q, W.q.cap_s), st)) != AZ_OK) return rc;
        if (!cams[0].serial_levels && (rc = W.EnsureSide()) != AZ_OK) return rc;
        AZ_CUDA_TRY(cudaMemcpyAsync(d_tiles.p, tiles.data() + ti, ntiles * sizeof(Tile), cudaMemcpyHostToDevice, st));
        TileWave tw{d_tiles.p, ntiles, d_next.p, d_slots.p, d_cams.p, d_films.p,
                    multi ? d_scenes.p : nullptr, multi ? &wave_dev : nullptr};
        rc = RenderWave(G, cams[0], W, 0, n, nullptr, st, sms, counters, nullptr, nullptr, false, false, &tw);
        if (rc != AZ_OK) return rc;
        AZ_CUDA_TRY(cudaMemcpyAsync(host_counts.data(), W.q.counts, AZ_COUNT_TOTAL * sizeof(uint32_t),
                                    cudaMemcpyDeviceToHost, st));
        AZ_CUDA_TRY(cudaEventRecord(ev.e1, st));
        AZ_CUDA_TRY(cudaEventSynchronize(ev.e1));
        if (host_counts[AZ_COUNT_ERROR])
            return SetError(AZ_ERR_CUDA, "BVH traversal exceeded its step limit (corrupt hierarchy)");
        if (host_counts[AZ_COUNT_OVERFLOW]) {
            // a queue overflowed: this wave wrote nothing; retry it with half the samples
            if (n <= kTile) return SetError(AZ_ERR_OUT_OF_MEMORY, "wave queue overflow with one tile");
            chunk = std::max<uint32_t>(n / 2, kTile);
            counters.retries++;
            continue;
        }
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, origin ? origin : ev.e0, ev.e1);
        for (uint32_t j = 0; j < nj; j++)
            if (last_tile[j] > ti && last_tile[j] <= te) jobs[j].done_ms = ms;
        for (uint32_t L = 1; L < AZ_MAX_LEVELS; L++) {
            counters.extend += host_counts[L];
            counters.shadow += host_counts[AZ_COUNT_SHADOW + L];
        }
        counters.nodes += host_counts[AZ_COUNT_NODES];
        counters.prims += host_counts[AZ_COUNT_NODES + 1];
        counters.snodes += host_counts[AZ_COUNT_SNODES];
        counters.sprims += host_counts[AZ_COUNT_SNODES + 1];
        counters.chunks++;
        ti = te;
    }
    if (stats) {
        float ms = 0.0f;
        cudaEventElapsedTime(&ms, ev.e0, ev.e1);
        stats->samples = total;
        stats->extend_rays = counters.extend;
        stats->shadow_rays = counters.shadow;
        stats->chunks = counters.chunks;
        stats->retries = counters.retries;
        stats->kernel_launches = counters.launches;
        stats->gpu_ms = ms;
        stats->node_visits = counters.nodes;
        stats->prim_visits = counters.prims;
        stats->shadow_node_visits = counters.snodes;
        stats->shadow_prim_visits = counters.sprims;
        stats->extend_launches = (uint32_t)counters.extend_launches;
    }
    return AZ_OK;
}

// Times every launch variant on a band of the frame (the middle eighth of the
// scissor's rows, all samples) and keeps the fastest for this scene.
int Autotune(GpuScene &G, const az_camera *camera, const az_epsilon_values *eps, az_scissor sc, int32_t filter,
             uint32_t cull, const az_render_opts *opts, cudaStream_t st, uint32_t *best_out, float *ms_out) {
    CameraParams cam;
    int rc = SetupCamera(camera, sc, filter, cull, eps, opts ? opts->seed : 0, cam);
    if (rc != AZ_OK) return rc;
    // at least ~2^20 samples so that the timing is not dominated by launch overhead
    const uint64_t per_row = (uint64_t)cam.wsc * cam.sqrt_spp * cam.sqrt_spp;
    uint32_t rows = std::max<uint32_t>(cam.hsc / 8, (uint32_t)std::min<uint64_t>(cam.hsc, (1u << 20) / std::max<uint64_t>(per_row, 1) + 1));
    rows = std::max<uint32_t>(1, std::min(rows, cam.hsc));
    az_scissor band = sc;
    band.Min.y = cam.r0 + (cam.hsc - rows) / 2;
    band.Max.y = band.Min.y + rows;
    band.Min.x = cam.c0;
    band.Max.x = cam.c0 + cam.wsc;
    size_t bytes = (size_t)cam.width * cam.height * sizeof(az_pixel);
    az_pixel *film = nullptr;
    AZ_CUDA_TRY(DeviceAlloc((void **)&film, bytes));
    float best_ms = FLT_MAX;
    uint32_t best = 0;
    az_render_opts o;
    if (opts) o = *opts;
    else memset(&o, 0, sizeof(o));
    for (uint32_t v = 0; v < kVariantCount && rc == AZ_OK; v++) {
        o.variant = v + 1;
        o.flags &= ~(uint32_t)AZ_FLAG_TIME_STAGES;
        az_render_stats stats;
        float vms = FLT_MAX;
        for (int rep = 0; rep < 3 && rc == AZ_OK; rep++) {   // the first run warms caches and allocates queues
            rc = Render(G, film, camera, eps, band, filter, cull, &o, st, &stats);
            if (rep > 0) vms = std::min(vms, stats.gpu_ms);
        }
        if (rc == AZ_OK && vms < best_ms) {
            best_ms = vms;
            best = v;
        }
    }
    // then the queue ordering with that launch configuration, unless the caller fixed it
    const uint32_t order_flags = AZ_FLAG_ORDER_SHADOW | AZ_FLAG_ORDER_EXTEND | AZ_FLAG_ORDER_NONE;
    uint32_t best_order = QueueOrder(G, opts);
    if (rc == AZ_OK && !(opts && (opts->flags & order_flags))) {
        o.variant = best + 1;
        for (uint32_t ord : {0u, kOrderShadow, kOrderExtend, kOrderShadow | kOrderExtend}) {
            if (ord == best_order || rc != AZ_OK) continue;
            o.flags = (o.flags & ~(order_flags | (uint32_t)AZ_FLAG_TIME_STAGES)) |
                      (ord == 0 ? (uint32_t)AZ_FLAG_ORDER_NONE
                                : ((ord & kOrderShadow) ? (uint32_t)AZ_FLAG_ORDER_SHADOW : 0u) |
                                      ((ord & kOrderExtend) ? (uint32_t)AZ_FLAG_ORDER_EXTEND : 0u));
            az_render_stats stats;
            float oms = FLT_MAX;
            for (int rep = 0; rep < 3 && rc == AZ_OK; rep++) {
                rc = Render(G, film, camera, eps, band, filter, cull, &o, st, &stats);
                if (rep > 0) oms = std::min(oms, stats.gpu_ms);
            }
            if (rc == AZ_OK && oms < best_ms) {
                best_ms = oms;
                best_order = ord;
            }
        }
    }
    // then the shadow queries' configuration alone, with the extension's fixed
    uint32_t best_shadow = best;
    if (rc == AZ_OK) {
        const uint32_t keep_variant = G.variant, keep_order = G.order, keep_shadow = G.shadow_variant;
        G.variant = best;
        G.order = best_order;
        o.variant = 0;   // the scene's configuration, with the shadow variant under test
        o.flags &= ~(uint32_t)AZ_FLAG_TIME_STAGES;
        if (!(opts && (opts->flags & order_flags))) o.flags &= ~order_flags;
        for (uint32_t v = 0; v < kVariantCount && rc == AZ_OK; v++) {
            if (v == best) continue;
            G.shadow_variant = v;
            az_render_stats stats;
            float vms = FLT_MAX;
            for (int rep = 0; rep < 3 && rc == AZ_OK; rep++) {
                rc = Render(G, film, camera, eps, band, filter, cull, &o, st, &stats);
                if (rep > 0) vms = std::min(vms, stats.gpu_ms);
            }
            if (rc == AZ_OK && vms < best_ms) {
                best_ms = vms;
                best_shadow = v;
            }
        }
        G.variant = keep_variant;
        G.order = keep_order;
        G.shadow_variant = keep_shadow;
    }
    cudaFree(film);
    if (rc != AZ_OK) return rc;
    G.variant = best;
    G.shadow_variant = best_shadow;
    G.order = best_order;
    if (best_out) *best_out = best + 1;
    if (ms_out) *ms_out = best_ms;
    return AZ_OK;
}

// ---- closest-hit queries for the parity tests ----
namespace {
template <bool WT>
__global__ void k_closest(DevScene S, const az_ray3 *rays, uint32_t n, uint32_t cull, float eps, uint32_t *hit,
                          uint32_t *uid, uint32_t *face, float *t) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    az_ray3 rr = rays[i];
    Ray r;
    r.o = mk(rr.Origin.x, rr.Origin.y, rr.Origin.z);
    r.d = mk(rr.Direction.x, rr.Direction.y, rr.Direction.z);
    r.time = rr.T;
    Hit h;
    bool ok = trace<Q_CLOSEST, WT>(S, r, cull != 0, eps, FLT_MAX, h);
    hit[i] = ok ? 1u : 0u;
    uid[i] = ok ? S.ents[h.ent].uid : 0xFFFFFFFFu;
    face[i] = ok && h.prim != 0xFFFFFFFFu ? S.tri_attr[h.prim].face_id : 0xFFFFFFFFu;
    t[i] = ok ? h.t : 0.0f;
}
}  // namespace

int ClosestHit(GpuScene &G, const az_ray3 *rays, uint32_t n, int32_t cull, float eps, uint32_t *out_hit,
               uint32_t *out_uid, uint32_t *out_face, float *out_t, cudaStream_t st, bool watertight) {
    if (n == 0) return AZ_OK;
    PoolBuf<char> buf;
    AZ_CUDA_TRY(buf.alloc((size_t)n * (sizeof(az_ray3) + 3 * sizeof(uint32_t) + sizeof(float)) + 64, st));
    char *p = buf.p;
    az_ray3 *d_rays = (az_ray3 *)p;
    p += ((size_t)n * sizeof(az_ray3) + 15) & ~(size_t)15;
    uint32_t *d_hit = (uint32_t *)p;
    uint32_t *d_uid = d_hit + n;
    uint32_t *d_face = d_uid + n;
    float *d_t = (float *)(d_face + n);
    int rc = AZ_OK;
    cudaError_t e = cudaMemcpyAsync(d_rays, rays, (size_t)n * sizeof(az_ray3), cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        if (watertight)
            k_closest<true><<<(n + 127) / 128, 128, 0, st>>>(G.dev, d_rays, n, (uint32_t)cull, eps, d_hit, d_uid,
                                                              d_face, d_t);
        else
            k_closest<false><<<(n + 127) / 128, 128, 0, st>>>(G.dev, d_rays, n, (uint32_t)cull, eps, d_hit, d_uid,
                                                               d_face, d_t);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(out_hit, d_hit, n * 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(out_uid, d_uid, n * 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(out_face, d_face, n * 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaMemcpyAsync(out_t, d_t, n * 4, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) rc = CudaError(e, "closest-hit query");
    return rc;
}

}  // namespace az

// ---------------------------------------------------------------------------
// az_gpu_render_noalloc: the same render with the wave queues in a fixed
// static device array, for callers that must not allocate device memory.
// ---------------------------------------------------------------------------
namespace az {
namespace {

constexpr uint32_t kStaticWave = 16384;                          // camera samples per wave, maximum
constexpr uint32_t kStaticCapQ = kStaticWave + kStaticWave / 2;  // path-queue entries per level buffer
constexpr uint32_t kStaticCapS = 4 * kStaticCapQ;                // light-sample (shadow) entries
constexpr size_t Align256(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t kQ16 = Align256((size_t)kStaticCapQ * 16), kQ4 = Align256((size_t)kStaticCapQ * 4);
constexpr size_t kS16 = Align256((size_t)kStaticCapS * 16), kS4 = Align256((size_t)kStaticCapS * 4);
constexpr size_t kA16 = Align256((size_t)kStaticWave * 16), kC4 = Align256((size_t)AZ_COUNT_TOTAL * 4);
constexpr size_t kStaticBytes = 2 * (4 * kQ16 + kQ4) + kQ16 + 3 * kS16 + kS4 + kA16 + kC4;  // 9,110,784 B

// One copy per GPU that loads this library, held until the process exits.
// Host code must not use this name as an address: it resolves the device
// address once per device with cudaGetSymbolAddress (StaticWaveScratch).
static __device__ __align__(256) unsigned char g_wave_scratch[kStaticBytes];

std::mutex g_wave_scratch_mu;
void *g_wave_scratch_addr[256] = {};

// Device address of g_wave_scratch on the current device (set-up on first use).
int StaticWaveScratch(int device, void **out) {
    std::lock_guard<std::mutex> lock(g_wave_scratch_mu);
    if (device < 0 || device >= 256) return SetError(AZ_ERR_INVALID_ARGUMENT, "device ordinal out of range");
    if (!g_wave_scratch_addr[device]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_wave_scratch);
        if (e != cudaSuccess) return CudaError(e, "cudaGetSymbolAddress(wave scratch)");
        g_wave_scratch_addr[device] = p;
    }
    *out = g_wave_scratch_addr[device];
    return AZ_OK;
}

WaveQueues CarveStaticQueues(unsigned char *p) {
    WaveQueues q;
    memset(&q, 0, sizeof(q));
    for (int b = 0; b < 2; b++) {
        q.o[b] = (float4 *)p; p += kQ16;
        q.d[b] = (float4 *)p; p += kQ16;
        q.tp[b] = (float4 *)p; p += kQ16;
        q.att[b] = (float4 *)p; p += kQ16;
        q.digits[b] = (uint32_t *)p; p += kQ4;
    }
    q.hit = (uint4 *)p; p += kQ16;
    q.so = (float4 *)p; p += kS16;
    q.sd = (float4 *)p; p += kS16;
    q.sc = (float4 *)p; p += kS16;
    q.smeta = (uint32_t *)p; p += kS4;
    q.accum = (float4 *)p; p += kA16;
    q.counts = (uint32_t *)p;
    q.cap_q = kStaticCapQ;
    q.cap_s = kStaticCapS;
    return q;
}

}  // namespace
}  // namespace az

extern "C" int az_gpu_render_noalloc(az_gpu_scene *scene, az_pixel *film, const az_camera *camera,
                                     const az_epsilon_values *epsilons, az_scissor scissor, int32_t filter_type,
                                     uint32_t backface_culling, const az_render_opts *opts) {
    using namespace az;
    if (!scene || !scene->impl || !film || !camera) return SetError(AZ_ERR_INVALID_ARGUMENT, "null argument");
    const GpuScene &G = *scene->impl;
    const int device = opts ? opts->device : G.device;
    uint32_t wave = opts && opts->chunk_samples ? opts->chunk_samples : kStaticWave;
    if (wave > kStaticWave)
        return SetError(AZ_ERR_INVALID_ARGUMENT,
                        "chunk_samples " + std::to_string(wave) + " exceeds the static wave scratch of " +
                            std::to_string(kStaticWave) + " camera samples");
    if (G.dev.max_depth + 1 > AZ_MAX_LEVELS - 2) return SetError(AZ_ERR_UNSUPPORTED, "MaxRecursionDepth above 61");
    AZ_CUDA_TRY(cudaSetDevice(device));
    cudaStream_t st = opts && opts->stream ? (cudaStream_t)opts->stream : cudaStreamPerThread;
    void *base = nullptr;
    int rc = StaticWaveScratch(device, &base);
    if (rc != AZ_OK) return rc;
    CameraParams cam;
    rc = SetupCamera(camera, scissor, filter_type, backface_culling, epsilons, opts ? opts->seed : 0, cam);
    if (rc != AZ_OK) return rc;
    if ((rc = ChooseVariants(G, opts, cam)) != AZ_OK) return rc;
    // flags whose work would need buffers of their own or a statistics output
    const uint32_t flags = opts ? opts->flags : 0u;
    const uint32_t refused = AZ_FLAG_COUNT_TRAVERSAL | AZ_FLAG_TIME_STAGES | AZ_FLAG_ORDER_SHADOW | AZ_FLAG_ORDER_EXTEND;
    if (flags & refused)
        return SetError(AZ_ERR_INVALID_ARGUMENT,
                        "az_gpu_render_noalloc does not take AZ_FLAG_COUNT_TRAVERSAL, AZ_FLAG_TIME_STAGES, "
                        "AZ_FLAG_ORDER_SHADOW or AZ_FLAG_ORDER_EXTEND");
    cam.env_importance = (flags & AZ_FLAG_ENV_IMPORTANCE) && G.dev.env_rows ? 1u : 0u;
    cam.watertight = (flags & AZ_FLAG_WATERTIGHT) ? 1u : 0u;
    const uint64_t total = cam.npix * (uint64_t)cam.sqrt_spp * cam.sqrt_spp;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const WaveQueues Q = CarveStaticQueues((unsigned char *)base);
    const uint32_t levels = std::min<uint32_t>(G.dev.max_depth + 1, AZ_MAX_LEVELS - 2);
    const int grid = sms * 16;
    uint32_t host_counts[AZ_COUNT_TOTAL];
    uint64_t pos = 0;
    while (pos < total) {
        const uint32_t n = (uint32_t)std::min<uint64_t>(wave, total - pos);
        // the array keeps the previous call's contents: the counters start at
        // zero, every other entry is written before it is read
        AZ_CUDA_TRY(cudaMemsetAsync(Q.counts, 0, AZ_COUNT_TOTAL * sizeof(uint32_t), st));
        AZ_CUDA_TRY(cudaMemcpyAsync(Q.counts + 1, &n, sizeof(uint32_t), cudaMemcpyHostToDevice, st));
        k_camera<<<(n + 255) / 256, 256, 0, st>>>(cam, Q, pos, n);
        for (uint32_t L = 1; L <= levels; L++) {
            LaunchTraversalVariant(cam.variant, false, sms, G.dev, cam, Q, L, st);
            LaunchShade(grid, G.dev, cam, Q, pos, L, st);
            LaunchTraversalVariant(cam.shadow_variant, true, sms, G.dev, cam, Q, L, st);
        }
        k_splat<<<(n + 255) / 256, 256, 0, st>>>(cam, Q, pos, n, film);
        AZ_CUDA_TRY(cudaGetLastError());
        AZ_CUDA_TRY(cudaMemcpyAsync(host_counts, Q.counts, sizeof(host_counts), cudaMemcpyDeviceToHost, st));
        AZ_CUDA_TRY(cudaStreamSynchronize(st));
        if (host_counts[AZ_COUNT_ERROR])
            return SetError(AZ_ERR_CUDA, "BVH traversal exceeded its step limit (corrupt hierarchy)");
        if (host_counts[AZ_COUNT_OVERFLOW]) {
            // the wave wrote nothing to the film; rerun it with half the samples
            if (n <= 256) return SetError(AZ_ERR_OUT_OF_MEMORY, "static wave queues overflow with 256 samples");
            wave = n / 2;
            continue;
        }
        pos += n;
    }
    return AZ_OK;
}
