// Wavefront path-trace kernels for sm_100a.
//
// One render batch holds P window pixels x S samples = N paths whose state
// lives in HBM as structure-of-arrays (PathBuffers).  Per path step:
//   k_intersect  closest hit of every queued path (two-level BVH)
//   k_closest_exact  the few closest hits that depend on the order of visits
//   k_sort_*     long queues grouped by material and lamp kind, misses first
//   k_shade_miss the sorted queue's misses: lamps, background
//   k_light_pick light tree: the paths' picks and forward pdfs
//   k_shade      emission + forward MIS / roulette / AOV / NEE sample + BSDF
//                evaluation (writes one shadow ray) / closure sample +
//                path-state transition; survivors are compacted into the
//                next queue with warp-aggregated atomics
//   k_shadow     transmittance of the queued shadow rays, adds NEE radiance
// k_tail takes a queue that has become short through its remaining steps,
// and after the last step k_film adds each path's sample into the film in
// sample order.  The kernels reproduce the Psycles Luisa megakernel
// (src/luisa/path_kernel_pipeline.cpp:73-183) path by path: the queue order
// never changes a path's result.
#include "psy_device.cuh"
#include "psy_kernels.h"

#include <algorithm>
#include "psy_light_tree.cuh"

namespace psy {

// Warp-aggregated queue append: one atomic per warp, slots in lane order.
// Every lane of the warp must call it (the callers' loops are warp-uniform).
__device__ __forceinline__ uint32_t warp_push(uint32_t *counter, bool pred) {
    const unsigned ballot = __ballot_sync(0xffffffffu, pred);
    const int lane = threadIdx.x & 31;
    uint32_t base = 0u;
    if (lane == 0 && ballot != 0u) base = atomicAdd(counter, uint32_t(__popc(ballot)));
    base = __shfl_sync(0xffffffffu, base, 0);
    return base + uint32_t(__popc(ballot & ((1u << lane) - 1u)));
}

__device__ __forceinline__ Xform xform12(const float *m) { return {ld3(m), ld3(m + 3), ld3(m + 6), ld3(m + 9)}; }

__device__ __forceinline__ void add3(float *d, f3 v) {
    d[0] += v.x;
    d[1] += v.y;
    d[2] += v.z;
}
__device__ __forceinline__ void set3(float *d, f3 v) {
    d[0] = v.x;
    d[1] = v.y;
    d[2] = v.z;
}

// ------------------------------------------------------------------ raygen
// begin_path_sample / construct_camera_ray (src/luisa/path_kernel_setup.cpp:485-700,
// src/luisa/path_tracer_camera.cpp:10-246).
// sample_regular_polygon / sample_aperture (include/psycles/luisa/camera_sampling.h:
// 118-152): a corner triangle of the blade polygon, sampled by area.
__device__ __forceinline__ f2 sample_aperture(f2 r, uint32_t blades, float rotation) {
    if (blades == 0u) return sample_uniform_disk(r);
    const float corners = static_cast<float>(blades);
    float u = r.x, v = r.y;
    const float corner = floorf(u * corners);
    u = u * corners - corner;
    u = sqrtf(u);
    v *= u;
    u = 1.0f - u;
    const float half_corner = kPi / corners;
    const f2 point = mk2((u + v) * cos_(half_corner), (u - v) * sin_(half_corner));
    const float angle = rotation + corner * (2.0f * half_corner);
    const float c = cos_(angle), s = sin_(angle);
    return mk2(c * point.x - s * point.y, s * point.x + c * point.y);
}

// construct_camera_ray (src/luisa/path_tracer_camera.cpp:51-246): the camera-space
// ray of the projection (screen coordinates sx, sy in [-1, 1] plus lens
// shift), then the thin-lens update for depth of field.  `clip_cos` is the
// pinhole direction's cosine that scales the clipping range.
__device__ __forceinline__ void camera_local_ray(const RenderParams &p, float sx, float sy, f2 lens_sample, f3 &origin,
                                                 f3 &direction, float &clip_cos) {
    origin = mk3(0.0f);
    direction = mk3(0.0f, 0.0f, -1.0f);
    clip_cos = 1.0f;
    if (p.projection == PSY_CAMERA_PERSPECTIVE) {
        direction = normalize(mk3(sx * p.htan, sy * p.vtan, -1.0f));
        clip_cos = -direction.z;
    } else if (p.projection == PSY_CAMERA_ORTHOGRAPHIC) {
        const float aspect = static_cast<float>(p.full_w) / static_cast<float>(p.full_h);
        origin = mk3(sx * p.ortho_span * aspect * 0.5f, sy * p.ortho_span * 0.5f, 0.0f);
    } else {
        const float longitude = sx * kPi;
        const float latitude = sy * kPi * 0.5f;
        const float cos_lat = cos_(latitude);
        direction = mk3(cos_lat * sin_(longitude), sin_(latitude), -cos_lat * cos_(longitude));
    }
    if (p.depth_of_field) {
        f2 lens = sample_aperture(lens_sample, p.aperture_blades, p.aperture_rotation) * p.aperture_radius;
        lens.x /= maxf_(p.aperture_ratio, 1.0e-5f);
        const float focus_scale = p.focal_distance / maxf_(-direction.z, 1.0e-6f);
        const f3 focus = direction * focus_scale;
        origin = mk3(lens.x, lens.y, 0.0f);
        direction = normalize(focus - origin);
    }
}

__device__ __forceinline__ void raygen_path(const RenderParams &p, const PathBuffers &b, uint32_t i, uint32_t local,
                                            uint32_t sample, uint32_t trace_path, psy_path_trace *trace) {
    const uint32_t x = p.win_x + local % p.win_w;
    const uint32_t y = p.win_y + local / p.win_w;
    const uint32_t cycles_y = p.full_h - 1u - y;
    const uint32_t rng_hash = pixel_hash(x, cycles_y, p.seed);
    const float4 fs = sample_4d(p, sample, rng_hash, 0u);
    const f2 filter = sample == 0u ? mk2(0.5f, 0.5f) : mk2(fs.x, fs.y);
    const float jx = pixel_filter_sample(p.filter, filter.x);
    const float jy = 1.0f - pixel_filter_sample(p.filter, filter.y);
    const float W = static_cast<float>(p.full_w), H = static_cast<float>(p.full_h);
    const float sx = 2.0f * (static_cast<float>(x) + jx) / W - 1.0f + 2.0f * p.shift_x;
    const float sy = 1.0f - 2.0f * (static_cast<float>(y) + jy) / H + 2.0f * p.shift_y;
    f3 local_origin, local_dir;
    float clip_cos;
    f2 lens_sample = mk2(0.0f, 0.0f);
    if (p.depth_of_field) {
        // sample_3d at camera_lens_time_dimension, lens = .yz (path_tracer_camera.cpp:35-45)
        const float4 lt = sample_4d(p, sample, rng_hash, 1u);
        lens_sample = mk2(lt.y, lt.z);
    }
    camera_local_ray(p, sx, sy, lens_sample, local_origin, local_dir, clip_cos);
    const Xform cam = xform12(p.cam);
    f3 origin = xform_point(cam, local_origin);
    const f3 dir = safe_normalize(xform_direction(cam, local_dir), mk3(0.0f, 0.0f, -1.0f));
    const float safe_cos = maxf_(fabsf(clip_cos), 1.0e-20f);
    const float near_t = p.near_clip / safe_cos;
    const float far_t = (p.far_clip - p.near_clip) / safe_cos;
    origin = origin + dir * near_t;
    store_pair(b.ray_o, i, make_float4(origin.x, origin.y, origin.z, 0.0f), make_float4(dir.x, dir.y, dir.z, far_t));
    store_pair(b.tp, i, make_float4(1.0f, 1.0f, 1.0f, 0.0f), make_float4(0.0f, 0.0f, 0.0f, 0.0f));
    // initial_state (include/psycles/luisa/cycles_path_state.h:187-199)
    store_pair(b.st, i, make_uint4(128u | 512u, 1u, 16u, 0u), make_uint4(kSt2Delta, kInvalid, kInvalid, local));
    b.sample[i] = sample;
    b.aov_n[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    b.aov_a[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    b.mis_n[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    b.queue_in[i] = i;
    if (i == trace_path && trace) {
        trace->pixel_x = x;
        trace->pixel_y = y;
        trace->sample = sample;
        trace->rng_hash = rng_hash;
        trace->filter[0] = filter.x;
        trace->filter[1] = filter.y;
        set3(trace->ray_origin, origin);
        set3(trace->ray_direction, dir);
        trace->valid = 1u;
        trace->event_count = 0u;
    }
}

__global__ void k_raygen(RenderParams p, PathBuffers b, uint32_t pixels, uint32_t paths, uint32_t sample_base,
                         uint32_t trace_path, psy_path_trace *trace) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < paths; i += gridDim.x * blockDim.x)
        raygen_path(p, b, i, i % pixels, sample_base + i / pixels, trace_path, trace);
}

// The item of a batched wavefront that holds `index` (items sorted by the
// field `begin` selects).
template <typename Begin>
__device__ __forceinline__ uint32_t find_item(const BatchItem *items, uint32_t n, uint32_t index, Begin begin) {
    uint32_t lo = 0u, hi = n;
    while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (begin(items[mid]) <= index) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Camera rays of every item of a batched wavefront; records each path's job.
// The wavefront's shape comes from device memory (round[0] paths, round[2]
// items) so one captured launch serves every wavefront.
__global__ void k_raygen_batch(const JobGpu *jobs, const BatchItem *items, const uint32_t *round, PathBuffers b) {
    const uint32_t paths = round[0], item_count = round[2];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < paths; i += gridDim.x * blockDim.x) {
        const BatchItem it = items[find_item(items, item_count, i, [](const BatchItem &t) { return t.path_begin; })];
        const uint32_t r = i - it.path_begin;
        b.job[i] = it.job;
        raygen_path(jobs[it.job].p, b, i, r % it.pixels, it.sample_base + r / it.pixels, kInvalid, nullptr);
    }
}

// --------------------------------------------------------------- intersect
// Cycles ray visibility of a path: contract_visibility (cycles_path_state.h:449-491).
__device__ __forceinline__ uint32_t contract_visibility(uint32_t v) {
    const uint32_t tv = (v & 2u) ? (v & ~(4u | 8u)) : v;
    uint32_t r = 0u;
    if (tv & 1u) r |= PSY_VISIBILITY_CAMERA;
    if (tv & 2u) r |= PSY_VISIBILITY_TRANSMISSION;
    if (tv & 4u) r |= PSY_VISIBILITY_DIFFUSE;
    if (tv & 8u) r |= PSY_VISIBILITY_GLOSSY;
    if (tv & 16u) r |= PSY_VISIBILITY_VOLUME_SCATTER;
    return r;
}

// Persistent closest-hit kernel: each lane owns one ray at a time and, when
// some have finished, the warp refills its idle lanes from a global fetch
// counter (one atomic per warp), so lanes do not wait for the warp's longest
// ray.  Refilling at 12 idle lanes measured best of 4, 8, 12 and 16.
//
// Both traversal kernels were bound by L1 wavefronts (72 % of peak for closest
// hits: a 128-byte node in eight 16-byte loads, each a wavefront per lane)
// and by divergence (9 and 7 of 32 lanes).  With 64-byte nodes in two loads
// and steps taken together (traverse_warp) they are issue-bound, and the lower
// register budgets give the latency more warps to hide in.  1080p procedural
// frame, 64 spp: closest hits 224 -> 152 ms at 7 blocks of 128 an SM (8, where
// closest_ambiguous spills: 157), shadow rays 185 -> 81 ms at 8.
#ifndef PSY_REFILL_LANES
#define PSY_REFILL_LANES 12
#endif
#ifndef PSY_INTERSECT_MIN_BLOCKS
#define PSY_INTERSECT_MIN_BLOCKS 7
#endif
#ifndef PSY_SHADE_MIN_BLOCKS
#define PSY_SHADE_MIN_BLOCKS 4
#endif
#ifndef PSY_TAIL_MIN_BLOCKS
#define PSY_TAIL_MIN_BLOCKS 3
#endif
#ifndef PSY_PICK_MIN_BLOCKS
#define PSY_PICK_MIN_BLOCKS 8
#endif
#ifndef PSY_MISS_MIN_BLOCKS
#define PSY_MISS_MIN_BLOCKS 8
#endif
#ifndef PSY_SHADOW_MIN_BLOCKS
#define PSY_SHADOW_MIN_BLOCKS 8
#endif
// Lanes that finish before a warp is refilled.
constexpr int kRefillLanes = PSY_REFILL_LANES;
constexpr uint32_t kFullMask = 0xffffffffu;

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31u; }

// Hands the next queue slot below `count` to every lane with `need`, or
// kInvalid.  Warp-uniform: every lane calls it, and `exhausted` (uniform
// across the warp) stops further atomics once the queue is used up.
__device__ __forceinline__ uint32_t warp_fetch(uint32_t *fetch_counter, uint32_t count, bool need, bool &exhausted) {
    if (exhausted) return kInvalid;
    const unsigned mask = __ballot_sync(kFullMask, need);
    if (mask == 0u) return kInvalid;
    uint32_t base = 0u;
    if (lane_id() == 0u) base = atomicAdd(fetch_counter, uint32_t(__popc(mask)));
    base = __shfl_sync(kFullMask, base, 0);
    if (base + uint32_t(__popc(mask)) >= count) exhausted = true;
    if (!need) return kInvalid;
    const uint32_t q = base + uint32_t(__popc(mask & ((1u << lane_id()) - 1u)));
    return q < count ? q : kInvalid;
}

// A path's closest hit so far.
struct ClosestHit {
    float t, u, v;
    uint32_t instance;  // kInvalid: none yet
    uint32_t slot;      // its triangle's place in SceneView::tris
};

__device__ __forceinline__ void closest_begin(ClosestHit &best, TraversalState &t, const SceneView &s,
                                              const PathBuffers &b, uint32_t path) {
    float4 o, d;
    uint4 st, st2;
    load_pair(b.ray_o, path, o, d);
    load_pair(b.st, path, st, st2);
    const Ray ray{mk3(o.x, o.y, o.z), mk3(d.x, d.y, d.z), o.w, d.w};
    traversal_begin(t, s, ray, contract_visibility(st.y), st2.y, st2.z, kInvalid, kInvalid);
    best.t = ray.tmax;
    best.u = best.v = 0.0f;
    best.instance = best.slot = kInvalid;
}

// Equal distances go to the greatest (object, primitive).  t.stack[kStackVisitor]
// is the distance of the next hit behind the closest; to see one that lies within
// rounding, hits a little behind it are looked at too.
__device__ __forceinline__ bool closest_hit(ClosestHit &best, TraversalState &t, const SceneView &s, uint32_t instance,
                                            uint32_t prim, uint32_t slot, float th, float u, float v) {
    if (best.instance != kInvalid && !(th < best.t)) {
        const bool wins = th == best.t && (instance > best.instance ||
                                           (instance == best.instance &&
                                            prim > __float_as_uint(__ldg(&s.tris[best.slot].v0.w))));
        if (!wins) {
            t.stack[kStackVisitor] = __float_as_uint(fminf(__uint_as_float(t.stack[kStackVisitor]), th));
            return false;
        }
    }
    t.stack[kStackVisitor] = __float_as_uint(best.t);
    best = {th, u, v, instance, slot};
    t.tmax = fmaf(th, 1.00000095367431640625f, 1.0e-30f);
    return false;
}

// Whether the closest hit of a finished ray depends on the order of visits, or is
// none.  A subtree is culled if the ray enters its box behind the closest hit so
// far; where rounding puts a triangle's hit before its box, that can happen to
// the closest one if another hit lies between the two.  `prim`: its primitive.
__device__ __forceinline__ bool closest_ambiguous(const ClosestHit &best, const TraversalState &t, const SceneView &s,
                                                  uint32_t &prim) {
    prim = kInvalid;
    if (best.instance == kInvalid) return false;
    uint4 w0, w1, ua, ub, uc, ud;
    const EntryGpu *ep = s.entries + best.instance;
    load_sector_nc(ep, w0, w1);
    const uint4 w2 = __ldg(reinterpret_cast<const uint4 *>(ep->w2o + 8));
    const TriGpu *tp = s.tris + best.slot;
    load_sector_nc(tp, ua, ub);
    load_sector_nc(&tp->v2, uc, ud);
    prim = ua.w;
    const float4 e = floats4(ud);
    float near;
    if (!box_admits(entry_slabs(w0, w1, w2, t.ray), mk3(__uint_as_float(ub.w), __uint_as_float(uc.w), e.x),
                    mk3(e.y, e.z, e.w), t.ray.tmin, kInf, near))
        return true;
    float entry;
    if (!instance_admits(s, best.instance, make_slab_ray(t.ray.o, t.ray.d), t.ray.tmin, kInf, entry)) return true;
    near = fmaxf(near, entry);
    return __uint_as_float(t.stack[kStackVisitor]) < near || t.tmax < near;
}

// The closest hit of an ambiguous ray, for which the order of visits counts:
// nodes nearest first by their float boxes, a node's triangles before its
// other children, these only if the ray enters them before the closest hit so
// far.  This order, which defines the renderer's results, is the one of
// traversing float boxes throughout; the byte boxes give the same hit for all
// other rays.  (Restated on the CPU, 220 M rays aimed at shared edges from up to
// 1e4 mesh sizes away: at most 1 % ambiguous, one other hit; ordinary
// rays are ambiguous about once in 1e7.)
__device__ __noinline__ ClosestHit closest_exact(const NodeGpu *nodes, const BoxGpu *node_boxes, const TriGpu *tris,
                                                 const EntryGpu *entries, const BoxGpu *instance_boxes, Ray ray,
                                                 uint32_t visibility, uint32_t src_obj, uint32_t src_prim) {
    uint32_t stack[kStackSize];
    uint32_t sp = 0u, node = 0u, instance = kInvalid, prim_offset = 0u;
    SlabRay cur = make_slab_ray(ray.o, ray.d);
    float tmax = ray.tmax;
    stack_push(stack, sp, kLinkDone);
    ClosestHit best{ray.tmax, 0.0f, 0.0f, kInvalid, kInvalid};
    uint32_t best_prim = kInvalid;
    while (node != kLinkDone) {
        if (node == kLinkLeave) {
            cur = make_slab_ray(ray.o, ray.d);
            instance = kInvalid;
            node = stack[--sp];
            continue;
        }
        if (node >= kLinkInstance) {
            const EntryGpu &e = entries[node & ~kLinkInstance];
            if ((e.visibility & visibility) == 0u) {
                node = stack[--sp];
                continue;
            }
            const Xform w2o = xform12(e.w2o);
            cur = make_slab_ray(xform_point(w2o, ray.o), xform_direction(w2o, ray.d));
            instance = node & ~kLinkInstance;
            prim_offset = e.prim_offset;
            stack_push(stack, sp, kLinkLeave);
            node = e.root;
            continue;
        }
        float key[4] = {kInf, kInf, kInf, kInf};
        uint32_t val[4], leaves = 0u;
        const uint32_t *link = nodes[node].link;
        for (uint32_t k = 0; k < 4u; ++k) {
            const uint32_t v = link[k];
            float near;
            if (v == kInvalid) continue;
            if ((v & kLinkLeaf) != 0u) {
                const TriGpu &tri = tris[v & ~kLinkLeaf];
                const float4 e = tri.lo_z_hi;
                if (box_admits(cur, mk3(tri.v1.w, tri.v2.w, e.x), mk3(e.y, e.z, e.w), ray.tmin, tmax, near))
                    leaves |= 1u << k;
                continue;
            }
            const bool inner = v < kLinkInstance;
            const float *box = inner ? node_boxes[v].lo : instance_boxes[v & ~kLinkInstance].lo;
            const uint32_t slot = inner ? node_boxes[v].slot : k;
            val[slot] = v;
            if (box_admits(cur, ld3(box), ld3(box + 3), ray.tmin, tmax, near)) key[slot] = near;
        }
        for (uint32_t k = 0; k < 4u; ++k) {
            if ((leaves >> k & 1u) == 0u) continue;
            const TriGpu &tri = tris[link[k] & ~kLinkLeaf];
            const uint32_t prim = __float_as_uint(tri.v0.w);
            if (src_obj == instance && src_prim == prim_offset + prim) continue;
            float th, u, v;
            if (!intersect_triangle(cur.o, cur.d, ray.tmin, tmax, ld3(tri.v0), ld3(tri.v1), ld3(tri.v2), th, u, v))
                continue;
            const bool later = instance > best.instance || (instance == best.instance && prim > best_prim);
            if (best.instance != kInvalid && !(th < best.t || (th == best.t && later))) continue;
            best = {th, u, v, instance, link[k] & ~kLinkLeaf};
            best_prim = prim;
            tmax = th;
        }
        for (uint32_t k = 0; k < 4u; ++k)
            if (!(key[k] <= tmax)) key[k] = kInf;
        sort_children(key, val);
        for (uint32_t k = 3u; k >= 1u; --k)
            if (key[k] != kInf) stack_push(stack, sp, val[k]);
        node = key[0] != kInf ? val[0] : stack[--sp];
    }
    return best;
}

// The ray of a path as its record holds it, traced so.
__device__ __forceinline__ ClosestHit closest_exact(const SceneView &s, const PathBuffers &b, uint32_t path) {
    float4 o, d;
    uint4 st, st2;
    load_pair(b.ray_o, path, o, d);
    load_pair(b.st, path, st, st2);
    return closest_exact(s.nodes, s.node_boxes, s.tris, s.entries, s.instance_boxes, {mk3(o.x, o.y, o.z), mk3(d.x, d.y, d.z), o.w, d.w},
                         contract_visibility(st.y), st2.y, st2.z);
}

__device__ __forceinline__ uint32_t closest_prim(const ClosestHit &best, const SceneView &s) {
    return best.instance == kInvalid ? kInvalid : __float_as_uint(__ldg(&s.tris[best.slot].v0.w));
}

__device__ __forceinline__ void closest_store(const ClosestHit &best, uint32_t prim, const PathBuffers &b,
                                              uint32_t path) {
    store_pair(b.hit, path, make_float4(best.t, best.u, best.v, __uint_as_float(best.instance)),
               make_uint4(prim, 0u, 0u, 0u));
}

// kMulti: paths of a batched wavefront, each traced in its job's scene.
template <bool kMulti>
__global__ void __launch_bounds__(128, PSY_INTERSECT_MIN_BLOCKS)
    k_intersect(const __grid_constant__ SceneView s_arg, const __grid_constant__ PathBuffers b, const JobGpu *jobs,
                uint32_t sort_threshold) {
    const uint32_t count = b.counters[0];
    if (b.counters[kCounterTail] != 0u) return;
    const bool sorted = sort_threshold != 0u && count >= sort_threshold;
    TraversalState t;
    t.node = kLinkDone;
    t.leaves = 0u;
    ClosestHit best;
    bool active = false, exhausted = false;
    uint32_t path = 0u, job = 0u;
    for (;;) {
        const uint32_t q = warp_fetch(&b.counters[3], count, !active, exhausted);
        if (q != kInvalid) {
            path = sorted ? b.queue_sorted[q] : b.queue_in[q];
            if (kMulti) job = b.job[path];
        }
        const SceneView &s = kMulti ? jobs[job].s : s_arg;
        if (q != kInvalid) {
            closest_begin(best, t, s, b, path);
            active = true;
        }
        const int busy = __popc(__ballot_sync(kFullMask, active));
        if (busy == 0) break;
        traverse_warp<true>(t, s, exhausted ? 32 : min(32, 32 - busy + kRefillLanes),
                            [&](uint32_t ii, uint32_t local, uint32_t, uint32_t slot, float th, float u, float v) {
            return closest_hit(best, t, s, ii, local, slot, th, u, v);
        });
        if (active && t.node == kLinkDone && t.leaves == 0u) {
            uint32_t prim;
            if (closest_ambiguous(best, t, s, prim)) b.ambiguous[atomicAdd(&b.counters[kCounterAmbiguous], 1u)] = path;
            closest_store(best, prim, b, path);
            active = false;
        }
    }
}

// The closest hits of the paths k_intersect has found ambiguous, mostly none.
// Called from k_intersect itself, closest_exact cost that kernel registers
// (1080p procedural frame, 64 spp: 291 -> 308 ms).
template <bool kMulti>
__global__ void __launch_bounds__(128)
    k_closest_exact(const __grid_constant__ SceneView s_arg, const __grid_constant__ PathBuffers b, const JobGpu *jobs) {
    const uint32_t count = b.counters[kCounterAmbiguous];
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x) {
        const uint32_t path = b.ambiguous[q];
        const SceneView &s = kMulti ? jobs[b.job[path]].s : s_arg;
        const ClosestHit best = closest_exact(s, b, path);
        closest_store(best, closest_prim(best, s), b, path);
    }
}

// ------------------------------------------------------------------- shade

__device__ __forceinline__ float power_heuristic(float a, float c) {
    const float a2 = a * a, c2 = c * c;
    return a2 / maxf_(a2 + c2, 1.0e-20f);
}

// forward_light_weight / nee_light_weight (src/luisa/path_tracer_lighting.cpp:35-72)
// for the effective direct-light mode.
__device__ __forceinline__ float forward_light_weight(uint32_t mode, float forward_pdf, float nee_pdf, bool competing,
                                                      bool nee_available) {
    if (mode == PSY_DIRECT_LIGHT_FORWARD) return 1.0f;
    if (mode == PSY_DIRECT_LIGHT_NEE) return (competing && nee_available) ? 0.0f : 1.0f;
    return (competing && nee_available) ? power_heuristic(forward_pdf, nee_pdf) : 1.0f;
}
__device__ __forceinline__ float nee_light_weight(uint32_t mode, float nee_pdf, float forward_pdf) {
    if (mode == PSY_DIRECT_LIGHT_NEE) return 1.0f;
    if (mode == PSY_DIRECT_LIGHT_FORWARD) return forward_pdf <= 0.0f ? 1.0f : 0.0f;
    return power_heuristic(nee_pdf, forward_pdf);
}

// film_clamp_light (include/psycles/luisa/cycles_film_light.h:15-49).
__device__ __forceinline__ f3 clamp_contribution(f3 c, uint32_t depth, const RenderParams &p) {
    c = mk3(isfinite(c.x) ? c.x : 0.0f, isfinite(c.y) ? c.y : 0.0f, isfinite(c.z) ? c.z : 0.0f);
    const float limit = depth > 0u ? p.clamp_indirect : p.clamp_direct;
    const float mag = fabsf(c.x) + fabsf(c.y) + fabsf(c.z);
    if (limit > 0.0f && mag > limit) return c * (limit / maxf_(mag, 1.0e-20f));
    return c;
}

__device__ __forceinline__ float light_roulette_weight(f3 unshadowed, float random, float inv_threshold) {
    const float m = max_abs_component(unshadowed);
    const float pr = m * inv_threshold;
    const bool roulette = inv_threshold > 0.0f && pr < 1.0f;
    const bool survives = !roulette || random < pr;
    const float inv_p = roulette ? 1.0f / maxf_(pr, 1.0e-20f) : 1.0f;
    return survives ? inv_p : 0.0f;
}

constexpr uint32_t kFlagReflect = 1u, kFlagSingular = 2u, kFlagTransparent = 4u, kFlagImportanceBake = 8u,
                   kFlagDiffuseAncestor = 16u, kFlagMisHadTransmission = 64u, kFlagMisSkip = 128u,
                   kFlagSinglePassDone = 256u, kFlagTransparentBackground = 512u,
                   kFlagTerminateOnNextSurface = 1024u, kFlagTerminateAfterTransparent = 4096u,
                   kFlagSurfacePass = 1u << 18u, kFlagVolumePass = 1u << 19u;

struct PathState {
    uint32_t flag, visibility, bounce, diffuse_bounce, glossy_bounce, transmission_bounce, transparent_bounce,
        rng_offset;
};

// cycles_path_state::next_surface (include/psycles/luisa/cycles_path_state.h:205-338).
__device__ __forceinline__ PathState next_surface(const PathState &before, uint32_t label, uint32_t runtime,
                                                  const RenderParams &p) {
    if ((label & (kLabelTransparent | 512u)) != 0u) {
        PathState t = before;
        t.transparent_bounce += 1u;
        t.rng_offset += 16u;
        t.flag |= kFlagTransparent;
        if (t.transparent_bounce >= p.transparent_max) t.flag |= kFlagTerminateOnNextSurface;
        if ((runtime & 4096u) != 0u) t.flag |= kFlagMisSkip;
        return t;
    }
    PathState s = before;
    s.bounce += 1u;
    s.rng_offset += 16u;
    if (s.bounce >= p.maximum) s.flag |= kFlagTerminateAfterTransparent;
    s.visibility = 0u;
    s.flag &= ~(kFlagReflect | kFlagSingular | kFlagTransparent | kFlagImportanceBake | kFlagMisSkip |
                kFlagMisHadTransmission);
    const bool reflection = (label & kLabelReflect) != 0u;
    const bool diffuse = (label & kLabelDiffuse) != 0u;
    const bool glossy = (label & kLabelGlossy) != 0u;
    const bool transmit_transparent = (label & 128u) != 0u;
    if (reflection) s.flag |= kFlagReflect;
    if (reflection || !transmit_transparent) s.flag &= ~kFlagTransparentBackground;
    const bool diffuse_reflection = reflection && diffuse;
    const bool glossy_reflection = reflection && !diffuse;
    const bool transmission = !reflection;
    if (diffuse_reflection) s.diffuse_bounce += 1u;
    if (glossy_reflection) s.glossy_bounce += 1u;
    if (transmission) s.transmission_bounce += 1u;
    if (diffuse_reflection && s.diffuse_bounce >= p.max_diffuse) s.flag |= kFlagTerminateAfterTransparent;
    if (glossy_reflection && s.glossy_bounce >= p.max_glossy) s.flag |= kFlagTerminateAfterTransparent;
    if (transmission && s.transmission_bounce >= p.max_transmission) s.flag |= kFlagTerminateAfterTransparent;
    if (transmission) s.visibility |= 2u;
    s.visibility |= diffuse ? 4u : 8u;
    if (diffuse) s.flag |= kFlagDiffuseAncestor;
    if (!diffuse && !glossy) s.flag |= kFlagSingular | kFlagMisSkip;
    if ((runtime & kRuntimeBsdfHasTransmission) != 0u) s.flag |= kFlagMisHadTransmission;
    if ((s.flag & (kFlagSurfacePass | kFlagVolumePass)) == 0u && (s.flag & kFlagTransparentBackground) == 0u)
        s.flag |= kFlagSurfacePass;
    return s;
}

__device__ __forceinline__ PathState unpack_state(uint4 st, uint4 st2) {
    return {st.x, st.y, st.w & 0xffu, (st.w >> 8) & 0xffu, (st.w >> 16) & 0xffu, st.w >> 24, st2.x & 0xffu, st.z};
}

__device__ __forceinline__ float next_float_up(float t) {
    return t == 0.0f ? 1.17549435e-38f : __uint_as_float(__float_as_uint(t) + 1u);
}

// ------------------------------------------------------ sort by material
__device__ __forceinline__ uint32_t surface_material(const SceneView &s, uint32_t instance, uint32_t cycles_prim);

// The kind of lamp a path's next-event sample will take under the flat
// light distribution, estimated from the same random number the shading
// kernel draws (the lamps share the distribution's tail equally): 1
// emissive triangle, 2 sun, 3 / 4 rectangle / ellipse, 5 delta point or
// spot, 6 disk, 7 sphere; 0 without a flat-distribution pick.  Only the
// queue order depends on it, so an estimate at a bin edge costs
// coherence, never a result.
__device__ __forceinline__ uint32_t nee_kind_hint(const SceneView &s, const RenderParams &p, const PathBuffers &b,
                                                  uint32_t i) {
    if (p.use_light_tree || !p.nee || s.emitter_count == 0u) return 0u;
    uint4 st, st2;
    load_pair(b.st, i, st, st2);
    const uint32_t local = st2.w;
    const uint32_t x = p.win_x + local % p.win_w, y = p.win_y + local / p.win_w;
    const uint32_t rng_hash = pixel_hash(x, p.full_h - 1u - y, p.seed);
    const float u = sample_4d(p, b.sample[i], rng_hash, st.z + 1u).z;
    const uint32_t tri_n = s.triangle_emitters, light_n = s.light_count;
    const float c0 = tri_n > 0u ? s.distribution[tri_n].cumulative : 0.0f;
    if (light_n == 0u || u < c0) return 1u;
    const uint32_t li = min(uint32_t((u - c0) / fmaxf(1.0f - c0, 1.0e-20f) * float(light_n)), light_n - 1u);
    const psy_light_desc &l = s.lights[li];
    if (l.type == PSY_LIGHT_DISTANT) return 2u;
    if (l.type == PSY_LIGHT_AREA) return (l.flags & PSY_LIGHT_FLAG_ELLIPSE) != 0u ? 4u : 3u;
    if (!(l.radius > 0.0f)) return 5u;
    return (l.flags & PSY_LIGHT_FLAG_SPHERE) != 0u ? 7u : 6u;
}

// Queues of at least `threshold` paths are grouped before shading by
// material and by the kind of lamp the path's next-event sample takes, so
// a warp mostly runs one closure program and one light-sampling branch: a
// bucket per queue entry (misses in bucket 0, hits by material, lamp kind
// and job hashed into the other buckets), a histogram, its exclusive scan
// and a scatter.  Order inside a bucket is arbitrary; no path's result
// depends on the queue order.
template <bool kMulti>
__global__ void k_sort_count(const __grid_constant__ SceneView s_arg, const __grid_constant__ RenderParams p_arg,
                             const __grid_constant__ PathBuffers b, const JobGpu *jobs, uint32_t threshold) {
    __shared__ uint32_t local[kSortBuckets];
    const uint32_t count = b.counters[0];
    if (count < threshold || b.counters[kCounterTail] != 0u) return;
    for (uint32_t k = threadIdx.x; k < kSortBuckets; k += blockDim.x) local[k] = 0u;
    __syncthreads();
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x) {
        const uint32_t i = b.queue_in[q];
        float4 h4;
        uint4 hp4;
        load_pair(b.hit, i, h4, hp4);
        const uint32_t prim = hp4.x;
        uint32_t key = 0u;
        if (prim != kInvalid) {
            const uint32_t job = kMulti ? b.job[i] : 0u;
            const SceneView &s = kMulti ? jobs[job].s : s_arg;
            const RenderParams &p = kMulti ? jobs[job].p : p_arg;
            const uint32_t instance = __float_as_uint(h4.w);
            const uint32_t mat =
                surface_material(s, instance, s.entries[instance].prim_offset + prim) & ~kMaterialTransparent;
            key = 1u + (mat * 8u + nee_kind_hint(s, p, b, i) + job * 977u) % (kSortBuckets - 1u);
        }
        b.sort_keys[q] = key;
        atomicAdd(&local[key], 1u);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < kSortBuckets; k += blockDim.x)
        if (local[k]) atomicAdd(&b.sort_hist[k], local[k]);
}

// One block of 1024 threads: offsets = exclusive scan of the histogram,
// which is cleared for the next sort.
// `counter`: 0 sorts the shading queue, 2 the shadow queue.  `misses`: the
// queue is the shading queue, whose bucket 0 holds the misses.
__global__ void k_sort_scan(const __grid_constant__ PathBuffers b, uint32_t threshold, uint32_t counter, bool misses) {
    __shared__ uint32_t part[1024];
    if (b.counters[counter] < threshold || b.counters[kCounterTail] != 0u) return;
    constexpr uint32_t kPer = kSortBuckets / 1024u;
    const uint32_t t = threadIdx.x;
    uint32_t v[kPer], sum = 0u;
    for (uint32_t k = 0; k < kPer; ++k) {
        v[k] = b.sort_hist[t * kPer + k];
        sum += v[k];
    }
    if (misses && t == 0u) b.counters[kCounterMisses] = v[0];
    part[t] = sum;
    __syncthreads();
    for (uint32_t d = 1u; d < 1024u; d <<= 1) {  // inclusive Hillis-Steele scan
        const uint32_t add = t >= d ? part[t - d] : 0u;
        __syncthreads();
        part[t] += add;
        __syncthreads();
    }
    uint32_t run = part[t] - sum;
    for (uint32_t k = 0; k < kPer; ++k) {
        b.sort_offsets[t * kPer + k] = run;
        run += v[k];
        b.sort_hist[t * kPer + k] = 0u;
    }
}

// Scatter in three passes over each block's contiguous chunk of the queue:
// ranks inside the block from warp-aggregated shared-memory atomics (stored
// beside the 11-bit bucket), one global reservation per non-empty bucket
// per block, then the writes.  Global atomics drop from one per path to one
// per bucket and block.
// The shading queue sorts its path indices; the shadow queue sorts its
// slot numbers (a permutation k_shadow reads its rays through).
__global__ void __launch_bounds__(256) k_sort_scatter(const __grid_constant__ PathBuffers b, uint32_t threshold,
                                                      uint32_t counter) {
    __shared__ uint32_t hist[kSortBuckets];
    const uint32_t count = b.counters[counter];
    if (count < threshold || b.counters[kCounterTail] != 0u) return;
    const uint32_t chunk = (count + gridDim.x - 1u) / gridDim.x;
    const uint32_t begin = blockIdx.x * chunk;
    const uint32_t end = min(count, begin + chunk);
    for (uint32_t k = threadIdx.x; k < kSortBuckets; k += blockDim.x) hist[k] = 0u;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t base = begin; base < end; base += blockDim.x) {
        const uint32_t q = base + threadIdx.x;
        const bool live = q < end;
        const uint32_t key = live ? b.sort_keys[q] : kSortBuckets;  // sentinel outside the histogram
        const uint32_t peers = __match_any_sync(kFullMask, key);
        const uint32_t leader = __ffs(peers) - 1u;
        const uint32_t rank_in_warp = __popc(peers & ((1u << lane) - 1u));
        uint32_t first = 0u;
        if (live && lane == leader) first = atomicAdd(&hist[key], __popc(peers));
        first = __shfl_sync(peers, first, leader);
        if (live) b.sort_keys[q] = key | ((first + rank_in_warp) << 11);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < kSortBuckets; k += blockDim.x)
        if (hist[k]) hist[k] = atomicAdd(&b.sort_offsets[k], hist[k]);
    __syncthreads();
    for (uint32_t q = begin + threadIdx.x; q < end; q += blockDim.x) {
        const uint32_t packed = b.sort_keys[q];
        b.queue_sorted[hist[packed & (kSortBuckets - 1u)] + (packed >> 11)] = counter == 0u ? b.queue_in[q] : q;
    }
}

// Closest-hit rays grouped by where they start and where they head: the
// direction octant and an 8 x 8 x 4 cell of the scene's bounds around the
// origin, so a warp's rays walk the same part of the BVH.  Rays of a
// batched wavefront are grouped per job as well.
template <bool kMulti>
__global__ void k_sort_count_rays(const __grid_constant__ SceneView s_arg, const __grid_constant__ PathBuffers b,
                                  const JobGpu *jobs, uint32_t threshold) {
    __shared__ uint32_t local[kSortBuckets];
    const uint32_t count = b.counters[0];
    if (count < threshold || b.counters[kCounterTail] != 0u) return;
    for (uint32_t k = threadIdx.x; k < kSortBuckets; k += blockDim.x) local[k] = 0u;
    __syncthreads();
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x) {
        const uint32_t i = b.queue_in[q];
        const uint32_t job = kMulti ? b.job[i] : 0u;
        const SceneView &s = kMulti ? jobs[job].s : s_arg;
        float4 o, d;
        load_pair(b.ray_o, i, o, d);
        auto cell = [](float v, float lo, float hi, float n) {
            const float f = hi > lo ? (v - lo) / (hi - lo) : 0.0f;
            return uint32_t(fminf(fmaxf(f * n, 0.0f), n - 1.0f));
        };
        const uint32_t cx = cell(o.x, s.world_lo.x, s.world_hi.x, 8.0f);
        const uint32_t cy = cell(o.y, s.world_lo.y, s.world_hi.y, 8.0f);
        const uint32_t cz = cell(o.z, s.world_lo.z, s.world_hi.z, 4.0f);
        const uint32_t octant = (d.x < 0.0f ? 1u : 0u) | (d.y < 0.0f ? 2u : 0u) | (d.z < 0.0f ? 4u : 0u);
        const uint32_t key = ((octant << 8 | cz << 6 | cy << 3 | cx) + job * 977u) & (kSortBuckets - 1u);
        b.sort_keys[q] = key;
        atomicAdd(&local[key], 1u);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < kSortBuckets; k += blockDim.x)
        if (local[k]) atomicAdd(&b.sort_hist[k], local[k]);
}

// Shadow rays grouped by direction (octahedral map of the direction into a
// 45 x 45 grid), so a warp's rays head the same way -- mostly towards the
// same light from nearby points.
__global__ void k_sort_count_shadow(const __grid_constant__ PathBuffers b, uint32_t threshold) {
    __shared__ uint32_t local[kSortBuckets];
    const uint32_t count = b.counters[2];
    if (count < threshold || b.counters[kCounterTail] != 0u) return;
    for (uint32_t k = threadIdx.x; k < kSortBuckets; k += blockDim.x) local[k] = 0u;
    __syncthreads();
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x) {
        const float4 d = b.sh_d[q];
        const float l1 = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
        float u = l1 > 0.0f ? d.x / l1 : 0.0f, v = l1 > 0.0f ? d.y / l1 : 0.0f;
        if (d.z < 0.0f) {
            const float uu = (1.0f - fabsf(v)) * (u >= 0.0f ? 1.0f : -1.0f);
            v = (1.0f - fabsf(u)) * (v >= 0.0f ? 1.0f : -1.0f);
            u = uu;
        }
        const uint32_t iu = min(44u, uint32_t(fmaxf(u * 0.5f + 0.5f, 0.0f) * 45.0f));
        const uint32_t iv = min(44u, uint32_t(fmaxf(v * 0.5f + 0.5f, 0.0f) * 45.0f));
        const uint32_t key = iv * 45u + iu;
        b.sort_keys[q] = key;
        atomicAdd(&local[key], 1u);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < kSortBuckets; k += blockDim.x)
        if (local[k]) atomicAdd(&b.sort_hist[k], local[k]);
}

// Lamps in front of the event at `event_distance` (the mesh hit or the ray's
// end) are transparent events that add their emission without a new bounce
// or new dimensions (src/luisa/path_kernel_pipeline.cpp:78-126,
// src/luisa/path_kernel_forward_light.cpp:14-118).  False once they used up
// the path's transparent budget.
__device__ __forceinline__ bool lamp_events(const SceneView &s, const RenderParams &p, const PathBuffers &b, uint32_t i,
                                            const Ray &ray, float event_distance, uint32_t ray_visibility,
                                            f3 throughput, float previous_bsdf_pdf, bool previous_delta, PathState &ps,
                                            f3 &radiance, psy_path_event *ev) {
    const uint32_t depth = ps.bounce;
    uint32_t excluded = kInvalid;
    float tmin = ray.tmin;
    for (uint32_t guard = 0; guard <= s.lamp_count; ++guard) {
        const float4 mn = b.mis_n[i];
        const LampHit lh = closest_lamp(s, ray.o, ray.d, tmin, event_distance, ray_visibility, excluded,
                                        mk3(mn.x, mn.y, mn.z), (ps.flag & kFlagMisHadTransmission) != 0u);
        if (!lh.valid) break;
        float selection_pdf = s.light_selection_pdf;
        if (p.use_light_tree)
            selection_pdf = lt_pdf(s, s.triangle_emitters + lh.index, ray.o, mk3(mn.x, mn.y, mn.z),
                                   (ps.flag & kFlagMisHadTransmission) != 0u);
        const float light_pdf = lh.pdf * selection_pdf;
        const bool competing = depth > 0u && !previous_delta;
        const float w = forward_light_weight(p.direct_mode, previous_bsdf_pdf, light_pdf, competing, light_pdf > 0.0f);
        const psy_light_desc &l = s.lights[lh.index];
        const f3 lr = ld3(l.color) * (l.power * lh.eval_factor);
        const f3 c = clamp_contribution(throughput * lr * w, depth, p);
        radiance = radiance + c;
        if (ev) add3(ev->emission, c);
        ps.transparent_bounce += 1u;
        tmin = next_float_up(lh.distance);
        excluded = lh.index;
        if (ps.transparent_bounce >= p.transparent_max) {
            if (ev) ev->terminated = 1u;
            return false;
        }
    }
    return true;
}

// BackgroundEventStage (src/luisa/path_kernel_background_event.cpp:14-160).
__device__ __forceinline__ void background_event(const SceneView &s, const RenderParams &p, uint32_t ray_visibility,
                                                 f3 throughput, const PathState &ps, f3 &radiance, float &transparency,
                                                 psy_path_event *ev) {
    const f3 bg = ld3(s.background);
    const f3 c = clamp_contribution(throughput * bg * 1.0f, ps.bounce, p);
    const bool world_visible = (s.world_visibility & ray_visibility) != 0u;
    if (p.transparent_background != 0u && (ps.flag & kFlagTransparentBackground) != 0u) {
        transparency += (throughput.x + throughput.y + throughput.z) * (1.0f / 3.0f);
    } else if (world_visible) {
        radiance = radiance + c;
        if (ev) add3(ev->emission, c);
    }
}

// Shades the paths that left the scene: in a sorted queue they come first
// (counters[kCounterMisses] of them).  They end here, so this kernel pushes
// nothing and runs 8 blocks an SM instead of k_shade's 4; with it and without the
// light-distribution search of paths that take no light sample, shading a
// 1080p procedural frame (64 spp) went from 138 to 114 ms.
template <bool kMulti>
__global__ void __launch_bounds__(128, PSY_MISS_MIN_BLOCKS)
    k_shade_miss(const __grid_constant__ SceneView s_arg, const __grid_constant__ RenderParams p_arg,
                 const __grid_constant__ PathBuffers b, const JobGpu *jobs, uint32_t sort_threshold) {
    if (b.counters[0] < sort_threshold || b.counters[kCounterTail] != 0u) return;
    const uint32_t count = b.counters[kCounterMisses];
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x) {
        const uint32_t i = b.queue_sorted[q];
        const uint32_t job = kMulti ? b.job[i] : 0u;
        const SceneView &s = kMulti ? jobs[job].s : s_arg;
        const RenderParams &p = kMulti ? jobs[job].p : p_arg;
        float4 ro, rd, tp4, rad4;
        uint4 st, st2;
        load_pair(b.ray_o, i, ro, rd);
        load_pair(b.tp, i, tp4, rad4);
        load_pair(b.st, i, st, st2);
        const Ray ray{mk3(ro.x, ro.y, ro.z), mk3(rd.x, rd.y, rd.z), ro.w, rd.w};
        const f3 throughput = mk3(tp4.x, tp4.y, tp4.z);
        f3 radiance = mk3(rad4.x, rad4.y, rad4.z);
        float transparency = rad4.w;
        PathState ps = unpack_state(st, st2);
        const uint32_t ray_visibility = contract_visibility(ps.visibility);
        bool alive = true;
        if (s.lamp_count > 0u)
            alive = lamp_events(s, p, b, i, ray, ray.tmax, ray_visibility, throughput, tp4.w,
                                (st2.x & kSt2Delta) != 0u, ps, radiance, nullptr);
        if (alive) background_event(s, p, ray_visibility, throughput, ps, radiance, transparency, nullptr);
        b.rad_final[i] = make_float4(radiance.x, radiance.y, radiance.z, transparency);
    }
}

// continuation_probability (cycles_path_state.h:413-447).
__device__ __forceinline__ float continuation_probability(const PathState &ps, const RenderParams &p, f3 throughput) {
    const bool tr_state = (ps.flag & kFlagTransparent) != 0u;
    const bool before_min = tr_state ? ps.transparent_bounce <= p.transparent_min : ps.bounce <= p.minimum;
    return before_min ? 1.0f : minf_(sqrtf(max_abs_component(throughput)), 1.0f);
}

// light_tree.forward_pdf (src/luisa/path_tracer_light_tree.cpp:799-838) of a hit
// emissive triangle, seen from the previous scatter (its normal `mn`).
__device__ __forceinline__ float tree_forward_pdf(const SceneView &s, const SurfacePoint &sp, f3 origin, float4 mn,
                                                  uint32_t flag) {
    return lt_pdf(s, lt_triangle_emitter(s, sp.object, sp.cycles_prim), origin, mk3(mn.x, mn.y, mn.z),
                  (flag & kFlagMisHadTransmission) != 0u);
}

// The light tree's work of a shading step, ahead of k_shade: each hit path's
// pick and, where it hit an emitter, the forward pdf, left in the unused words
// of its hit sector.  A descent evaluates about thirty importances; inside
// k_shade it ran at that kernel's 4 blocks an SM and evicted its code.
template <bool kMulti>
__global__ void __launch_bounds__(128, PSY_PICK_MIN_BLOCKS)
    k_light_pick(const __grid_constant__ SceneView s_arg, const __grid_constant__ RenderParams p_arg,
                 const __grid_constant__ PathBuffers b, const JobGpu *jobs, uint32_t sort_threshold) {
    if (b.counters[kCounterTail] != 0u || (kMulti && b.counters[kCounterWaveTree] == 0u)) return;
    const uint32_t count = b.counters[0];
    const bool sorted = sort_threshold != 0u && count >= sort_threshold;
    const uint32_t *queue = sorted ? b.queue_sorted : b.queue_in;
    const uint32_t begin = sorted ? b.counters[kCounterMisses] : 0u;
    for (uint32_t q = begin + blockIdx.x * blockDim.x + threadIdx.x; q < count; q += gridDim.x * blockDim.x) {
        const uint32_t i = queue[q];
        const uint32_t job = kMulti ? b.job[i] : 0u;
        const SceneView &s = kMulti ? jobs[job].s : s_arg;
        const RenderParams &p = kMulti ? jobs[job].p : p_arg;
        float4 h4, ro, rd;
        uint4 hp4, st, st2;
        load_pair(b.hit, i, h4, hp4);
        if (hp4.x == kInvalid || !p.use_light_tree || !p.nee) continue;
        load_pair(b.ray_o, i, ro, rd);
        load_pair(b.st, i, st, st2);
        const PathState ps = unpack_state(st, st2);
        const Hit h{h4.x, h4.y, h4.z, __float_as_uint(h4.w), hp4.x, __float_as_uint(h4.w)};
        const SurfacePoint sp = surface_point(s, h, mk3(rd.x, rd.y, rd.z));
        const BakedMaterialGpu mat = s.baked[sp.material];
        float forward = 0.0f;
        if (s.triangle_emitters > 0u && mat.emission_sampling != 0u && mat.has_emission)
            forward = tree_forward_pdf(s, sp, mk3(ro.x, ro.y, ro.z), b.mis_n[i], ps.flag);
        // paths that end here, or have nothing to evaluate a light with, pick
        // none (a lamp event on the way may still change a transparent
        // path's continuation)
        bool pick = (mat.runtime & kRuntimeBsdfHasEval) != 0u && (st2.x & kSt2TermNext) == 0u;
        const uint32_t x = p.win_x + st2.w % p.win_w, y = p.win_y + st2.w / p.win_w;
        const uint32_t rng_hash = pixel_hash(x, p.full_h - 1u - y, p.seed);
        const uint32_t sample = b.sample[i];
        if (pick && (s.lamp_count == 0u || (ps.flag & kFlagTransparent) == 0u)) {
            const float4 tp = b.tp[i];
            const float cp = continuation_probability(ps, p, mk3(tp.x, tp.y, tp.z));
            pick = !(cp <= 0.0f) && (cp == 1.0f || !(sample_4d(p, sample, rng_hash, ps.rng_offset).x >= cp));
        }
        uint32_t entry = kInvalid;
        float pdf = 0.0f;
        if (pick) {
            const DistEntryGpu e = lt_sample(s, sample_4d(p, sample, rng_hash, ps.rng_offset + 1u).z, sp.position, sp.n,
                                             (mat.runtime & kRuntimeBsdfHasTransmission) != 0u);
            if (e.kind <= 1u) {
                entry = e.kind == 0u ? e.index : s.triangle_emitters + e.index;
                pdf = e.selection_pdf;
            }
        }
        b.hit_prim[i] = make_uint4(hp4.x, entry, __float_as_uint(pdf), __float_as_uint(forward));
    }
}

// What shading a path leaves for its queues.
struct ShadeResult {
    bool keep;    // the path goes on
    bool shadow;  // and / or sends the shadow ray below
    bool final;   // it ends here: its radiance and shadow contribution go to rad_final
    float4 sh_o, sh_d, sh_c;
    uint4 sh_ids;
};

// One path step after its closest hit: background / emission + forward MIS,
// roulette, AOV, NEE sample, closure sample and path-state transition.  Reads
// and writes path i's record.
// kTrace selects the variant that records the per-path trace; the render
// variant carries no trace code.
// kPicked: k_light_pick has left the light tree's pick and forward pdf in the
// path's record.
template <bool kTrace, bool kGlossy, bool kPicked>
__device__ __forceinline__ ShadeResult shade_path(const SceneView &s, const RenderParams &p, const PathBuffers &b,
                                                  uint32_t i, uint32_t step, uint32_t trace_path,
                                                  psy_path_trace *trace) {
    ShadeResult out;
    out.keep = out.shadow = out.final = false;
    psy_path_event *ev = nullptr;
    if (kTrace && trace && i == trace_path && step < PSY_TRACE_MAX_EVENTS) {
        ev = &trace->events[step];
        trace->event_count = step + 1u;
    }
    float4 ro, rd, tp4, rad4, h4;
    uint4 st, st2, hp4;
    load_pair(b.ray_o, i, ro, rd);
    load_pair(b.tp, i, tp4, rad4);
    load_pair(b.st, i, st, st2);
    load_pair(b.hit, i, h4, hp4);
    Ray ray{mk3(ro.x, ro.y, ro.z), mk3(rd.x, rd.y, rd.z), ro.w, rd.w};
    f3 throughput = mk3(tp4.x, tp4.y, tp4.z);
    float previous_bsdf_pdf = tp4.w;
    f3 radiance = mk3(rad4.x, rad4.y, rad4.z);
    float transparency = rad4.w;
    PathState ps = unpack_state(st, st2);
    bool previous_delta = (st2.x & kSt2Delta) != 0u;
    bool primary_recorded = (st2.x & kSt2Primary) != 0u;
    const bool terminate_on_next_surface = (st2.x & kSt2TermNext) != 0u;
    const bool terminate_after_transparent = (st2.x & kSt2TermAfter) != 0u;
    const uint32_t ray_visibility = contract_visibility(ps.visibility);
    const uint32_t sample = b.sample[i];
    const uint32_t local = st2.w;
    const uint32_t x = p.win_x + local % p.win_w;
    const uint32_t y = p.win_y + local / p.win_w;
    const uint32_t rng_hash = pixel_hash(x, p.full_h - 1u - y, p.seed);
    const float terminate_sample = sample_4d(p, sample, rng_hash, ps.rng_offset + 0u).x;
    const float4 ls4 = sample_4d(p, sample, rng_hash, ps.rng_offset + 1u);
    const f3 light_sample = mk3(ls4.x, ls4.y, ls4.z);
    const float light_terminate = sample_4d(p, sample, rng_hash, ps.rng_offset + 2u).x;
    const float4 bs4 = sample_4d(p, sample, rng_hash, ps.rng_offset + 3u);
    // the flat distribution's pick; without a trace to record it, only
    // paths that take a light sample search for theirs
    DistEntryGpu selected{0.0f, 0.0f, 3u, 0u};
    if (kTrace && !p.use_light_tree) selected = distribution_sample(s, light_sample.z);
    const uint32_t prim = hp4.x;
    if (ev) {
        ev->rng_offset = ps.rng_offset;
        ev->random_terminate = terminate_sample;
        set3(ev->random_light, light_sample);
        ev->random_light_terminate = light_terminate;
        set3(ev->random_bsdf, mk3(bs4.x, bs4.y, bs4.z));
        ev->light_kind = selected.kind;
        ev->light_index = selected.index;
        const bool missed = prim == kInvalid;
        ev->hit_t = missed ? 0.0f : h4.x;
        ev->hit_u = missed ? 0.0f : h4.y;
        ev->hit_v = missed ? 0.0f : h4.z;
        ev->closure_index = kInvalid;
        ev->hit_object = kInvalid;
        ev->hit_primitive = kInvalid;
    }
    const uint32_t depth = ps.bounce;
    bool alive = true;
    if (s.lamp_count > 0u)
        alive = lamp_events(s, p, b, i, ray, prim == kInvalid ? ray.tmax : h4.x, ray_visibility, throughput,
                            previous_bsdf_pdf, previous_delta, ps, radiance, ev);
    if (!alive) {
        // a lamp event used up the transparent budget
    } else if (prim == kInvalid) {
        background_event(s, p, ray_visibility, throughput, ps, radiance, transparency, ev);
        if (ev) ev->terminated = 1u;
        alive = false;
    } else {
        Hit h;
        h.t = h4.x;
        h.u = h4.y;
        h.v = h4.z;
        h.instance = __float_as_uint(h4.w);
        h.prim = prim;
        h.object = h.instance;
        const SurfacePoint sp = surface_point(s, h, ray.d);
        if (ev) {
            ev->hit_object = h.object;
            ev->hit_primitive = sp.cycles_prim;
        }
        const BakedMaterialGpu mat = s.baked[sp.material];
        SurfaceClosures<kGlossy> closures;
        const ClosurePoint cpt{sp.n, sp.ng, -ray.d, safe_normalize(-ray.d, sp.n), mat.bump_correction != 0u,
                               sp.back_facing};
        collect_surface<kGlossy>(s, mat, cpt, closures);
        // SurfaceShadingStageImpl::emit (src/luisa/path_kernel_surface_shading.cpp:117-250)
        float emission_weight = 1.0f;
        if (p.nee && s.triangle_emitters > 0u && mat.emission_sampling != 0u && mat.has_emission) {
            const bool competing = depth > 0u && !previous_delta;
            float selection_pdf =
                0.5f * length(cross(sp.wp1 - sp.wp0, sp.wp2 - sp.wp0)) * s.triangle_area_pdf;
            if (p.use_light_tree) {
                if constexpr (kPicked) selection_pdf = __uint_as_float(hp4.w);
                else selection_pdf = tree_forward_pdf(s, sp, ray.o, b.mis_n[i], ps.flag);
            }
            const float light_pdf = emissive_forward_pdf(selection_pdf, mat.emission_sampling, ray.o,
                                                         sp.position, sp.wp0, sp.wp1, sp.wp2,
                                                         // the geometric normal before the back-face
                                                         // flip (path_kernel_surface_shading.cpp:130-134)
                                                         sp.back_facing ? -sp.ng : sp.ng);
            const bool available = light_pdf > 0.0f;
            emission_weight = forward_light_weight(p.direct_mode, previous_bsdf_pdf, light_pdf, competing, available);
        }
        const f3 ec = clamp_contribution(throughput * closures.emission * emission_weight, depth, p);
        radiance = radiance + ec;
        if (ev) add3(ev->emission, ec);
        if (terminate_on_next_surface) {
            alive = false;
            if (ev) ev->terminated = 1u;
        }
        if (alive) {
            const float cp = continuation_probability(ps, p, throughput);
            if (ev) ev->continuation_probability = cp;
            if (cp <= 0.0f) {
                alive = false;
            } else if (cp != 1.0f) {
                if (terminate_sample >= cp) alive = false;
                else throughput = throughput / cp;
            }
            if (!alive && ev) ev->terminated = 1u;
        }
        if (alive) {
            if (depth == 0u) {
                f3 aov_albedo, aov_normal, aov_transparency;
                surface_aov<kGlossy>(closures, cpt, aov_albedo, aov_normal, aov_transparency);
                const float4 a4 = b.aov_a[i];
                const f3 acc = mk3(a4.x, a4.y, a4.z) + throughput * aov_albedo;
                b.aov_a[i] = make_float4(acc.x, acc.y, acc.z, 0.0f);
                const f3 alpha = clamp3(mk3(1.0f) - aov_transparency, 0.0f, 1.0f);
                const float average_alpha = (alpha.x + alpha.y + alpha.z) * (1.0f / 3.0f);
                const bool writes_normal = !primary_recorded && (p.pass_alpha_threshold == 0.0f ||
                                                                 average_alpha >= p.pass_alpha_threshold);
                if (writes_normal) {
                    b.aov_n[i] = make_float4(aov_normal.x, aov_normal.y, aov_normal.z, 0.0f);
                    primary_recorded = true;
                    ps.flag |= kFlagSinglePassDone;
                }
            }
            const uint32_t runtime = mat.runtime | (sp.back_facing ? kRuntimeBackfacing : 0u);
            if (p.use_light_tree) {
                // light-tree pick after shading (src/luisa/path_kernel_pipeline.cpp:150-159)
                if constexpr (kPicked) {
                    if (hp4.y != kInvalid)
                        selected = {0.0f, __uint_as_float(hp4.z), hp4.y < s.triangle_emitters ? 0u : 1u,
                                    hp4.y < s.triangle_emitters ? hp4.y : hp4.y - s.triangle_emitters};
                } else {
                    selected = lt_sample(s, light_sample.z, sp.position, sp.n,
                                         (runtime & kRuntimeBsdfHasTransmission) != 0u);
                }
                if (ev) {
                    ev->light_kind = selected.kind;
                    ev->light_index = selected.index;
                }
            }
            const uint32_t lobe_mask = terminate_after_transparent ? kEventTransparent : 0xffffffffu;
            // Direct lighting (src/luisa/path_kernel_pipeline.cpp:160-172)
            if (p.nee && (runtime & kRuntimeBsdfHasEval) != 0u) {
                if (!kTrace && !p.use_light_tree) selected = distribution_sample(s, light_sample.z);
                f3 lp = mk3(0.0f), ldir = mk3(0.0f);
                float ldist = 0.0f;
                bool distant = false;
                f3 surviving = mk3(0.0f);
                uint32_t light_obj = kInvalid, light_prim = kInvalid;
                bool emit = false;
                // The light sample of either kind, then one BSDF
                // evaluation, MIS weight and light roulette shared by
                // both (a warp's lanes that picked triangles and lamps
                // evaluate together).
                bool sampled = false, weigh_mis = true;
                f3 light_radiance = mk3(0.0f);
                float light_pdf = 0.0f, pdf_divisor = 1.0f;
                if (selected.kind == 0u) {
                    // EmissiveMeshLightingComponent (src/luisa/path_kernel_nee_emissive_mesh.cpp:32-296)
                    const Emitter em = load_emitter(s.emitters + selected.index);
                    const TriSample ls = sample_triangle(sp.position, em.p0, em.p1, em.p2,
                                                         mk2(light_sample.x, light_sample.y));
                    const bool side = sampled_side(em.emission_sampling, em.ng, ls.direction);
                    const float pdf = ls.pdf * selected.selection_pdf;
                    if (ls.valid && side && em.area > 0.0f && pdf > 0.0f) {
                        const bool is_transmission = dot(ls.direction, sp.n) < 0.0f;
                        const bool same_primitive = em.cycles_prim == sp.cycles_prim && em.object == sp.object;
                        const f3 oriented = is_transmission ? -sp.ng : sp.ng;
                        const bool reject_self = same_primitive && dot(ls.direction, oriented) > 0.0f;
                        if (!reject_self) {
                            sampled = true;
                            light_radiance = ld3(__ldg(&s.baked[em.material].emission));
                            light_pdf = pdf;
                            pdf_divisor = pdf;
                            lp = ls.position;
                            light_obj = em.object;
                            light_prim = em.cycles_prim;
                            ldir = ls.direction;
                        }
                    }
                } else if (selected.kind == 1u) {
                    // AnalyticLightingComponent (src/luisa/path_kernel_nee_analytic.cpp:98-428)
                    const psy_light_desc &l = s.lights[selected.index];
                    if (!(depth > l.max_bounces)) {
                        const AnalyticSample a =
                            sample_analytic(l, s.lamp_consts[selected.index], sp.position, sp.n,
                                            (runtime & kRuntimeBsdfHasTransmission) != 0u,
                                            mk2(light_sample.x, light_sample.y));
                        const float pdf = a.pdf * selected.selection_pdf;
                        if (a.valid && pdf > 0.0f) {
                            sampled = true;
                            light_radiance = ld3(l.color) * (l.power * a.eval_factor);
                            light_pdf = pdf;
                            pdf_divisor = maxf_(pdf, 1.0e-20f);
                            // MIS only for lamps a BSDF ray can also hit
                            // (path_kernel_nee_analytic.cpp:286-292)
                            weigh_mis = (l.flags & kLightFlagForward) != 0u;
                            lp = a.position;
                            ldir = a.direction;
                            distant = l.type == PSY_LIGHT_DISTANT;
                        }
                    }
                }
                if (sampled) {
                    const Evaluation e = evaluate_mixture<kGlossy>(closures, cpt, ldir, lobe_mask, -1);
                    const float mis = weigh_mis ? nee_light_weight(p.direct_mode, light_pdf, e.pdf) : 1.0f;
                    const f3 weighted = e.f * light_radiance * (mis / pdf_divisor);
                    if (any_nonzero(weighted)) {
                        const f3 unshadowed = weighted * mk3(1.0f);
                        surviving =
                            unshadowed * light_roulette_weight(unshadowed, light_terminate, p.inv_rr_threshold);
                        emit = any_nonzero(surviving);
                    }
                }
                if (emit) {
                    // make_shadow_origin (src/luisa/path_kernel_surface_geometry.cpp:168-185)
                    const Xform w2o = world_to_object(s, sp.instance);
                    const f3 so = origin_with_self_exclusion(sp, xform_point(w2o, sp.position),
                                                             xform_direction(w2o, ldir));
                    const f3 off = lp - so;
                    const float fd = sqrtf(maxf_(dot(off, off), 1.0e-20f));
                    const f3 sdir = distant ? ldir : off / fd;
                    ldist = distant ? 1.0e30f : fd;
                    const f3 c = throughput * surviving;
                    out.sh_o = make_float4(so.x, so.y, so.z, ldist);
                    out.sh_d = make_float4(sdir.x, sdir.y, sdir.z, __uint_as_float(ps.transparent_bounce));
                    out.sh_c = make_float4(c.x, c.y, c.z, __uint_as_float(depth));
                    out.sh_ids = make_uint4(sp.object, sp.cycles_prim, light_obj, light_prim);
                    out.shadow = true;
                }
            }
            // SurfaceScatterStageImpl::emit (src/luisa/path_kernel_surface_scatter.cpp:136-291)
            const SurfaceSample ss = sample_surface<kGlossy>(closures, cpt, bs4.z, mk2(bs4.x, bs4.y), lobe_mask);
            if (ev) {
                ev->closure_index = ss.closure_index;
                ev->bsdf_pdf = ss.eval.pdf;
                set3(ev->wi, ss.wi);
            }
            if (!ss.valid || ss.eval.pdf <= 0.0f) {
                alive = false;
            } else {
                const bool transparent = (ss.eval.events & kEventTransparent) != 0u;
                const bool singular = (ss.eval.events & kEventSingular) != 0u;
                const uint32_t label = label_from_events(ss.eval.events);
                throughput = throughput * (ss.eval.f / ss.eval.pdf);
                if (ev) {
                    ev->label = label;
                    set3(ev->throughput, throughput);
                }
                if (any_nan(throughput) || throughput.x < 0.0f || throughput.y < 0.0f || throughput.z < 0.0f) {
                    alive = false;
                } else {
                    ps = next_surface(ps, label, runtime, p);
                    if (!transparent) {
                        previous_bsdf_pdf = ss.eval.pdf;
                        previous_delta = singular;
                        b.mis_n[i] = make_float4(sp.n.x, sp.n.y, sp.n.z, 0.0f);
                    }
                    if (ev) {
                        ev->bounce = ps.bounce;
                        ev->transparent_bounce = ps.transparent_bounce;
                        ev->flag = ps.flag;
                        ev->visibility = ps.visibility;
                    }
                    if (transparent) {
                        ray.tmin = next_float_up(h.t);
                    } else {
                        const f3 wi = normalize(ss.wi);
                        const Xform w2o = world_to_object(s, sp.instance);
                        ray.o = origin_with_self_exclusion(sp, sp.object_position, xform_direction(w2o, wi));
                        ray.d = wi;
                        ray.tmin = 0.0f;
                        ray.tmax = 1.0e30f;
                    }
                    out.keep = true;
                    st2.y = sp.object;
                    st2.z = sp.cycles_prim;
                }
            }
            if (!out.keep && ev) ev->terminated = 1u;
        }
    }
    const float4 rad_out = make_float4(radiance.x, radiance.y, radiance.z, transparency);
    // an ended path's radiance goes to the film's array; a path still
    // alive after the last step (none, by the step bound) is written
    // there as well
    out.final = !out.keep || step + 1u >= p.steps;
    if (out.final) b.rad_final[i] = rad_out;
    if (out.keep) {
        store_pair(b.ray_o, i, make_float4(ray.o.x, ray.o.y, ray.o.z, ray.tmin),
                   make_float4(ray.d.x, ray.d.y, ray.d.z, ray.tmax));
        store_pair(b.tp, i, make_float4(throughput.x, throughput.y, throughput.z, previous_bsdf_pdf), rad_out);
        const uint4 st_out = make_uint4(ps.flag, ps.visibility, ps.rng_offset,
                                        ps.bounce | (ps.diffuse_bounce << 8) | (ps.glossy_bounce << 16) |
                                            (ps.transmission_bounce << 24));
        uint32_t bits = ps.transparent_bounce & 0xffu;
        if (previous_delta) bits |= kSt2Delta;
        if (primary_recorded) bits |= kSt2Primary;
        if ((ps.flag & kFlagTerminateOnNextSurface) != 0u) bits |= kSt2TermNext;
        if ((ps.flag & kFlagTerminateAfterTransparent) != 0u) bits |= kSt2TermAfter;
        st2.x = bits;
        store_pair(b.st, i, st_out, st2);
    }
    return out;
}

// kMulti: paths of a batched wavefront, each shaded with its job's scene and
// parameters.
template <bool kTrace, bool kMulti, bool kGlossy>
__global__ void __launch_bounds__(128, PSY_SHADE_MIN_BLOCKS)
    k_shade(const __grid_constant__ SceneView s_arg, const __grid_constant__ RenderParams p_arg,
            const __grid_constant__ PathBuffers b, uint32_t step, uint32_t trace_path, psy_path_trace *trace,
            const JobGpu *jobs, uint32_t sort_threshold) {
    // a batched wavefront launches both variants; the one that does not
    // match the wavefront's glossy flag (set by k_begin_round) returns
    if (kMulti && (b.counters[kCounterWaveGlossy] != 0u) != kGlossy) return;
    const uint32_t count = b.counters[0];
    if (b.counters[kCounterTail] != 0u) return;
    const bool sorted = sort_threshold != 0u && count >= sort_threshold;
    const uint32_t *queue = sorted ? b.queue_sorted : b.queue_in;
    // a sorted queue's misses are k_shade_miss's (a traced launch takes all)
    const uint32_t begin = sorted && !kTrace ? b.counters[kCounterMisses] : 0u;
    const uint32_t rounds = (count - begin + gridDim.x * blockDim.x - 1u) / (gridDim.x * blockDim.x);
    // Every lane runs the same number of rounds so the warp-aggregated queue
    // pushes see the whole warp.
    for (uint32_t round = 0; round < rounds; ++round) {
        const uint32_t q = begin + round * gridDim.x * blockDim.x + blockIdx.x * blockDim.x + threadIdx.x;
        const bool active = q < count;
        ShadeResult r{};
        uint32_t i = 0u;
        if (active) {
            i = queue[q];
            const uint32_t job = kMulti ? b.job[i] : 0u;
            const SceneView &s = kMulti ? jobs[job].s : s_arg;
            const RenderParams &p = kMulti ? jobs[job].p : p_arg;
            r = shade_path<kTrace, kGlossy, !kTrace>(s, p, b, i, step, trace_path, trace);
        }
        const uint32_t slot = warp_push(&b.counters[1], r.keep);
        if (r.keep) b.queue_out[slot] = i;
        const uint32_t sslot = warp_push(&b.counters[2], r.shadow);
        if (r.shadow) {
            b.sh_o[sslot] = r.sh_o;
            b.sh_d[sslot] = r.sh_d;
            b.sh_c[sslot] = r.sh_c;
            b.sh_ids[sslot] = r.sh_ids;
            b.sh_path[sslot] = i | (r.final ? kShadowFinal : 0u);
        }
    }
}

// A triangle's padded extent on one axis: as the host pads its boxes
// (padded in psy_host.cpp), in double, rounded outward.
__device__ __forceinline__ void pad_axis(float a, float b, float c, float &lo, float &hi) {
    const double l = fminf(a, fminf(b, c)), h = fmaxf(a, fmaxf(b, c));
    const double pad = 1e-5 * (h - l) + 1e-6 * fmax(fabs(l), fabs(h)) + 1e-30;
    lo = nextafterf(float(l - pad), -INFINITY);
    hi = nextafterf(float(h + pad), INFINITY);
}

// Triangle records of all meshes from their vertex arrays: thread i takes
// leaf slot i, which holds triangle order[i] of its mesh.
__global__ void k_pack_triangles(const MeshGpu *meshes, uint32_t mesh_count, const float *positions,
                                 const float *normals, const uint32_t *indices, const uint32_t *tri_materials,
                                 const uint32_t *order, uint32_t triangles, TriGpu *tris, ShadeTriGpu *shade_tris) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= triangles) return;
    // the last mesh that begins at or before the slot (meshes without
    // triangles share their successor's first slot)
    uint32_t lo = 0u, hi = mesh_count;
    while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (meshes[mid].tri_offset <= i) lo = mid;
        else hi = mid;
    }
    const MeshGpu m = meshes[lo];
    const uint32_t local = order[i];
    const uint32_t *idx = indices + m.index_offset + 3u * local;
    const float *P = positions + 3u * m.vertex_offset, *N = normals + 3u * m.vertex_offset;
    f3 p[3], n[3];
    for (int k = 0; k < 3; ++k) {
        p[k] = ld3(P + 3u * idx[k]);
        n[k] = m.smooth ? ld3(N + 3u * idx[k]) : mk3(0.0f);
    }
    float bl[3], bh[3];
    pad_axis(p[0].x, p[1].x, p[2].x, bl[0], bh[0]);
    pad_axis(p[0].y, p[1].y, p[2].y, bl[1], bh[1]);
    pad_axis(p[0].z, p[1].z, p[2].z, bl[2], bh[2]);
    TriGpu t;
    t.v0 = make_float4(p[0].x, p[0].y, p[0].z, __uint_as_float(local));
    t.v1 = make_float4(p[1].x, p[1].y, p[1].z, bl[0]);
    t.v2 = make_float4(p[2].x, p[2].y, p[2].z, bl[1]);
    t.lo_z_hi = make_float4(bl[2], bh[0], bh[1], bh[2]);
    tris[i] = t;
    const f3 ng = safe_normalize(cross(p[1] - p[0], p[2] - p[0]), mk3(0.0f, 0.0f, 1.0f));
    ShadeTriGpu o;
    for (int k = 0; k < 3; ++k) {
        float *op = k == 0 ? o.p0 : k == 1 ? o.p1 : o.p2, *on = k == 0 ? o.n0 : k == 1 ? o.n1 : o.n2;
        op[0] = p[k].x, op[1] = p[k].y, op[2] = p[k].z;
        on[0] = n[k].x, on[1] = n[k].y, on[2] = n[k].z;
    }
    o.ng[0] = ng.x, o.ng[1] = ng.y, o.ng[2] = ng.z;
    o.material = m.material_offset == kInvalid ? kInvalid : tri_materials[m.material_offset + local];
    o.pad[0] = o.pad[1] = 0u;
    shade_tris[m.tri_offset + local] = o;
}

// Evaluates the closure programs of materials [first, first + count), one
// material a thread (microseconds, when a scene is compiled or a material
// edited).  While shading and shadow rays walked the programs per path, the
// walk's arrays took 1.6 of the shading kernel's 1.9 KB of local memory and
// most of the shadow kernel's, whose register budget they also held up: 1080p
// procedural frame, 64 spp: shading 182 -> 148 ms, shadow rays 108 -> 82 ms (now
// 8 blocks an SM); value programs, 512x512 at 4 spp: 5.3 -> 2.7 ms.
__global__ void k_bake_materials(const __grid_constant__ SceneView s, BakedMaterialGpu *baked, BakedClosureGpu *closures,
                                 uint32_t first, uint32_t count) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const MaterialGpu m = s.materials[first + i];
    baked[first + i] = bake_material(s, m, closures + m.closure_first);
}

// ------------------------------------------------------------------ shadow
// make_trace_shadow_callable (src/luisa/path_tracer_geometry.cpp:75-174)
// iterates closest hits: a transparent surface multiplies its extinction
// and advances tmin past its distance, an opaque one or the
// transparent_max_bounces budget blocks the ray.  The transmittance that
// loop produces depends only on the set of surfaces in [0, tmax]: zero if
// any is opaque or if more than (max - depth) surfaces lie on it, else the
// product in distance order (coincident distances count once, the greatest
// identity standing for them).  The kernel computes it with one any-hit
// traversal: it stops at the first opaque surface, collects transparent
// ones, and multiplies them sorted by distance.  A ray with more surfaces
// than the collector holds keeps the nearest, multiplies them, and is traced
// again from behind the last of them.

constexpr int kShadowList = 8;

// The material of a surface, with kMaterialTransparent where it has
// transparent closures.
__device__ __forceinline__ uint32_t surface_material(const SceneView &s, uint32_t instance, uint32_t cycles_prim) {
    const uint32_t m = __ldg(&s.entries[instance].material);
    return m != kInvalid ? m : __ldg(&s.shade_tris[cycles_prim].material);
}

// The transparent surfaces a shadow ray has met, and their product so far.
struct ShadowHits {
    float t[kShadowList];
    uint32_t object[kShadowList], prim[kShadowList], material[kShadowList];
    int n;
    uint32_t passed;  // surfaces before the ray's current start
    f3 transmittance;  // and their product
    bool blocked, overflow;
};

__device__ __forceinline__ void shadow_begin(ShadowHits &h, uint32_t transparent_depth) {
    h.blocked = h.overflow = false;
    h.n = 0;
    h.passed = transparent_depth;
    h.transmittance = mk3(1.0f);
}

// A surface on the ray; true once it is known to be blocked.
__device__ __forceinline__ bool shadow_hit(ShadowHits &h, const SceneView &s, const RenderParams &p, uint32_t instance,
                                           uint32_t cycles_prim, float t) {
    // opaque-only scenes stop at the first accepted candidate
    const uint32_t tagged = s.any_transparent ? surface_material(s, instance, cycles_prim) : 0u;
    if ((tagged & kMaterialTransparent) == 0u) {
        h.blocked = true;
        return true;
    }
    const uint32_t material = tagged & ~kMaterialTransparent;
    for (int k = 0; k < h.n; ++k) {
        if (h.t[k] == t) {  // coincident: keep the greatest identity
            if (instance > h.object[k] || (instance == h.object[k] && cycles_prim > h.prim[k])) {
                h.object[k] = instance;
                h.prim[k] = cycles_prim;
                h.material[k] = material;
            }
            return false;
        }
    }
    int slot = h.n;
    if (h.n == kShadowList) {
        // more surfaces than the collector holds: keep the nearest, unless
        // they exceed the ray's budget already
        if (h.passed + uint32_t(kShadowList) >= p.transparent_max) {
            h.blocked = true;
            return true;
        }
        h.overflow = true;
        slot = 0;
        for (int k = 1; k < kShadowList; ++k)
            if (h.t[k] > h.t[slot]) slot = k;
        if (t > h.t[slot]) return false;
    } else {
        ++h.n;
    }
    h.t[slot] = t;
    h.object[slot] = instance;
    h.prim[slot] = cycles_prim;
    h.material[slot] = material;
    return false;
}

// Multiplies the surfaces met in distance order.  False if the ray has to go
// on from behind them: `t` has been restarted there.
__device__ __forceinline__ bool shadow_resolve(ShadowHits &h, TraversalState &t, const SceneView &s,
                                               const RenderParams &p) {
    // (transparent_max - passed surfaces may still lie on the ray)
    if (uint32_t(h.n) > (h.passed >= p.transparent_max ? 0u : p.transparent_max - h.passed)) h.blocked = true;
    if (!h.blocked) {
        for (int i = 1; i < h.n; ++i) {
            const float kt = h.t[i];
            const uint32_t km = h.material[i];
            int j = i - 1;
            while (j >= 0 && h.t[j] > kt) {
                h.t[j + 1] = h.t[j];
                h.material[j + 1] = h.material[j];
                --j;
            }
            h.t[j + 1] = kt;
            h.material[j + 1] = km;
        }
        for (int i = 0; i < h.n; ++i) {
            const f3 e = clamp3(ld3(__ldg(&s.baked[h.material[i]].extinction)), 0.0f, 1.0f);
            if (!(max_component(e) > 0.0f)) {
                h.blocked = true;
                break;
            }
            h.transmittance = h.transmittance * e;
        }
        if (!h.blocked && h.overflow) {
            h.passed += uint32_t(h.n);
            Ray ray = t.ray;
            ray.tmin = next_float_up(h.t[h.n - 1]);
            traversal_begin(t, s, ray, PSY_VISIBILITY_SHADOW, t.src_obj, t.src_prim, t.light_obj, t.light_prim);
            h.overflow = false;
            h.n = 0;
            return false;
        }
    }
    if (h.blocked) h.transmittance = mk3(0.0f);
    return true;
}

// The NEE contribution of a resolved shadow ray, added to its path's radiance.
__device__ __forceinline__ f3 shadow_contribute(const PathBuffers &b, const RenderParams &p, f3 transmittance, float4 c,
                                                uint32_t path, bool final) {
    f3 contribution = mk3(0.0f);
    if (transmittance.x > 0.0f || transmittance.y > 0.0f || transmittance.z > 0.0f) {
        contribution = clamp_contribution(mk3(c.x, c.y, c.z) * transmittance, __float_as_uint(c.w), p);
        float4 &dst = final ? b.rad_final[path] : b.rad[path];
        float4 r = dst;
        r.x += contribution.x;
        r.y += contribution.y;
        r.z += contribution.z;
        dst = r;
    }
    return contribution;
}

// Persistent any-hit shadow kernel (same refill scheme as k_intersect):
// transparent hits are collected per lane and resolved by distance once the
// traversal ends.
// A warp's rays wait for one another's steps, so a queue too short to fill
// the `warps` resident warps is spread over them, as few rays to a warp as it
// takes: 1080p procedural frame, 64 spp 79.4 -> 76.9 ms, value materials at 512x512
// 0.76 -> 0.66 ms.  (k_intersect loses more to the registers this takes: 142.5
// -> 148.4 ms.)
// kMulti: shadow rays of a batched wavefront, each in its path's job.
template <bool kMulti>
__global__ void __launch_bounds__(128, PSY_SHADOW_MIN_BLOCKS)
    k_shadow(const __grid_constant__ SceneView s_arg, const __grid_constant__ RenderParams p_arg,
             const __grid_constant__ PathBuffers b, uint32_t step, uint32_t trace_path, psy_path_trace *trace,
             const JobGpu *jobs, uint32_t sort_threshold, uint32_t warps) {
    const uint32_t count = b.counters[2];
    if (b.counters[kCounterTail] != 0u) return;
    const bool sorted = sort_threshold != 0u && count >= sort_threshold;
    const bool takes = lane_id() < min(32u, max(1u, (count + warps - 1u) / warps));
    TraversalState t;
    t.node = kLinkDone;
    t.leaves = 0u;
    bool active = false, exhausted = false;
    uint32_t q_cur = 0u, job = 0u;
    ShadowHits h;
    shadow_begin(h, 0u);
    for (;;) {
        uint32_t q = warp_fetch(&b.counters[4], count, takes && !active, exhausted);
        if (sorted && q != kInvalid) q = b.queue_sorted[q];
        if (kMulti && q != kInvalid) job = b.job[b.sh_path[q] & ~kShadowFinal];
        const SceneView &s = kMulti ? jobs[job].s : s_arg;
        const RenderParams &p = kMulti ? jobs[job].p : p_arg;
        if (q != kInvalid) {
            q_cur = q;
            const float4 o = b.sh_o[q], d = b.sh_d[q];
            const uint4 ids = b.sh_ids[q];
            const Ray ray{mk3(o.x, o.y, o.z), mk3(d.x, d.y, d.z), 0.0f, o.w};
            traversal_begin(t, s, ray, PSY_VISIBILITY_SHADOW, ids.x, ids.y, ids.z, ids.w);
            shadow_begin(h, __float_as_uint(d.w));
            active = true;
        }
        const int busy = __popc(__ballot_sync(kFullMask, active));
        if (busy == 0) break;
        traverse_warp<false>(t, s, exhausted ? 32 : min(32, 32 - busy + kRefillLanes),
                             [&](uint32_t ii, uint32_t, uint32_t cp, uint32_t, float th, float, float) {
            return shadow_hit(h, s, p, ii, cp, th);
        });
        if (!active || t.node != kLinkDone || t.leaves != 0u) continue;
        if (!shadow_resolve(h, t, s, p)) continue;
        active = false;
        const uint32_t owner = b.sh_path[q_cur], path = owner & ~kShadowFinal;
        const f3 contribution =
            shadow_contribute(b, p, h.transmittance, b.sh_c[q_cur], path, (owner & kShadowFinal) != 0u);
        if (trace && path == trace_path && step < PSY_TRACE_MAX_EVENTS) set3(trace->events[step].nee, contribution);
    }
}

// -------------------------------------------------------------------- tail
// All remaining steps of a queue that has become short (k_end_step marks the
// step from which counters[0] is below the limit), one path a lane: closest
// hit, shading and shadow ray follow one another without a launch between.
// In a short queue a step's three launches each wait for their longest ray
// while the GPU idles, so a path that still bounces pays that wait for
// every step; here it pays only for the paths of its own warp, and a warp
// takes few of them (as many as spread the queue over all resident warps).
// 128x128 procedural viewport at 1 spp: 2.44 -> 1.11 ms; value materials at
// 512x512, 4 spp: 2.68 -> 2.19 ms.  A path's steps take longer here than spread
// over wavefronts (fewer warps an SM, all kinds of steps in one), so a queue has
// to leave most lanes idle: the limit of 20 Ki paths is about a third of the
// resident lanes.  Device ms of renders of 8 scenes, 96x96 to 1280x720 at 1 spp,
// with limits of 0 / 16 Ki / 20 Ki / 32 Ki / 64 Ki paths: closed box, 255x257 0.50 / 0.44 /
// 0.44 / 0.48 / 0.84; glass, 1024x512 2.22 / 2.31 / 2.30 / 2.58 / 2.82; glossy with the light
// tree, 181x181 1.16 / 0.66 / 0.75 / 0.62 / 0.62; procedural, 512x512 3.86 / 3.06 / 3.08 /
// 3.00 / 3.62.
template <bool kMulti, bool kGlossy>
__global__ void __launch_bounds__(128, PSY_TAIL_MIN_BLOCKS)
    k_tail(const __grid_constant__ SceneView s_arg, const __grid_constant__ RenderParams p_arg,
           const __grid_constant__ PathBuffers b, const uint32_t *odd_queue, const JobGpu *jobs,
           unsigned long long *stats) {
    if (kMulti && (b.counters[kCounterWaveGlossy] != 0u) != kGlossy) return;
    if (b.counters[kCounterTail] == 0u) return;
    const uint32_t start = b.counters[kCounterTail] - 1u, count = b.counters[0];
    const uint32_t *queue = (start & 1u) != 0u ? odd_queue : b.queue_in;
    const uint32_t warps = gridDim.x * 4u, warp = blockIdx.x * 4u + (threadIdx.x >> 5);
    const uint32_t share = min(32u, (count + warps - 1u) / warps);
    uint32_t closest_rays = 0u, shadow_rays = 0u;
    for (uint32_t base = warp * share; base < count; base += warps * share) {
        const uint32_t q = base + lane_id();
        bool active = lane_id() < share && q < count;
        const uint32_t i = active ? queue[q] : 0u;
        const uint32_t job = kMulti && active ? b.job[i] : 0u;
        const SceneView &s = kMulti ? jobs[job].s : s_arg;
        const RenderParams &p = kMulti ? jobs[job].p : p_arg;
        for (uint32_t step = start; __any_sync(kFullMask, active); ++step) {
            TraversalState t;
            t.node = kLinkDone;
            t.leaves = 0u;
            ClosestHit best;
            if (active) {
                closest_begin(best, t, s, b, i);
                closest_rays += 1u;
            }
            traverse_warp<true>(t, s, 32, [&](uint32_t ii, uint32_t local, uint32_t, uint32_t slot, float th, float u, float v) {
                return closest_hit(best, t, s, ii, local, slot, th, u, v);
            });
            ShadeResult r{};
            if (active) {
                uint32_t prim;
                if (closest_ambiguous(best, t, s, prim)) {
                    best = closest_exact(s, b, i);
                    prim = closest_prim(best, s);
                }
                closest_store(best, prim, b, i);
                r = shade_path<false, kGlossy, false>(s, p, b, i, step, kInvalid, nullptr);
            }
            if (__any_sync(kFullMask, r.shadow)) {
                ShadowHits h;
                shadow_begin(h, __float_as_uint(r.sh_d.w));
                t.node = kLinkDone;
                t.leaves = 0u;
                bool pending = r.shadow;
                if (pending) {
                    const Ray ray{ld3(r.sh_o), ld3(r.sh_d), 0.0f, r.sh_o.w};
                    traversal_begin(t, s, ray, PSY_VISIBILITY_SHADOW, r.sh_ids.x, r.sh_ids.y, r.sh_ids.z, r.sh_ids.w);
                    shadow_rays += 1u;
                }
                while (__any_sync(kFullMask, pending)) {
                    traverse_warp<false>(t, s, 32, [&](uint32_t ii, uint32_t, uint32_t cp, uint32_t, float th, float, float) {
                        return shadow_hit(h, s, p, ii, cp, th);
                    });
                    if (pending && shadow_resolve(h, t, s, p)) {
                        shadow_contribute(b, p, h.transmittance, r.sh_c, i, r.final);
                        pending = false;
                    }
                }
            }
            active = r.keep && step + 1u < p.steps;
        }
    }
    closest_rays = __reduce_add_sync(kFullMask, closest_rays);
    shadow_rays = __reduce_add_sync(kFullMask, shadow_rays);
    if (lane_id() == 0u && closest_rays != 0u) {
        atomicAdd(&stats[0], (unsigned long long)closest_rays);
        atomicAdd(&stats[1], (unsigned long long)shadow_rays);
    }
}

// -------------------------------------------------------------------- film
// accumulate_path_sample + write_film (src/luisa/path_kernel_setup.cpp:903-1062):
// samples are added in sample order.
// One window pixel: its samples of the batch added to the film in sample
// order, one at a time, so the film does not depend on how the samples were
// grouped into batches.
__device__ __forceinline__ void film_pixel(const PathBuffers &b, uint32_t px, uint32_t pixels, uint32_t samples,
                                           uint32_t path_begin, float4 *combined, float4 *normal, float4 *albedo,
                                           uint32_t *sample_count, uint32_t trace_path, psy_path_trace *trace) {
    float4 c = combined[px], n = normal[px], a = albedo[px];
    auto add = [&](uint32_t i, const float4 &r, const float4 &nn, const float4 &aa) {
        f3 rad = mk3(r.x, r.y, r.z);
        if (any_nan(rad)) rad = mk3(0.0f);
        c.x += rad.x;
        c.y += rad.y;
        c.z += rad.z;
        c.w += r.w;
        n.x += nn.x;
        n.y += nn.y;
        n.z += nn.z;
        n.w += 1.0f;
        a.x += aa.x;
        a.y += aa.y;
        a.z += aa.z;
        a.w += 1.0f;
        if (trace && i == trace_path) set3(trace->radiance, rad);
    };
    // Four samples' loads are issued before any of them is added (the
    // trace store could alias them, so the compiler would not hoist a later
    // sample's loads above it); the sums still run in sample order.
    constexpr uint32_t kGroup = 4u;
    uint32_t k = 0;
    for (; k + kGroup <= samples; k += kGroup) {
        float4 r[kGroup], nn[kGroup], aa[kGroup];
#pragma unroll
        for (uint32_t u = 0; u < kGroup; ++u) {
            const uint32_t i = path_begin + (k + u) * pixels + px;
            r[u] = b.rad_final[i];
            nn[u] = b.aov_n[i];
            aa[u] = b.aov_a[i];
        }
#pragma unroll
        for (uint32_t u = 0; u < kGroup; ++u) add(path_begin + (k + u) * pixels + px, r[u], nn[u], aa[u]);
    }
    for (; k < samples; ++k) {
        const uint32_t i = path_begin + k * pixels + px;
        add(i, b.rad_final[i], b.aov_n[i], b.aov_a[i]);
    }
    combined[px] = c;
    normal[px] = n;
    albedo[px] = a;
    sample_count[px] += samples;
}

__global__ void k_film(PathBuffers b, uint32_t pixels, uint32_t samples, float4 *combined, float4 *normal,
                       float4 *albedo, uint32_t *sample_count, uint32_t trace_path, psy_path_trace *trace) {
    for (uint32_t px = blockIdx.x * blockDim.x + threadIdx.x; px < pixels; px += gridDim.x * blockDim.x)
        film_pixel(b, px, pixels, samples, 0u, combined, normal, albedo, sample_count, trace_path, trace);
}

// Film of every item of a batched wavefront (a job appears in at most one
// item per wavefront, so its pixels have one writer).
__global__ void k_film_batch(const JobGpu *jobs, const BatchItem *items, const uint32_t *round, PathBuffers b) {
    const uint32_t film_pixels = round[1], item_count = round[2];
    for (uint32_t g = blockIdx.x * blockDim.x + threadIdx.x; g < film_pixels; g += gridDim.x * blockDim.x) {
        const BatchItem it = items[find_item(items, item_count, g, [](const BatchItem &t) { return t.film_begin; })];
        const JobGpu &j = jobs[it.job];
        film_pixel(b, g - it.film_begin, it.pixels, it.samples, it.path_begin, j.combined, j.normal, j.albedo,
                   j.sample_count, kInvalid, nullptr);
    }
}

// Start of a batched wavefront: the wavefront `*cursor` of a planned call
// becomes current (its header and items copied to the fixed buffers every
// later kernel reads), the queue counters are set, and the cursor advances.
// One block.
__global__ void k_begin_round(uint32_t *counters, uint32_t *round, BatchItem *items, const uint32_t *plan_rounds,
                              const BatchItem *plan_items, uint32_t *cursor, uint32_t max_items,
                              uint32_t tail_paths) {
    const uint32_t w = *cursor;
    const uint32_t n = plan_rounds[4u * w + 2u];
    for (uint32_t k = threadIdx.x; k < n && k < max_items; k += blockDim.x)
        items[k] = plan_items[size_t(w) * max_items + k];
    __syncthreads();
    if (threadIdx.x == 0) {
        round[0] = plan_rounds[4u * w];
        round[1] = plan_rounds[4u * w + 1u];
        round[2] = n;
        counters[kCounterWaveGlossy] = plan_rounds[4u * w + 3u] & 1u;
        counters[kCounterWaveTree] = plan_rounds[4u * w + 3u] >> 1;
        counters[0] = round[0];
        counters[1] = counters[2] = counters[3] = counters[4] = counters[kCounterAmbiguous] = 0u;
        counters[kCounterTail] = round[0] < tail_paths ? 1u : 0u;
        *cursor = w + 1u;
    }
}

// End of step `step`: its rays are counted, the survivors become the next
// step's queue, and a queue shorter than `tail_paths` is marked for k_tail --
// the launches of later steps find the mark and return.
__global__ void k_end_step(uint32_t *counters, unsigned long long *stats, uint32_t step, uint32_t tail_paths) {
    if (counters[kCounterTail] != 0u) return;
    stats[0] += counters[0];
    stats[1] += counters[2];
    counters[0] = counters[1];
    counters[1] = 0u;
    counters[2] = 0u;
    counters[3] = 0u;
    counters[4] = 0u;
    counters[kCounterAmbiguous] = 0u;
    if (counters[0] < tail_paths) counters[kCounterTail] = step + 2u;
}

__global__ void k_set_counters(uint32_t *counters, uint32_t n, uint32_t tail_paths) {
    counters[0] = n;
    counters[1] = 0u;
    counters[2] = 0u;
    counters[3] = 0u;
    counters[4] = 0u;
    counters[kCounterAmbiguous] = 0u;
    counters[kCounterTail] = n < tail_paths ? 1u : 0u;
}

__global__ void k_check_counts(const uint32_t *counts, uint32_t n, uint32_t expected, uint32_t *mismatch) {
    bool bad = false;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        bad = bad || counts[i] != expected;
    if (__any_sync(kFullMask, bad) && (threadIdx.x & 31u) == 0u) atomicOr(mismatch, 1u);
}

// write_passes (src/luisa/path_tracer_session.cpp:71-270): Combined = sum x
// exposure / samples with alpha 1 - transparency / samples clamped to [0, 1];
// Normal and Albedo = sum / samples; Sample Count as a float.
__global__ void k_resolve_pass(const float4 *film, const uint32_t *counts, uint32_t n, uint32_t kind, float exposure,
                               float *out) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t c = counts[i];
        if (kind == 2u) {
            out[i] = float(c);
            continue;
        }
        const float den = float(c > 1u ? c : 1u);
        float4 v = film[i];
        if (kind == 0u) {
            const float k = exposure / den;
            v.x *= k;
            v.y *= k;
            v.z *= k;
            const float a = 1.0f - v.w / den;
            v.w = a < 0.0f ? 0.0f : (1.0f < a ? 1.0f : a);
        } else {
            v.x /= den;
            v.y /= den;
            v.z /= den;
            v.w /= den;
        }
        reinterpret_cast<float4 *>(out)[i] = v;
    }
}

__global__ void k_debug_sobol(const float4 *table, uint32_t size, const uint32_t *queries, uint32_t count, float4 *out,
                              uint32_t *out_index) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const uint32_t *q = queries + 5u * i;
    const uint32_t h = pixel_hash(q[0], q[1], q[2]);
    const uint32_t idx = shuffled_sample_index(q[3], q[4], h, size);
    out[i] = table[idx];
    out_index[i] = idx;
}

__global__ void k_debug_light_distribution(const __grid_constant__ SceneView s, const float *u, uint32_t count,
                                           uint32_t *out_kind, uint32_t *out_index, float *out_pdf) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const DistEntryGpu e = distribution_sample(s, u[i]);
    out_kind[i] = e.kind;
    out_index[i] = e.index;
    out_pdf[i] = e.selection_pdf;
}

__global__ void k_debug_light_tree(const __grid_constant__ SceneView s, const float4 *queries, const uint32_t *pdf_emitters, uint32_t count,
                                   uint32_t *out_emitters, float *out_sample_pdf, float *out_reverse_pdf) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float4 a = queries[2u * i], b = queries[2u * i + 1u];
    const f3 point = mk3(a.x, a.y, a.z), n = mk3(b.x, b.y, b.z);
    const bool tr = b.w != 0.0f;
    const DistEntryGpu e = lt_sample(s, a.w, point, n, tr);
    const bool valid = e.kind == 0u || e.kind == 1u;
    out_emitters[i] = valid ? (e.kind == 0u ? e.index : s.triangle_emitters + e.index) : kInvalid;
    out_sample_pdf[i] = valid ? e.selection_pdf : 0.0f;
    out_reverse_pdf[i] = lt_pdf(s, pdf_emitters[i], point, n, tr);
}

// ----------------------------------------------------------------- launches

int launch_grid(uint32_t work, int block, const LaunchConfig &lc) {
    const uint32_t blocks = (work + uint32_t(block) - 1u) / uint32_t(block);
    const uint32_t cap = uint32_t(lc.sms) * lc.stream_blocks_per_sm;
    return int(blocks < 1u ? 1u : (blocks > cap ? cap : blocks));
}

uint32_t launch_raygen(cudaStream_t st, const LaunchConfig &lc, const RenderParams &p, const PathBuffers &b, uint32_t pixels,
                   uint32_t paths, uint32_t sample_base, uint32_t trace_path, psy_path_trace *trace) {
    k_raygen<<<launch_grid(paths, int(lc.stream_block), lc), lc.stream_block, 0, st>>>(p, b, pixels, paths, sample_base,
                                                                                    trace_path, trace);
    return 1u;
}
uint32_t launch_set_counters(cudaStream_t st, const LaunchConfig &lc, uint32_t *counters, uint32_t n) {
    k_set_counters<<<1, 1, 0, st>>>(counters, n, lc.tail_paths);
    return 1u;
}
// Persistent kernels: enough resident warps to fill every SM (bounded by the
// work so small queues launch few blocks).
int shade_grid(uint32_t work, const LaunchConfig &lc) {
    const uint32_t blocks = (work + 127u) / 128u;
    const uint32_t cap = uint32_t(lc.sms) * lc.shade_blocks_per_sm;
    return int(blocks < 1u ? 1u : (blocks > cap ? cap : blocks));
}
// A queue of at most `max_work` paths can reach the sort threshold; where it
// cannot, the sort's launches are left out.
bool sorts_queue(const LaunchConfig &lc, uint32_t max_work) {
    return lc.sort_threshold != 0u && max_work >= lc.sort_threshold;
}
template <bool kMulti>
uint32_t launch_sort(cudaStream_t st, const LaunchConfig &lc, const SceneView &s, const RenderParams &p, const PathBuffers &b,
                 const JobGpu *jobs, uint32_t max_work) {
    k_sort_count<kMulti><<<launch_grid(max_work, 256, lc), 256, 0, st>>>(s, p, b, jobs, lc.sort_threshold);
    k_sort_scan<<<1, 1024, 0, st>>>(b, lc.sort_threshold, 0u, true);
    // ranks are packed in 21 bits: keep every block's chunk below 2^20 paths
    const int scatter_blocks = std::max(launch_grid(max_work, 256, lc), int((max_work >> 20) + 1u));
    k_sort_scatter<<<scatter_blocks, 256, 0, st>>>(b, lc.sort_threshold, 0u);
    return 3u;
}
uint32_t launch_shadow_sort(cudaStream_t st, const LaunchConfig &lc, const PathBuffers &b, uint32_t max_work) {
    const uint32_t thr = lc.shadow_sort_threshold;
    k_sort_count_shadow<<<launch_grid(max_work, 256, lc), 256, 0, st>>>(b, thr);
    k_sort_scan<<<1, 1024, 0, st>>>(b, thr, 2u, false);
    const int scatter_blocks = std::max(launch_grid(max_work, 256, lc), int((max_work >> 20) + 1u));
    k_sort_scatter<<<scatter_blocks, 256, 0, st>>>(b, thr, 2u);
    return 3u;
}
int persistent_grid(uint32_t work, const LaunchConfig &lc) {
    const uint32_t blocks = (work + 127u) / 128u;
    const uint32_t cap = uint32_t(lc.sms) * lc.traversal_blocks_per_sm;
    return int(blocks < 1u ? 1u : (blocks > cap ? cap : blocks));
}

// Warps of a persistent grid that are resident at once.
uint32_t resident_warps(int grid, int blocks_per_sm, const LaunchConfig &lc) {
    return 4u * uint32_t(std::min(grid, lc.sms * blocks_per_sm));
}

template <bool kMulti>
uint32_t launch_ray_sort(cudaStream_t st, const LaunchConfig &lc, const SceneView &s, const PathBuffers &b, const JobGpu *jobs,
                     uint32_t max_work) {
    const uint32_t thr = lc.ray_sort_threshold;
    k_sort_count_rays<kMulti><<<launch_grid(max_work, 256, lc), 256, 0, st>>>(s, b, jobs, thr);
    k_sort_scan<<<1, 1024, 0, st>>>(b, thr, 0u, false);
    const int scatter_blocks = std::max(launch_grid(max_work, 256, lc), int((max_work >> 20) + 1u));
    k_sort_scatter<<<scatter_blocks, 256, 0, st>>>(b, thr, 0u);
    return 3u;
}
uint32_t launch_intersect(cudaStream_t st, const LaunchConfig &lc, const SceneView &s, const PathBuffers &b, uint32_t max_work) {
    const uint32_t sort = lc.ray_sort_threshold == 0u ? 0u : launch_ray_sort<false>(st, lc, s, b, nullptr, max_work);
    k_intersect<false><<<persistent_grid(max_work, lc), 128, 0, st>>>(s, b, nullptr, lc.ray_sort_threshold);
    k_closest_exact<false><<<lc.sms, 128, 0, st>>>(s, b, nullptr);
    return sort + 2u;
}
uint32_t launch_shade(cudaStream_t st, const LaunchConfig &lc, const SceneView &s, const RenderParams &p, const PathBuffers &b,
                  uint32_t max_work, uint32_t step, uint32_t trace_path, psy_path_trace *trace) {
    const bool sorts = sorts_queue(lc, max_work);
    uint32_t launches = sorts ? launch_sort<false>(st, lc, s, p, b, nullptr, max_work) : 0u;
    const int grid = shade_grid(max_work, lc);
    if (sorts && !trace) {
        k_shade_miss<false><<<grid, 128, 0, st>>>(s, p, b, nullptr, lc.sort_threshold);
        ++launches;
    }
    if (p.use_light_tree && !trace) {
        k_light_pick<false><<<grid, 128, 0, st>>>(s, p, b, nullptr, lc.sort_threshold);
        ++launches;
    }
    if (trace && s.has_glossy)
        k_shade<true, false, true><<<grid, 128, 0, st>>>(s, p, b, step, trace_path, trace, nullptr, lc.sort_threshold);
    else if (trace)
        k_shade<true, false, false><<<grid, 128, 0, st>>>(s, p, b, step, trace_path, trace, nullptr, lc.sort_threshold);
    else if (s.has_glossy)
        k_shade<false, false, true><<<grid, 128, 0, st>>>(s, p, b, step, trace_path, trace, nullptr, lc.sort_threshold);
    else
        k_shade<false, false, false><<<grid, 128, 0, st>>>(s, p, b, step, trace_path, trace, nullptr, lc.sort_threshold);
    return launches + 1u;
}
uint32_t launch_shadow(cudaStream_t st, const LaunchConfig &lc, const SceneView &s, const RenderParams &p, const PathBuffers &b,
                   uint32_t max_work, uint32_t step, uint32_t trace_path, psy_path_trace *trace) {
    const uint32_t sort = lc.shadow_sort_threshold == 0u ? 0u : launch_shadow_sort(st, lc, b, max_work);
    const int grid = persistent_grid(max_work, lc);
    k_shadow<false><<<grid, 128, 0, st>>>(s, p, b, step, trace_path, trace, nullptr, lc.shadow_sort_threshold,
                                          resident_warps(grid, PSY_SHADOW_MIN_BLOCKS, lc));
    return sort + 1u;
}
uint32_t launch_begin_round(cudaStream_t st, const LaunchConfig &lc, uint32_t *counters, uint32_t *round, BatchItem *items,
                        const uint32_t *plan_rounds, const BatchItem *plan_items, uint32_t *cursor, uint32_t max_items) {
    k_begin_round<<<1, 256, 0, st>>>(counters, round, items, plan_rounds, plan_items, cursor, max_items, lc.tail_paths);
    return 1u;
}
uint32_t launch_end_step(cudaStream_t st, const LaunchConfig &lc, uint32_t *counters, unsigned long long *stats,
                     uint32_t step) {
    k_end_step<<<1, 1, 0, st>>>(counters, stats, step, lc.tail_paths);
    return 1u;
}
// Blocks of the tail kernel: all that are resident, but no more than give
// each warp a path.
int tail_grid(const LaunchConfig &lc, uint32_t max_work) {
    return int(std::min(uint32_t(lc.sms) * PSY_TAIL_MIN_BLOCKS, (std::min(max_work, lc.tail_paths) + 3u) / 4u));
}
uint32_t launch_tail(cudaStream_t st, const LaunchConfig &lc, const SceneView &s, const RenderParams &p, const PathBuffers &b,
                 uint32_t max_work, unsigned long long *stats) {
    if (lc.tail_paths == 0u) return 0u;
    const int grid = tail_grid(lc, max_work);
    if (s.has_glossy) k_tail<false, true><<<grid, 128, 0, st>>>(s, p, b, b.queue_out, nullptr, stats);
    else k_tail<false, false><<<grid, 128, 0, st>>>(s, p, b, b.queue_out, nullptr, stats);
    return 1u;
}
uint32_t launch_tail_batch(cudaStream_t st, const LaunchConfig &lc, const JobGpu *jobs, const PathBuffers &b,
                       uint32_t max_work, unsigned long long *stats) {
    if (lc.tail_paths == 0u) return 0u;
    const int grid = tail_grid(lc, max_work);
    k_tail<true, false><<<grid, 128, 0, st>>>(SceneView{}, RenderParams{}, b, b.queue_out, jobs, stats);
    k_tail<true, true><<<grid, 128, 0, st>>>(SceneView{}, RenderParams{}, b, b.queue_out, jobs, stats);
    return 2u;
}
void launch_check_counts(cudaStream_t st, const uint32_t *counts, uint32_t n, uint32_t expected, uint32_t *mismatch) {
    cudaMemsetAsync(mismatch, 0, sizeof(uint32_t), st);
    const uint32_t blocks = n == 0u ? 1u : (n + 255u) / 256u;
    k_check_counts<<<blocks < 1184u ? blocks : 1184u, 256, 0, st>>>(counts, n, expected, mismatch);
}
void launch_resolve_pass(cudaStream_t st, const float4 *film, const uint32_t *counts, uint32_t n, uint32_t kind,
                         float exposure, float *out) {
    const uint32_t blocks = n == 0u ? 1u : (n + 255u) / 256u;
    k_resolve_pass<<<blocks < 2368u ? blocks : 2368u, 256, 0, st>>>(film, counts, n, kind, exposure, out);
}
uint32_t launch_film(cudaStream_t st, const LaunchConfig &lc, const PathBuffers &b, uint32_t pixels, uint32_t samples, float4 *combined,
                 float4 *normal, float4 *albedo, uint32_t *sample_count, uint32_t trace_path, psy_path_trace *trace) {
    k_film<<<launch_grid(pixels, int(lc.stream_block), lc), lc.stream_block, 0, st>>>(b, pixels, samples, combined, normal,
                                                                                      albedo, sample_count, trace_path,
                                                                                      trace);
    return 1u;
}
// Batched wavefront: every kernel reads each path's job record.
uint32_t launch_raygen_batch(cudaStream_t st, const LaunchConfig &lc, const JobGpu *jobs, const BatchItem *items, const uint32_t *round,
                         const PathBuffers &b, uint32_t max_paths) {
    k_raygen_batch<<<launch_grid(max_paths, int(lc.stream_block), lc), lc.stream_block, 0, st>>>(jobs, items, round, b);
    return 1u;
}
uint32_t launch_intersect_batch(cudaStream_t st, const LaunchConfig &lc, const JobGpu *jobs, const PathBuffers &b, uint32_t max_work) {
    const uint32_t sort = lc.ray_sort_threshold == 0u ? 0u : launch_ray_sort<true>(st, lc, SceneView{}, b, jobs, max_work);
    k_intersect<true><<<persistent_grid(max_work, lc), 128, 0, st>>>(SceneView{}, b, jobs, lc.ray_sort_threshold);
    k_closest_exact<true><<<lc.sms, 128, 0, st>>>(SceneView{}, b, jobs);
    return sort + 2u;
}
uint32_t launch_shade_batch(cudaStream_t st, const LaunchConfig &lc, const JobGpu *jobs, const PathBuffers &b, uint32_t max_work,
                        uint32_t step) {
    const bool sorts = sorts_queue(lc, max_work);
    uint32_t launches = sorts ? launch_sort<true>(st, lc, SceneView{}, RenderParams{}, b, jobs, max_work) : 0u;
    const int grid = shade_grid(max_work, lc);
    if (sorts) {
        k_shade_miss<true><<<grid, 128, 0, st>>>(SceneView{}, RenderParams{}, b, jobs, lc.sort_threshold);
        ++launches;
    }
    k_light_pick<true><<<grid, 128, 0, st>>>(SceneView{}, RenderParams{}, b, jobs, lc.sort_threshold);
    k_shade<false, true, false><<<grid, 128, 0, st>>>(SceneView{}, RenderParams{}, b, step, kInvalid, nullptr, jobs,
                                                      lc.sort_threshold);
    k_shade<false, true, true><<<grid, 128, 0, st>>>(SceneView{}, RenderParams{}, b, step, kInvalid, nullptr, jobs,
                                                     lc.sort_threshold);
    return launches + 3u;
}
uint32_t launch_shadow_batch(cudaStream_t st, const LaunchConfig &lc, const JobGpu *jobs, const PathBuffers &b, uint32_t max_work,
                         uint32_t step) {
    const uint32_t sort = lc.shadow_sort_threshold == 0u ? 0u : launch_shadow_sort(st, lc, b, max_work);
    const int grid = persistent_grid(max_work, lc);
    k_shadow<true><<<grid, 128, 0, st>>>(SceneView{}, RenderParams{}, b, step, kInvalid, nullptr, jobs,
                                         lc.shadow_sort_threshold, resident_warps(grid, PSY_SHADOW_MIN_BLOCKS, lc));
    return sort + 1u;
}
uint32_t launch_film_batch(cudaStream_t st, const LaunchConfig &lc, const JobGpu *jobs, const BatchItem *items, const uint32_t *round,
                       const PathBuffers &b, uint32_t max_pixels) {
    k_film_batch<<<launch_grid(max_pixels, int(lc.stream_block), lc), lc.stream_block, 0, st>>>(jobs, items, round, b);
    return 1u;
}

void launch_debug_light_tree(cudaStream_t st, const SceneView &s, const float4 *queries, const uint32_t *pdf_emitters,
                             uint32_t count, uint32_t *out_emitters, float *out_sample_pdf, float *out_reverse_pdf) {
    k_debug_light_tree<<<(count + 127u) / 128u, 128, 0, st>>>(s, queries, pdf_emitters, count, out_emitters,
                                                               out_sample_pdf, out_reverse_pdf);
}
void launch_debug_light_distribution(cudaStream_t st, const SceneView &s, const float *u, uint32_t count,
                                     uint32_t *out_kind, uint32_t *out_index, float *out_pdf) {
    k_debug_light_distribution<<<(count + 127u) / 128u, 128, 0, st>>>(s, u, count, out_kind, out_index, out_pdf);
}
void launch_bake_materials(cudaStream_t st, const SceneView &s, BakedMaterialGpu *baked, BakedClosureGpu *closures,
                           uint32_t first, uint32_t count) {
    if (count == 0u) return;
    k_bake_materials<<<(count + 31u) / 32u, 32, 0, st>>>(s, baked, closures, first, count);
}
void launch_pack_triangles(cudaStream_t st, const MeshGpu *meshes, uint32_t mesh_count, const float *positions,
                           const float *normals, const uint32_t *indices, const uint32_t *tri_materials,
                           const uint32_t *order, uint32_t triangles, TriGpu *tris, ShadeTriGpu *shade_tris) {
    if (triangles == 0u) return;
    k_pack_triangles<<<(triangles + 127u) / 128u, 128, 0, st>>>(meshes, mesh_count, positions, normals, indices,
                                                                tri_materials, order, triangles, tris, shade_tris);
}
void launch_debug_sobol(cudaStream_t st, const float4 *table, uint32_t size, const uint32_t *queries, uint32_t count,
                        float4 *out, uint32_t *out_index) {
    k_debug_sobol<<<(count + 127u) / 128u, 128, 0, st>>>(table, size, queries, count, out, out_index);
}

cudaError_t take_stack_overflows(cudaStream_t st, uint32_t *count) {
    unsigned int v = 0u;
    cudaError_t e = cudaMemcpyFromSymbolAsync(&v, g_stack_overflows, sizeof(v), 0, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e == cudaSuccess && v != 0u) {
        const unsigned int zero = 0u;
        e = cudaMemcpyToSymbolAsync(g_stack_overflows, &zero, sizeof(zero), 0, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    }
    *count = v;
    return e;
}

}  // namespace psy
