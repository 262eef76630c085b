// Wavefront form of the trace path.
//
// The reference traces each pixel's whole path in one thread
// (renderer/renderer_GPU.h:22-46 -> renderer/ray_tracer.h:19-108).  Here a
// frame is a sequence of stage kernels over queues in HBM, one round per
// bounce:
//
//   extend      closest hit of every queued ray  -> hit record      (scene/scene_tracer.h:26-98);
//               with meshes: scene candidates, persistent mesh pass, resolve
//   shadow_gen  shading frame of every hit, one shadow ray per facing
//               shadowing light -> shadow queue                      (surface_shader.h:49-59,147-160)
//   shadow      any-hit test of every shadow ray -> per-path occlusion bits
//   shade       full shading with the occlusion bits, area lights, IBL,
//               glow, throughput; reflective/refractive hits append the
//               next bounce ray to the next queue; finished paths are tone
//               mapped and written to the canvas                    (ray_tracer.h:42-107)
//
// Each trace stage keeps only traversal state live, so it runs at a much
// higher occupancy than the fused kernel.  Queues are appended with one
// atomic per warp (ballot + popc prefix).  Shading applies the lights in
// the reference's order from the occlusion bits, so every colour is summed
// in the same order as the reference's per-pixel loop.
#include "kernels.h"
#include "nrc.h"
#include "tracer_core.cuh"
#include "wide_bvh.cuh"

namespace slim {
namespace dev {

// Queue records.
//   ray:    float4 (origin.xyz, pixel)     float4 (direction.xyz, 0)
//   hit:    float4 (normal.xyz, distance)  float4 (u, v, uv_coverage, NdotRd)
//           float4 (geometry, from_behind, triangle id, 0)   -- ints as bits
//   shadow: float4 (origin.xyz, slot<<6 | light)  float4 (direction.xyz, max distance)

SLIM_D uint32_t lane_id() { return threadIdx.x & 31u; }

// Warp-aggregated queue append: one atomicAdd per warp, slots handed out
// by the ballot's prefix popcount.  Returns the slot of a thread whose
// `want` is set.
SLIM_D uint32_t warp_append(uint32_t *counter, bool want) {
    uint32_t active = __activemask();
    uint32_t ballot = __ballot_sync(active, want);
    uint32_t base = 0;
    if (ballot) {
        int leader = __ffs(ballot) - 1;
        if ((int)lane_id() == leader) base = atomicAdd(counter, (uint32_t)__popc(ballot));
        base = __shfl_sync(active, base, leader);
    }
    return base + (uint32_t)__popc(ballot & ((1u << lane_id()) - 1u));
}

// Hit records in three planes of `stride` float4 (one entry per queue slot):
//   plane 0 (normal.xyz, distance), plane 1 (u, v, uv coverage, N.Rd),
//   plane 2 (geometry, from behind, triangle, 0).
// A miss (geometry -1) writes and reads plane 2 only: most primary rays of
// an open scene miss, and their records then cost one 16-byte entry in
// the contiguous plane instead of 48 bytes.
SLIM_D void store_hit(float4 *hits, uint32_t stride, uint32_t slot, int g, const Hit &h) {
    hits[2 * (size_t)stride + slot] =
        make_float4(__int_as_float(g), __uint_as_float((uint32_t)h.from_behind), __uint_as_float(h.id), 0.0f);
    if (g < 0) return;
    hits[slot] = make_float4(h.normal.x, h.normal.y, h.normal.z, h.distance);
    hits[(size_t)stride + slot] = make_float4(h.u, h.v, h.uv_coverage, h.NdotRd);
}
SLIM_D int load_hit(const float4 *hits, uint32_t stride, uint32_t slot, Hit &h) {
    const float4 c = hits[2 * (size_t)stride + slot];
    const int g = __float_as_int(c.x);
    h.distance = INFINITY;
    if (g < 0) return g;
    const float4 a = hits[slot], b = hits[(size_t)stride + slot];
    h.normal = xyz(a);
    h.distance = a.w;
    h.u = b.x; h.v = b.y; h.uv_coverage = b.z; h.NdotRd = b.w;
    h.from_behind = __float_as_uint(c.y) != 0;
    h.id = __float_as_uint(c.z);
    return g;
}

template <bool COUNT>
SLIM_D void flush_stage(unsigned long long *counters, const Work &w) {
    if (!COUNT || !counters) return;
    uint32_t v[9] = {w.primary, w.shadow, w.bounce, w.scene_nodes, w.mesh_nodes, w.triangles, w.geometries,
                     w.mesh_fetches, w.taps};
#pragma unroll
    for (int k = 0; k < 9; k++) {
        unsigned long long s = v[k];
        for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xFFFFFFFFu, s, o);
        if (lane_id() == 0 && s) atomicAdd(counters + k, s);
    }
}

// Radiance-cache state of a frame (see kernels.h CacheFrame).
struct CacheArgs {
    float4 *features, *aux, *radiance;
    uint32_t *count;               // queries
    uint32_t *train_count;         // training paths
    uint32_t train_capacity;
    float4 *t_features, *t_targets, *t_color, *t_through;
    uint32_t *frame_counter;
    int mode;
    float4 *q_color, *q_through;   // per query: path colour + depth, throughput (null: path slots)
    float4 *q_hit;                 // per query: its hit record, 3 float4 (null: not kept)
};

struct QueueArgs {
    const float4 *rays_in;        // null: primary rays generated from the slot (= sample index)
    float4 *rays_out;
    const uint32_t *count_in;     // null: count = samples
    uint32_t *count_out;          // between rounds: the rays queued for the next
    uint32_t *round_counts;       // the next round's counters
    float4 *hits;                 // hit records, three planes of hit_stride entries
    uint32_t hit_stride;
    float4 *shadow_rays;
    uint32_t *shadow_count;
    unsigned long long *masks;    // per slot: bit i = light i occluded
    float4 *pairs;                // shadow ray x mesh instance candidates, 3 float4 each:
                                  // (local origin, aux distance) (local direction, tag) (walk_record)
    uint32_t *pair_count;
    uint32_t *pair_cursor;
    uint32_t pair_capacity;
    float4 *path_color;           // per path: colour, depth
    float4 *path_throughput;      // per path: throughput
    uint32_t samples;
    uint32_t depth;               // 1-based bounce of this round
    uint32_t light_begin, light_end;
    uint32_t early_depth;         // non-zero: shadow_gen writes every path's canvas depth, shade only colours
    uint32_t slot_begin, slot_end;  // shade: the slots [begin, end) of the queue (end 0: all)
    unsigned long long *counters; // this stage's counter slots, or null
    // radiance cache
    float4 *sink;                 // non-null: finished paths write their linear colour here
                                  // (indexed by the path slot) instead of the canvas
    uint32_t skip_glow_depth;     // no light glow on the segment of this depth (0 = none)
    CacheArgs cache;              // batched frames: queries of requests using the cache
    // batched requests (null in a single-request frame)
    const DevScene *scenes;
    const DevFrame *frames;
};

// Ray records: (origin.xyz, path) (direction.xyz, pid).  `path` indexes the
// path state (colour, throughput); `pid` names the canvas pixel: the pixel
// index in a single-request frame, (request << 23) | pixel in a batch.  The
// two differ for the radiance cache's training paths, whose state lives in
// their own slots, and for batched paths, whose slots are per wave.
constexpr uint32_t kBatchPixelBits = 23;

template <bool BATCH> SLIM_D uint32_t req_of(uint32_t pid) { return BATCH ? pid >> kBatchPixelBits : 0u; }
template <bool BATCH> SLIM_D uint32_t pix_of(uint32_t pid) {
    return BATCH ? pid & ((1u << kBatchPixelBits) - 1u) : pid;
}
template <bool BATCH> SLIM_D const DevScene &scene_of(const DevScene &S, const QueueArgs &A, uint32_t pid) {
    if constexpr (BATCH) return A.scenes[req_of<true>(pid)];
    else return S;
}
template <bool BATCH> SLIM_D const DevFrame &frame_of(const DevFrame &F, const QueueArgs &A, uint32_t pid) {
    if constexpr (BATCH) return A.frames[req_of<true>(pid)];
    else return F;
}

SLIM_D void primary_ray(const DevFrame &F, uint32_t x, uint32_t y, float3 &o, float3 &d) {
    const SlimCameraRayProjection &P = F.projection;
    o = f3(P.camera_position.x, P.camera_position.y, P.camera_position.z);
    d = normalized(primary_direction(P, (int)x, (int)y));
}


SLIM_D void load_ray(const DevFrame &F, const QueueArgs &A, uint32_t slot, float3 &o, float3 &d, uint32_t &path,
                     uint32_t &pid) {
    if (!A.rays_in) {
        const uint2 p = xy_of_slot(F.width, F.rows, slot);
        path = slot;
        pid = (F.row_begin + p.y) * F.width + p.x;
        primary_ray(F, p.x, F.row_begin + p.y, o, d);
        return;
    }
    float4 a = A.rays_in[2 * (size_t)slot], b = A.rays_in[2 * (size_t)slot + 1];
    o = xyz(a);
    path = __float_as_uint(a.w);
    d = xyz(b);
    pid = __float_as_uint(b.w);
}
template <bool BATCH> SLIM_D float cone_scaling(const DevFrame &F, uint32_t pid) {
    if (!F.cones_per_pixel) return 0.0f;
    const uint32_t p = pix_of<BATCH>(pid);
    return pixel_scaling(F.projection, (int)(p % F.width), (int)(p / F.width));
}
template <bool BATCH>
SLIM_D void write_pixel(const DevFrame &F, uint32_t pid, float3 color, float depth, bool with_depth = true) {
    const uint32_t offset = canvas_offset_of(F, pix_of<BATCH>(pid));
    set_color_at(F, offset, f3(tone_mapped_baked(color.x), tone_mapped_baked(color.y), tone_mapped_baked(color.z)));
    if (with_depth) set_depth_at(F, offset, depth);
}

// First statement of every kernel that RoundLaunch::launch may chain: the
// launch before it, and with it all earlier ones, is complete and its memory
// visible from here on.
SLIM_D void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

SLIM_D uint32_t queue_size(const QueueArgs &A) { return A.count_in ? *A.count_in : A.samples; }

// ---- extend: closest hit of every queued ray ----------------------------
template <bool COUNT, bool BATCH>
__global__ void __launch_bounds__(256) k_extend(DevScene S0, DevFrame F0, QueueArgs A) {
    chain_wait();
    uint32_t n = queue_size(A);
    uint32_t stack[kStackCapacity], mesh_stack[kStackCapacity];
    uint32_t err = 0;
    Work w = {};
    for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < n; slot += gridDim.x * blockDim.x) {
        float3 o, d;
        uint32_t path, pid;
        load_ray(F0, A, slot, o, d, path, pid);
        if (!A.rays_in) bump<COUNT>(w.primary);
        const DevScene &S = scene_of<BATCH>(S0, A, pid);
        Ray ray;
        reset(ray, o, d);
        Hit hit;
        int g = scene_trace<COUNT>(S, n, ray, hit, false, INFINITY, stack, mesh_stack, err, w);
        store_hit(A.hits, A.hit_stride, slot, g, hit);
    }
    if (err) atomicOr(F0.error_flags, err);
    flush_stage<COUNT>(A.counters, w);
}

// A batched request's path that reached its radiance-cache vertex: the
// cache answers there, so it is neither shaded nor lit (training paths,
// which carry a sink, are).
template <bool BATCH> SLIM_D bool at_cache_vertex(const DevFrame &F, const QueueArgs &A) {
    return BATCH && F.cache_depth == A.depth && !A.sink;
}

// ---- shadow_gen: one shadow ray per facing, shadowing light -------------
// In a single frame's first round it can also write the canvas depths (the
// shaded hit's depth, infinity where shade leaves none), which are final
// once the primary hits are: they download while the shadows are traced.
template <bool COUNT, bool BATCH>
__global__ void __launch_bounds__(256) k_shadow_gen(DevScene S0, DevFrame F0, QueueArgs A) {
    chain_wait();
    uint32_t n = queue_size(A);
    Work w = {};
    uint32_t stride = gridDim.x * blockDim.x;
    // Every thread of a warp runs the same number of iterations so the
    // queue appends stay warp-uniform.
    uint32_t rounds = (n + stride - 1) / stride;
    for (uint32_t r = 0, slot = blockIdx.x * blockDim.x + threadIdx.x; r < rounds; r++, slot += stride) {
        bool live = slot < n;
        Surface s;
        bool shaded = false;
        uint32_t lights = 0, pid = 0;
        if (live) {
            // a miss reads its 16-byte record and no ray
            Hit hit;
            const int g = load_hit(A.hits, A.hit_stride, slot, hit);
            if (g >= 0) {
                float3 o, d;
                uint32_t path;
                load_ray(F0, A, slot, o, d, path, pid);
                const DevScene &S = scene_of<BATCH>(S0, A, pid);
                const DevFrame &F = frame_of<BATCH>(F0, A, pid);
                lights = S.light_count;
                Geo geo = load_geo(S, (uint32_t)g);
                Mat m = load_mat(S, geo.material);
                if (!at_cache_vertex<BATCH>(F, A) &&
                    !((m.flags & SLIM_MATERIAL_IS_EMISSIVE) && geo.type == SLIM_GEOMETRY_QUAD && !hit.from_behind)) {
                    Ray ray;
                    reset(ray, scale_add(d, kTraceOffset, o), d);
                    prepare_for_shading<COUNT>(S, geo, m, ray, hit, cone_scaling<BATCH>(F, pid), s, w);
                    shaded = true;
                    // occluded-light bits: read by shade for shaded hits only
                    if (A.light_begin == 0) A.masks[slot] = 0ull;
                }
            }
            if (!BATCH && A.early_depth && A.light_begin == 0) {
                const uint2 p = xy_of_slot(F0.width, F0.rows, slot);
                set_depth_at(F0, canvas_offset_of(F0, (F0.row_begin + p.y) * F0.width + p.x),
                             shaded ? depth_at(F0.projection, hit.position) : INFINITY);
            }
        }
        if (!__any_sync(__activemask(), shaded)) continue;      // nothing to light in this warp
        for (uint32_t li = A.light_begin; li < A.light_end; li++) {
            bool want = false;
            if (shaded && li < lights) {
                LightRec l = load_light(scene_of<BATCH>(S0, A, pid), li);
                want = is_facing_light(s, l) && (l.flags & SLIM_LIGHT_IS_SHADOWING);
            }
            uint32_t q = warp_append(A.shadow_count, want);
            if (want) {
                bump<COUNT>(w.shadow);
                A.shadow_rays[2 * (size_t)q] = make_float4(s.P.x, s.P.y, s.P.z, __uint_as_float((slot << 6) | li));
                A.shadow_rays[2 * (size_t)q + 1] = make_float4(s.L.x, s.L.y, s.L.z, s.Ld);
            }
        }
    }
    flush_stage<COUNT>(A.counters, w);
}

// ---- shadow: any-hit tests ------------------------------------------------
//
// An any-hit result is the OR, over every (scene leaf, geometry) the segment
// reaches, of that geometry's test with the leaf's aux distance
// min(leaf far + EPS, max distance) (scene/scene_tracer.h:111-136): the
// culling distance never shrinks before the first hit ends the search, so
// the result does not depend on the order the candidates are tested in.
// The shadow stage uses that freedom:
//   shadow_scene  walks the scene BVH per shadow ray, tests implicit
//                 primitives on the spot and appends one (ray, mesh
//                 instance, aux distance) pair per reached mesh instance;
//   shadow_mesh   a persistent kernel in which every lane visits a node or
//                 two of a mesh's four-wide BVH per loop turn, lets a leaf
//                 wait until enough lanes have one, and fetches the next
//                 pair as soon as its own finishes, so warps stay full
//                 although walk lengths differ by orders of magnitude.

// Where the walk of a mesh with root node bytes `root` starts, for its record.
SLIM_D float4 walk_record(const DevScene &S, const DevMesh &m, float4 root) {
    if (S.binary_walks)
        return make_float4(__uint_as_float(m.node_offset + node_first(root)), __uint_as_float(m.tri_offset),
                           __uint_as_float(m.node_offset), 0.0f);
    return make_float4(__uint_as_float(m.wide_root), __uint_as_float(m.tri_offset), m.wide_extent, 0.0f);
}

SLIM_D bool local_box_test(const DevScene &S, const Geo &g, const Ray &local) {
    float mn[3], mx[3], n, f;
    if (g.type == SLIM_GEOMETRY_MESH) {
        const DevMesh &m = S.meshes[g.mesh];
        for (int i = 0; i < 3; i++) { mn[i] = m.aabb_min[i]; mx[i] = m.aabb_max[i]; }
    } else {
        float e = g.type == SLIM_GEOMETRY_TET ? kTetMax : 1.0f;
        mx[0] = mx[1] = mx[2] = e;
        mn[0] = mn[1] = mn[2] = -e;
        if (g.type == SLIM_GEOMETRY_QUAD) { mn[1] = -kEps; mx[1] = kEps; }
    }
    return hit_aabb(local, mn[0], mn[1], mn[2], mx[0], mx[1], mx[2], n, f);
}

// Candidates of one scene leaf: implicit primitives are tested here, mesh
// instances whose BVH root the local ray reaches become pairs carrying the
// local ray, so the mesh pass starts at the root's children.  Returns true
// once the ray is known occluded.
template <bool COUNT>
SLIM_D bool shadow_leaf(const DevScene &S, const QueueArgs &A, uint32_t tag, uint32_t first, uint32_t count, float lf,
                        const Ray &ray, float max_distance, uint32_t *mesh_stack, uint32_t &err, Work &w) {
    float aux = minr(lf + kEps, max_distance);
    for (uint32_t i = 0; i < count; i++) {
        uint32_t gi = __ldg(S.leaf_geometry + first + i);
        Geo g = load_geo(S, gi);
        if (!(g.flags & SLIM_GEOMETRY_IS_SHADOWING)) continue;
        bump<COUNT>(w.geometries);
        Ray local;
        localize(local, ray.o, ray.d, g);
        if (!local_box_test(S, g, local)) continue;
        bool transparent = (g.flags & SLIM_GEOMETRY_IS_TRANSPARENT) != 0;
        Hit h;
        h.distance = aux;
        switch (g.type) {
            case SLIM_GEOMETRY_QUAD: if (hit_quad(local, h, transparent)) return true; break;
            case SLIM_GEOMETRY_BOX: if (hit_box(local, h, transparent)) return true; break;
            case SLIM_GEOMETRY_SPHERE: if (hit_sphere(local, h, transparent, nullptr)) return true; break;
            case SLIM_GEOMETRY_TET: if (hit_tet(local, h, transparent)) return true; break;
            case SLIM_GEOMETRY_MESH: {
                const DevMesh &m = S.meshes[g.mesh];
                const float4 *nodes = S.mesh_nodes + 2 * (size_t)m.node_offset;
                float ln, lf2;
                float4 ra, rb;
                load_node(nodes, 0, ra, rb);
                bump<COUNT>(w.mesh_nodes);
                if (!(hit_node(local, ra, rb, ln, lf2) && ln < aux)) break;
                if (node_leaf_count(rb)) {
                    if (hit_triangles<COUNT>(S.tri_hot, m.tri_offset, m.tri_count, lf2, local, h, true, w)) return true;
                    break;
                }
                const bool queued = S.binary_walks || m.wide_root != kNoWideBVH;
                uint32_t slot = warp_append(A.pair_count, queued);
                if (queued && slot < A.pair_capacity) {
                    float4 *p = A.pairs + 3 * (size_t)slot;
                    p[0] = make_float4(local.o.x, local.o.y, local.o.z, aux);
                    p[1] = make_float4(local.d.x, local.d.y, local.d.z, __uint_as_float(tag));
                    p[2] = walk_record(S, m, rb);
                } else if (mesh_trace<COUNT>(S, m, local, h, true, mesh_stack, err, w)) {
                    return true;   // the pair queue is full: trace the instance here
                }
            } break;
            default: break;
        }
    }
    return false;
}

// Capped at 64 registers (4 blocks per SM): latency-bound, the extra warps pay
// for the few spills.  With 3 blocks the mesh frame at 1080p takes 1.149 ms and
// the textured one 393 us, with 4 1.147 and 394, with 5 1.153 and 400.
#ifndef SLIM_SHADOW_SCENE_BLOCKS
#define SLIM_SHADOW_SCENE_BLOCKS 4
#endif
template <bool COUNT, bool BATCH>
__global__ void __launch_bounds__(256, SLIM_SHADOW_SCENE_BLOCKS) k_shadow_scene(DevScene S0, DevFrame F, QueueArgs A) {
    chain_wait();
    uint32_t n = *A.shadow_count;
    uint32_t stack[kStackCapacity], mesh_stack[kStackCapacity];
    uint32_t err = 0;
    Work w = {};
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x) {
        float4 a = A.shadow_rays[2 * (size_t)q], b = A.shadow_rays[2 * (size_t)q + 1];
        uint32_t tag = __float_as_uint(a.w);
        const DevScene &S = scene_of<BATCH>(S0, A, BATCH ? __float_as_uint(A.rays_in[2 * (size_t)(tag >> 6) + 1].w) : 0u);
        Ray ray;
        float3 d = xyz(b);
        reset(ray, scale_add(d, kTraceOffset, xyz(a)), d);
        float Ld = b.w;
        bool occluded = false;
        float ln, rn, lf, rf;
        float4 ra, rb;
        const uint4 list = COUNT ? make_uint4(0, 0, 0, 0) : listed_leaves(S, n);
        if (!COUNT && list.x && finite_ray(ray)) {
            for (uint32_t leaves = leaves_hit(S, list.x, ray, Ld, list.w); leaves && !occluded; leaves &= leaves - 1u) {
                load_leaf(S, __ffs((int)leaves) - 1, ra, rb);
                hit_box_finite(ray, ra, rb, ln, lf);
                occluded = shadow_leaf<COUNT>(S, A, tag, node_first(rb), node_leaf_count(rb), lf, ray, Ld, mesh_stack,
                                              err, w);
            }
            if (occluded) atomicOr(A.masks + (tag >> 6), 1ull << (tag & 63u));
            continue;
        }
        load_node(S.scene_nodes, 0, ra, rb);
        bump<COUNT>(w.scene_nodes);
        if (hit_node(ray, ra, rb, ln, lf) && ln < Ld) {
            if (node_leaf_count(rb)) {
                occluded = shadow_leaf<COUNT>(S, A, tag, 0, S.geometry_count, lf, ray, Ld, mesh_stack, err, w);
            } else {
                uint32_t left = node_first(rb), top = 0;
                for (;;) {
                    float4 la, lb, xa, xb;
                    load_node(S.scene_nodes, left, la, lb);
                    load_node(S.scene_nodes, left + 1, xa, xb);
                    bump<COUNT>(w.scene_nodes, 2);
                    bool hl = hit_node(ray, la, lb, ln, lf) && ln < Ld;
                    bool hr = hit_node(ray, xa, xb, rn, rf) && rn < Ld;
                    uint32_t lc = node_first(lb), rc = node_first(xb);
                    bool go_left = hl && !node_leaf_count(lb), go_right = hr && !node_leaf_count(xb);
                    if (hl && node_leaf_count(lb) &&
                        shadow_leaf<COUNT>(S, A, tag, lc, node_leaf_count(lb), lf, ray, Ld, mesh_stack, err, w)) {
                        occluded = true;
                        break;
                    }
                    if (hr && node_leaf_count(xb) &&
                        shadow_leaf<COUNT>(S, A, tag, rc, node_leaf_count(xb), rf, ray, Ld, mesh_stack, err, w)) {
                        occluded = true;
                        break;
                    }
                    if (go_left) {
                        if (go_right) {
                            if (top >= (uint32_t)kStackCapacity) { err |= kErrStack; break; }
                            stack[top++] = rc;
                        }
                        left = lc;
                    } else if (go_right) {
                        left = rc;
                    } else {
                        if (top == 0) break;
                        left = stack[--top];
                    }
                }
            }
        }
        if (occluded) atomicOr(A.masks + (tag >> 6), 1ull << (tag & 63u));
    }
    if (err) atomicOr(F.error_flags, err);
    flush_stage<COUNT>(A.counters, w);
}


// The persistent mesh walks.  They run over the four-wide form of the mesh
// BVHs (wide_bvh.h).  What bounds them is instructions issued at 14-18 busy
// lanes of 32, then the L1 bytes of the nodes (each lane at its own), so the
// form was chosen by both, on the 1080p frame of the 81,920- and
// 130,050-triangle meshes (any-hit launch of the first round, ncu):
//   two-wide, 64 B a step, 24.4 steps per walk        281 M warp instr., 385 us
//   eight-wide, 8-bit planes, 80 B, 9.0 nodes         238 M, L1 50 %, 321 us
//   four-wide, 32-bit planes, 112 B read, 13 nodes    169 M, L1 83 %, 328 us
//   four-wide, 16-bit planes, 80 B, 11.7 nodes        201 M, L1 67 %, 292 us (this)
// (the last also goes to the child that reaches furthest first; 201.0 M, 287 us
// and 55 % of L1's whole throughput in the present build).  The frame: 1.455 ->
// 1.283 ms; with 8 bounces 2.865 -> 2.550 ms.
//
// Nodes a walking lane visits per loop turn: with one 1.35, three 1.38
// against 1.29 ms.
constexpr uint32_t kStepsPerTurn = 2;

// A warp's view of the candidate queue; uniform over the warp.  Idle lanes
// wait until a third of the warp is idle and then fetch together, so the
// fetch code -- one atomic, the candidate loads, the ray set-up -- runs for
// several lanes at once (a third 1.287, a quarter 1.291, a sixth 1.300 ms).
// A launch with few candidates spreads them over its warps, and idle lanes
// take over subtrees of their warp's walks: from the start of such a launch,
// at the end of a large one.
constexpr uint32_t kFetchFraction = 3;
// Candidates per warp below which a launch is such a one: at 8 the frame with
// 8 bounces takes 2.39 ms, at 16 the same, the light meshes at 637 x 359 0.67
// and 0.69 ms (not sharing: 2.53 and 0.70).
constexpr uint32_t kSparse = 8;
struct Feed {
    uint32_t n, quota;
    bool drained;
    SLIM_D Feed(uint32_t n_) : n(n_), drained(n_ == 0) {
        const uint32_t warps = gridDim.x * (blockDim.x >> 5);
        quota = min(32u, (n + warps - 1) / warps);
    }
    SLIM_D bool sparse() const { return quota < kSparse; }
    // lanes with a subtree to give, where idle lanes may take one
    SLIM_D uint32_t donors(bool donor) const {
        return drained || sparse() ? __ballot_sync(0xFFFFFFFFu, donor) : 0u;
    }
    SLIM_D bool fetch(uint32_t idle, uint32_t donors) const {
        if (drained) return false;
        return sparse() ? !donors && __popc(idle) >= 24 : kFetchFraction * (uint32_t)__popc(idle) >= 32u;
    }
    // Candidate of this lane (n: none) when the `idle` lanes fetch.
    SLIM_D uint32_t take(uint32_t *cursor, uint32_t idle) {
        const uint32_t lanes = min((uint32_t)__popc(idle), quota);
        uint32_t base = 0;
        if (lane_id() == 0) base = atomicAdd(cursor, lanes);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        drained = base + lanes >= n;
        const uint32_t rank = (uint32_t)__popc(idle & ((1u << lane_id()) - 1u));
        return (idle >> lane_id() & 1u) && rank < lanes ? min(base + rank, n) : n;
    }
};

// No node: as a reference it counts as a leaf, so no lane steps into it.
constexpr uint32_t kNone = 0xFFFFFFFFu;

// Warp-uniform decision: test waiting leaves now?  Once a third of the warp
// has a leaf waiting, or no lane can step (1.291 ms; a half or a quarter
// 1.296).
constexpr uint32_t kLeafFraction = 3;
SLIM_D bool leaf_round(bool waiting, bool can_step) {
    const uint32_t act = __activemask();
    const uint32_t wait_mask = __ballot_sync(act, waiting);
    const uint32_t step_mask = __ballot_sync(act, can_step);
    return wait_mask && (kLeafFraction * (uint32_t)__popc(wait_mask) >= (uint32_t)__popc(act) || !step_mask);
}
SLIM_D bool fetch_round(bool idle) {
    const uint32_t act = __activemask();
    const uint32_t idle_mask = __ballot_sync(act, idle);
    return idle_mask && (kFetchFraction * (uint32_t)__popc(idle_mask) >= (uint32_t)__popc(act) || idle_mask == act);
}

// 128-thread blocks, capped at 64 registers for the any-hit walks (32 warps
// per SM) and 72 for the closest-hit walks (28): 1.284 ms; any hit at 9 or
// 10 blocks 1.291 and 1.448 ms (spills), closest hit at 6 or 8 blocks 1.307
// and 1.292 ms.
constexpr int kMeshBlock = 128;
#ifndef SLIM_SHADOW_MESH_BLOCKS
#define SLIM_SHADOW_MESH_BLOCKS 8
#endif
#ifndef SLIM_EXTEND_MESH_BLOCKS
#define SLIM_EXTEND_MESH_BLOCKS 7
#endif

// Sharing of walks: an idle lane takes the deepest waiting subtree (the
// bottom entry of the stack) of a lane of its warp that is still walking, so
// the last walks of a launch, and the few walks of a small one, spread over
// their warps instead of running one lane each.  The i-th idle lane (in lane
// order) takes from the i-th lane with a waiting subtree; the giver removes
// the entry from its stack.
struct Steal {
    int from;                   // giving lane for a taker, else -1
    bool gave;
    uint32_t subtree, near;     // stack entry handed over (valid for a taker)
};
template <bool NEAR, typename Entry>
SLIM_D Steal steal_round(uint32_t idle_mask, uint32_t donor_mask, const Entry *stack, uint32_t &bottom, uint32_t &top) {
    const uint32_t below = (1u << lane_id()) - 1u;
    const uint32_t pairs = min((uint32_t)__popc(idle_mask), (uint32_t)__popc(donor_mask));
    const uint32_t my_idle_rank = (uint32_t)__popc(idle_mask & below);
    const bool taker = (idle_mask >> lane_id() & 1u) && my_idle_rank < pairs;
    Steal st;
    st.gave = (donor_mask >> lane_id() & 1u) && (uint32_t)__popc(donor_mask & below) < pairs;
    uint2 give = make_uint2(0, 0);
    if (st.gave) {
        if constexpr (sizeof(Entry) == sizeof(uint2)) give = stack[bottom];
        else give.x = stack[bottom];
        if (++bottom == top) bottom = top = 0;
    }
    uint32_t m = donor_mask;
    for (uint32_t j = 0; taker && j < my_idle_rank; j++) m &= m - 1u;
    const int src = taker ? __ffs((int)m) - 1 : (int)lane_id();
    st.subtree = __shfl_sync(0xFFFFFFFFu, give.x, src);
    st.near = NEAR ? __shfl_sync(0xFFFFFFFFu, give.y, src) : 0u;
    st.from = taker ? src : -1;
    return st;
}

// Scenes with a mesh that has no wide form (boxes that do not nest, or a walk
// that could have too many nodes waiting) walk every mesh's binary BVH in the
// same loops, one pair of children and their exact boxes per step (WIDE false).
// The 1080p frame of the 81,920- and 130,050-triangle meshes with one box of
// each outside its parent's: 1.32 ms, against 1.15 with the wide form and 3.24
// when such rays were traced whole.  A walk's references are then nodes: of an
// inner one the first child, of a leaf kWideLeaf | itself.
SLIM_D uint32_t binary_child(uint32_t node_offset, uint32_t i, float4 b) {
    return node_leaf_count(b) ? kWideLeaf | i : node_offset + node_first(b);
}
// Children i and i + 1 of an inner node against the ray, as wide_hits but exactly.
SLIM_D uint32_t binary_hits(const DevScene &S, uint32_t node_offset, uint32_t i, const Ray &r, float tmax,
                            uint32_t child[2], float t0[2], float t1[2]) {
    uint32_t hits = 0;
#pragma unroll
    for (uint32_t s = 0; s < 2; s++) {
        float4 a, b;
        load_node(S.mesh_nodes, i + s, a, b);
        child[s] = binary_child(node_offset, i + s, b);
        if (hit_node(r, a, b, t0[s], t1[s]) && t0[s] < tmax) hits |= 1u << s;
    }
    return hits;
}

// The hot record of triangle i of a leaf whose first triangle is `first`:
// the first two lie in a wide leaf's own line.
template <bool WIDE>
SLIM_D const float4 *leaf_triangle(const DevScene &S, const float4 *leaf, uint32_t first, uint32_t i) {
    return WIDE && i < 2 ? leaf + 2 + 3 * i : S.tri_hot + 3 * (size_t)(first + i);
}

// MeshTracer::hitTriangles (mesh_tracer.h:23-49) over a wide leaf, any hit
// closer than `closest`.
template <bool COUNT, bool WIDE>
SLIM_D bool any_triangle(const DevScene &S, const float4 *leaf, uint32_t tri_offset, float4 node, float closest,
                         const Ray &r, Work &w) {
    const uint32_t count = node_leaf_count(node), first = tri_offset + node_first(node);
    for (uint32_t i = 0; i < count; i++) {
        bump<COUNT>(w.triangles);
        const float4 *t4 = leaf_triangle<WIDE>(S, leaf, first, i);
        const float4 a = __ldg(t4), b = __ldg(t4 + 1), c = __ldg(t4 + 2);
        const float3 p = xyz(a), n = f3(a.w, b.x, b.y);
        float t; float3 pos; bool behind;
        if (!hit_plane(r, p, n, t, pos, behind)) continue;
        const float3 q = pos - p;
        const float ux = b.z * q.x + c.x * q.y + c.z * q.z;
        const float uy = b.w * q.x + c.y * q.y + c.w * q.z;
        if (!(ux < 0 || uy < 0 || (ux + uy) > 1 || t >= closest)) return true;
    }
    return false;
}

template <bool COUNT, bool WIDE>
__global__ void __launch_bounds__(kMeshBlock, SLIM_SHADOW_MESH_BLOCKS) k_shadow_mesh(DevScene S, DevFrame F, QueueArgs A) {
    chain_wait();
    Feed feed(min(*A.pair_count, A.pair_capacity));
    uint32_t stack[kStackCapacity];
    Work w = {};
    bool busy = false, hit = false;
    uint32_t idx = 0, tag = 0, top = 0, bottom = 0, tri_offset = 0, node_offset = 0;
    uint32_t next = kNone;          // node or leaf the walk goes to
    uint32_t waiting = kNone;       // a leaf to be tested
    float aux = 0.0f;
    Ray r;
    WideRay wr;
    // Where the walk goes after a node or a leaf: a leaf waits while the walk
    // goes on, so that `next` is a leaf only while another one waits.
    auto advance = [&]() {
        if (next == kNone && top > bottom) next = stack[--top];
        if (next != kNone && (next & kWideLeaf) && waiting == kNone) {
            waiting = next;
            next = top > bottom ? stack[--top] : kNone;
        }
    };
    // (shadow ray, instance) pair i from its root, or from a node of its walk
    auto start = [&](uint32_t i, uint32_t from) {
        const float4 *p = A.pairs + 3 * (size_t)i;
        float4 p0 = p[0], p1 = p[1], p2 = p[2];
        tag = __float_as_uint(p1.w);
        if ((A.masks[tag >> 6] >> (tag & 63u)) & 1ull) return;   // already known occluded
        idx = i;
        reset(r, xyz(p0), xyz(p1));
        if constexpr (WIDE) wr = wide_setup(r, p2.z);
        else node_offset = __float_as_uint(p2.z);
        aux = p0.w;
        tri_offset = __float_as_uint(p2.y);
        next = from == kNone ? __float_as_uint(p2.x) : from;
        top = bottom = 0;
        waiting = kNone;
        busy = true;
        advance();
    };
    for (;;) {
        // an occluded ray ends its other parts and pairs in this warp too
        // (8 bounces 2.150 -> 2.139 ms)
        for (uint32_t hits = __ballot_sync(0xFFFFFFFFu, hit); hits; hits &= hits - 1u) {
            const uint32_t occluded = __shfl_sync(0xFFFFFFFFu, tag, __ffs((int)hits) - 1);     // every lane takes part
            if (busy && tag == occluded) {
                busy = false;
                next = waiting = kNone;
                top = bottom = 0;
            }
        }
        hit = false;
        const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !busy);
        if (idle) {
            const uint32_t donors = feed.donors(busy && top > bottom);
            if (feed.fetch(idle, donors)) {
                const uint32_t i = feed.take(A.pair_cursor, idle);
                if (i < feed.n) start(i, kNone);
            } else if (donors) {
                const Steal st = steal_round<false>(idle, donors, stack, bottom, top);
                const uint32_t from_idx = __shfl_sync(0xFFFFFFFFu, idx, st.from >= 0 ? st.from : (int)lane_id());
                if (st.from >= 0) start(from_idx, st.subtree);
            } else if (feed.drained && idle == 0xFFFFFFFFu) {
                break;
            }
        }
#pragma unroll
        for (uint32_t sub = 0; sub < kStepsPerTurn; sub++) {
            if (busy && !(next & kWideLeaf)) {
                // One node of the any-hit walk: the hit child that reaches
                // furthest is next (a shadow ray's occluder is rarely the
                // surface it starts on), the others go on the stack.
                constexpr int kChildren = WIDE ? 4 : 2;
                uint32_t c[kChildren], hits;
                float t0[kChildren], t1[kChildren];
                if constexpr (WIDE) hits = wide_hits(S.wide_nodes, next, r, wr, aux, c, t0, t1);
                else hits = binary_hits(S, node_offset, next, r, aux, c, t0, t1);
                bump<COUNT>(w.mesh_nodes, kChildren);
                next = kNone;
                float reach = -1.0f;
#pragma unroll
                for (int s = 0; s < kChildren; s++)
                    if (hits >> s & 1u) {
                        const bool further = t1[s] > reach;
                        const uint32_t other = further ? next : c[s];
                        next = further ? c[s] : next;
                        reach = further ? t1[s] : reach;
                        if (other != kNone) stack[top++] = other;
                    }
                advance();
            }
        }
        if (leaf_round(waiting != kNone, busy && !(next & kWideLeaf)) && waiting != kNone) {
            const float4 *leaf = WIDE ? S.wide_leaves + 8 * (size_t)(waiting & ~kWideLeaf)
                                      : S.mesh_nodes + 2 * (size_t)(waiting & ~kWideLeaf);
            float4 a, b;
            load_node(leaf, 0, a, b);
            float ln, lf;
            waiting = kNone;
            if ((WIDE ? wide_leaf_box(r, wr, a, b, ln, lf) : hit_node(r, a, b, ln, lf)) && ln < aux &&
                any_triangle<COUNT, WIDE>(S, leaf, tri_offset, b, minr(lf, aux), r, w)) {
                atomicOr(A.masks + (tag >> 6), 1ull << (tag & 63u));
                hit = true;
                next = kNone;
                top = bottom = 0;
            }
            advance();
        }
        if (busy && next == kNone && waiting == kNone && top == bottom) busy = false;
    }
    flush_stage<COUNT>(A.counters, w);
}

// ---- extend, split: closest hit as scene candidates + a persistent mesh pass
//
// The closest hit the reference's SceneTracer::trace finds is the candidate
// with the smallest distance, ties going to the one it visits first: a later
// candidate replaces the current hit only when strictly closer
// (scene_tracer.h:129, mesh_tracer.h:37).  Culling by the current distance
// only skips candidates that cannot win, and a mesh walk started with a
// larger incoming distance finds a superset of hits in the same visiting
// order.  So the search splits exactly:
//   extend_scene   walks the scene BVH in the reference's order, numbering
//                  every geometry it visits (k), tests implicit primitives on
//                  the spot (culling by the best implicit hit so far) and
//                  appends one candidate per reached mesh instance;
//   extend_mesh    a persistent kernel: every lane walks one candidate at a
//                  time over the four-wide BVH, nearest child first, and
//                  fetches the next when its walk ends; finished candidates
//                  publish (distance, k) with a 64-bit atomicMin per ray;
//   extend_resolve the candidate whose (distance, k) is the ray's minimum
//                  writes the hit record.
// The candidates' walks end in any order, and within a mesh the walk visits
// leaves in another order than the reference, which keeps the first of two hits
// at the same distance and skips a leaf whose box begins at or beyond the
// current hit.  A hit beyond the near distances of the boxes above it is reached
// whatever was hit before, so the nearest hit is the reference's unless another
// -- of the same walk, of another candidate, or the best implicit one -- lies at
// the same distance or between it and those near distances (rounding can put
// these behind the hit).  A hit's key therefore says how far beyond it other
// hits matter; they are not culled, and such a ray is traced whole
// (k_extend_overflow; none in the 1080p mesh frames of 2 and 8 bounces).
// Few walks are shared like the any-hit ones (a loop of its own, without the
// sharing's cost for large launches, whose ends the other rays' walks cover):
// a part culls by the ray's published distance and, if its hit is still the
// ray's nearest when it ends, appends a record of its own; one whose hit is not,
// but in the held hit's reach, leaves the ray undecided, as do parts with hits
// at the same distance or with a hit that is not beyond its box's near distance.
// Candidate records (4 float4): (local origin, clip) (local direction, slot)
// (walk_record) (geometry, mesh, k, -near), near being the near distance of the
// boxes above the mesh; a walk that ends with a hit overwrites the third with
// (t, u, v, triangle | behind << 31) and the last word with the hit's own near
// distance, sign clear.  The ray keys live in the shadow-mask array, which is
// free until the shadow stage.

// A hit's key: its distance, its candidate's number (at most 2^24) and, in the
// low five bits, how far beyond the distance other hits matter: up to `near`,
// the near distance of the boxes above it, rounded up to 2^bits - 1 units in
// the last place (0: not beyond; at most 2^29, a factor of 2^64).
SLIM_D unsigned long long hit_key(float t, float near, uint32_t k) {
    const uint32_t beyond = __float_as_uint(maxr(t, near)) - __float_as_uint(t);
    return ((unsigned long long)__float_as_uint(t) << 32) | (k << 5) | min(32u - (uint32_t)__clz((int)beyond), 29u);
}
SLIM_D float key_distance(unsigned long long key) { return __uint_as_float((uint32_t)(key >> 32)); }
SLIM_D float key_reach(unsigned long long key) {
    uint32_t beyond;                // 2^bits - 1; the width wraps to its low five bits
    asm("bmsk.wrap.b32 %0, 0, %1;" : "=r"(beyond) : "r"((uint32_t)key));
    return __uint_as_float((uint32_t)(key >> 32) + beyond);
}
// No hit yet: distance +inf.
constexpr unsigned long long kNoHitKey = (0x7F800000ull << 32) | 0xFFFFFFE0ull;

template <bool COUNT, bool BATCH>
__global__ void __launch_bounds__(256, 2) k_extend_scene(DevScene S0, DevFrame F0, QueueArgs A) {
    chain_wait();
    uint32_t n = queue_size(A);
    uint32_t stack[kStackCapacity];
    uint32_t err = 0;
    Work w = {};
    const uint32_t cap = A.pair_capacity * 3u / 4u;
    uint32_t *overflow = reinterpret_cast<uint32_t *>(A.shadow_rays);   // free until shadow_gen
    for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < n; slot += gridDim.x * blockDim.x) {
        float3 o, d;
        uint32_t path, pid;
        load_ray(F0, A, slot, o, d, path, pid);
        if (!A.rays_in) bump<COUNT>(w.primary);
        const DevScene &S = scene_of<BATCH>(S0, A, pid);
        Ray r;
        reset(r, scale_add(d, kTraceOffset, o), d);
        Hit hit;
        hit.distance = INFINITY;
        int best_geo = -1;
        uint32_t best_k = 0, k = 0;
        float best_near = 0.0f;         // near distance of the boxes above the best implicit hit
        bool full = false;
        // A visible mesh instance of a leaf with near and far distances ln, lf:
        // a candidate, or a single-leaf mesh's triangles here.
        auto instance = [&](uint32_t gi, const Geo &g, float ln, float lf, Nearest *seen) {
            const float clip = lf + kEps;
            Ray local;
            bump<COUNT>(w.geometries);
            localize(local, r.o, r.d, g);
            const DevMesh &m = S.meshes[g.mesh];
            float bn, bf;
            if (!hit_aabb(local, m.aabb_min[0], m.aabb_min[1], m.aabb_min[2], m.aabb_max[0], m.aabb_max[1],
                          m.aabb_max[2], bn, bf))
                return;
            const float4 *nodes = S.mesh_nodes + 2 * (size_t)m.node_offset;
            float4 ra, rb;
            float rn, rf;
            load_node(nodes, 0, ra, rb);
            bump<COUNT>(w.mesh_nodes);
            // the root test with the largest distance the reference could have used:
            // in its order the best implicit hit so far's; out of it a hit just
            // in front of the root's box may count too
            const float reach = seen ? seen->reach(hit.distance) * kReachSlack + slab_margin(local) : hit.distance;
            if (!(hit_node(local, ra, rb, rn, rf) && rn < clip && rn <= reach)) return;
            if (node_leaf_count(rb)) {
                // a single-leaf mesh (mesh_tracer.h:66-70): its triangles here
                Hit mh;
                mh.distance = clip;
                if (hit_triangles<COUNT>(S.tri_hot, m.tri_offset, m.tri_count, rf, local, mh, false, w) &&
                    (seen ? seen->take(mh.distance, maxr(ln, rn), hit.distance) : mh.distance < hit.distance)) {
                    mh.uv_coverage = __ldg(&S.tri_cold[4 * (size_t)(m.tri_offset + mh.id) + 3].w);
                    best_geo = (int)gi;
                    best_k = k;
                    best_near = maxr(ln, rn);
                    hit = mh;
                    hit.NdotRd = -(dot(hit.normal, local.d));
                }
                return;
            }
            const bool queued = S.binary_walks || m.wide_root != kNoWideBVH;
            uint32_t q = warp_append(A.pair_count, queued);
            if (!queued || q >= cap) { full = true; return; }
            float4 *p = A.pairs + 4 * (size_t)q;
            p[0] = make_float4(local.o.x, local.o.y, local.o.z, clip);
            p[1] = make_float4(local.d.x, local.d.y, local.d.z, __uint_as_float(slot));
            p[2] = walk_record(S, m, rb);
            p[3] = make_float4(__uint_as_float(gi), __uint_as_float(g.mesh), __uint_as_float(k),
                               copysignf(maxr(ln, rn), -1.0f));
        };
        // one scene leaf: [first, first + count) geometries, near and far distances ln, lf
        auto leaf = [&](uint32_t first, uint32_t count, float ln, float lf) {
            Hit aux;
            aux.distance = minr(lf + kEps, hit.distance);
            Ray local;
            for (uint32_t i = 0; i < count; i++, k++) {
                uint32_t gi = __ldg(S.leaf_geometry + first + i);
                Geo g = load_geo(S, gi);
                if (!(g.flags & SLIM_GEOMETRY_IS_VISIBLE)) continue;
                if (g.type == SLIM_GEOMETRY_MESH) {
                    instance(gi, g, ln, lf, nullptr);
                } else if (hit_geometry_local<COUNT>(S, g, r, local, aux, false, nullptr, err, w) &&
                           aux.distance < hit.distance) {
                    best_geo = (int)gi;
                    best_k = k;
                    best_near = ln;
                    hit = aux;
                    hit.NdotRd = -(dot(hit.normal, local.d));
                }
            }
        };
        // Small scenes: every leaf's box, then the implicit primitives of the
        // hit ones, then their mesh instances, the best implicit hit already
        // known.  Candidates are numbered in that order from 1; an implicit hit
        // has 0.
        const uint4 list = COUNT ? make_uint4(0, 0, 0, 0) : listed_leaves(S, n);
        if (!COUNT && list.x && finite_ray(r)) {
            const uint32_t leaves = leaves_hit(S, list.x, r, INFINITY, list.y | list.z);
            Nearest seen;
            best_geo = closest_of_leaves<COUNT>(S, leaves & list.y, r, hit, seen, err, w);
            for (uint32_t rest = leaves & list.z; rest && !seen.unsure; rest &= rest - 1u) {
                float4 a, b;
                float ln, lf;
                load_leaf(S, __ffs((int)rest) - 1, a, b);
                hit_box_finite(r, a, b, ln, lf);
                if (ln > seen.reach(hit.distance) * kReachSlack + slab_margin(r)) continue;
                const uint32_t first = node_first(b), count = node_leaf_count(b);
                for (uint32_t i = 0; i < count; i++) {
                    const uint32_t gi = __ldg(S.leaf_geometry + first + i);
                    const Geo g = load_geo(S, gi);
                    if (!(g.flags & SLIM_GEOMETRY_IS_VISIBLE) || g.type != SLIM_GEOMETRY_MESH) continue;
                    k++;
                    instance(gi, g, ln, lf, &seen);
                }
            }
            best_k = 0;
            best_near = seen.near;
            full |= seen.unsure;
        } else {
        float ln, rn, lf, rf;
        float4 a, b;
        load_node(S.scene_nodes, 0, a, b);
        bump<COUNT>(w.scene_nodes);
        if (hit_node(r, a, b, ln, lf) && ln < hit.distance) {
            if (node_leaf_count(b)) {
                leaf(0, S.geometry_count, ln, lf);
            } else {
                uint32_t left = node_first(b), top = 0;
                for (;;) {
                    float4 la, lb, xa, xb;
                    load_node(S.scene_nodes, left, la, lb);
                    load_node(S.scene_nodes, left + 1, xa, xb);
                    bump<COUNT>(w.scene_nodes, 2);
                    bool hl = hit_node(r, la, lb, ln, lf) && ln < hit.distance;
                    bool hr = hit_node(r, xa, xb, rn, rf) && rn < hit.distance;
                    uint32_t lchild = node_first(lb), rchild = node_first(xb);
                    bool go_left = hl, go_right = hr;
                    if (hl && node_leaf_count(lb)) {
                        leaf(lchild, node_leaf_count(lb), ln, lf);
                        go_left = false;
                    }
                    if (hr && node_leaf_count(xb)) {
                        leaf(rchild, node_leaf_count(xb), rn, rf);
                        go_right = false;
                    }
                    if (go_left) {
                        if (go_right) {
                            if (ln > rn) { uint32_t t = lchild; lchild = rchild; rchild = t; }
                            if (top >= (uint32_t)kStackCapacity) { err |= kErrStack; break; }
                            stack[top++] = rchild;
                        }
                        left = lchild;
                    } else if (go_right) {
                        left = rchild;
                    } else {
                        if (top == 0) break;
                        left = stack[--top];
                    }
                }
            }
        }
        }
        if (full) {
            // the candidate queue ran out, or the order of the tests decides:
            // the ray is traced whole afterwards
            // (k_extend_overflow); key 0 matches no candidate (hit distances
            // are never 0: the plane test rejects an origin on the plane)
            A.masks[slot] = 0ull;
            overflow[atomicAdd(A.pair_count + 2, 1u)] = slot;
        } else {
            A.masks[slot] = best_geo >= 0 ? hit_key(hit.distance, best_near, best_k) : kNoHitKey;
            store_hit(A.hits, A.hit_stride, slot, best_geo, hit);
        }
    }
    if (err) atomicOr(F0.error_flags, err);
    flush_stage<COUNT>(A.counters, w);
}

// Rays whose candidates did not fit, or whose mesh walk left the nearest hit
// undecided: the reference's whole closest-hit walk.
template <bool COUNT, bool BATCH>
__global__ void __launch_bounds__(256) k_extend_overflow(DevScene S0, DevFrame F0, QueueArgs A) {
    chain_wait();
    const uint32_t n = A.pair_count[2];
    const uint32_t *overflow = reinterpret_cast<const uint32_t *>(A.shadow_rays);
    uint32_t stack[kStackCapacity], mesh_stack[kStackCapacity];
    uint32_t err = 0;
    Work w = {};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t slot = overflow[i];
        float3 o, d;
        uint32_t path, pid;
        load_ray(F0, A, slot, o, d, path, pid);
        const DevScene &S = scene_of<BATCH>(S0, A, pid);
        Ray ray;
        reset(ray, o, d);
        Hit hit;
        int g = scene_trace<COUNT>(S, n, ray, hit, false, INFINITY, stack, mesh_stack, err, w);
        store_hit(A.hits, A.hit_stride, slot, g, hit);
    }
    if (err) atomicOr(F0.error_flags, err);
    flush_stage<COUNT>(A.counters, w);
}

template <bool COUNT, bool SHARE, bool WIDE>
SLIM_D void extend_walks(const DevScene &S, const QueueArgs &A, Feed &feed, uint32_t cap) {
    uint2 stack[kStackCapacity];    // (node or leaf, its near distance)
    Work w = {};
    bool busy = false;
    uint32_t idx = 0, slot = 0, top = 0, bottom = 0, tri_offset = 0, node_offset = 0, tri = 0, k = 0;
    uint32_t next = kNone, waiting = kNone;
    float lc = 0.0f, lc_near = 0.0f, box_near = 0.0f, reach = 0.0f, bu = 0.0f, bv = 0.0f;
    bool found = false, behind = false, unsure = false;
    bool piece = false, shared = false;     // part of another lane's walk; a walk that gave parts away
    // Binary boxes need not nest: near distances of `next` and `waiting` are
    // then the largest of the boxes on the way there, and `margin` is the slab
    // test's rounding, which wide boxes have in them.
    float next_near = 0.0f, waiting_near = 0.0f, margin = 0.0f;
    Ray r;
    WideRay wr;
    auto slack = [&](float t) {
        if constexpr (WIDE) return t * kReachSlack;
        else return t * kReachSlack + margin;
    };
    // the nearest waiting entry that can still hold a closer hit
    auto pop = [&]() -> uint32_t {
        while (top > bottom) {
            const uint2 e = stack[--top];
            if (__uint_as_float(e.y) <= reach) {
                if (!WIDE) next_near = __uint_as_float(e.y);
                return e.x;
            }
        }
        return kNone;
    };
    auto advance = [&]() {          // as in k_shadow_mesh
        if (next == kNone) next = pop();
        if (next != kNone && (next & kWideLeaf) && waiting == kNone) {
            waiting = next;
            if (!WIDE) waiting_near = next_near;
            next = pop();
        }
    };
    // the ray's other candidates and, of a shared walk, its other parts cull by
    // the published distance; two with the same leave the ray undecided
    auto key = [&]() { return hit_key(lc, maxr(lc_near, box_near), k); };
    auto publish = [&]() { unsure |= key_distance(atomicMin(A.masks + slot, key())) == lc; };
    // candidate i from its root, or from a node of its walk
    auto start = [&](uint32_t i, uint32_t from, float near) {
        const float4 *p = A.pairs + 4 * (size_t)i;
        const float4 p0 = p[0], p1 = p[1], p3 = p[3];
        float4 p2 = p[2];
        piece = shared = SHARE && from != kNone;
        if (piece) {        // the walk's own result may have taken the place of its mesh
            const DevMesh &m = S.meshes[__float_as_uint(p3.y)];
            p2 = make_float4(__uint_as_float(from), __uint_as_float(m.tri_offset),
                             WIDE ? m.wide_extent : __uint_as_float(m.node_offset), 0.0f);
        }
        idx = i;
        reset(r, xyz(p0), xyz(p1));
        if constexpr (WIDE) {
            wr = wide_setup(r, p2.z);
        } else {
            node_offset = __float_as_uint(p2.z);
            margin = slab_margin(r);
            next_near = near;
        }
        lc = lc_near = p0.w;
        box_near = fabsf(p3.w);
        slot = __float_as_uint(p1.w);
        k = __float_as_uint(p3.z);
        reach = slack(fminf(lc, key_reach(A.masks[slot])));
        next = __float_as_uint(p2.x);
        waiting = kNone;
        tri_offset = __float_as_uint(p2.y);
        top = bottom = 0;
        found = unsure = false;
        busy = true;
        advance();
    };
    for (;;) {
        if constexpr (!SHARE) {
            const bool fetch = fetch_round(!busy);
            if (!busy && fetch) {
                uint32_t active = __activemask();
                int leader = __ffs(active) - 1;
                uint32_t base = 0;
                if ((int)lane_id() == leader) base = atomicAdd(A.pair_cursor, (uint32_t)__popc(active));
                base = __shfl_sync(active, base, leader);
                const uint32_t i = base + (uint32_t)__popc(active & ((1u << lane_id()) - 1u));
                if (i >= feed.n) break;
                start(i, kNone, 0.0f);
            }
        } else {
            const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !busy);
            if (idle) {
                const uint32_t donors = feed.donors(busy && top > bottom);
                if (feed.fetch(idle, donors)) {
                    const uint32_t i = feed.take(A.pair_cursor, idle);
                    if (i < feed.n) start(i, kNone, 0.0f);
                } else if (donors) {
                    const Steal st = steal_round<!WIDE>(idle, donors, stack, bottom, top);
                    if (st.gave) {
                        // a hit at or before its own box's near distance is sure
                        // only against hits of the same lane
                        unsure |= found && lc_near > lc;
                        if (found && !shared) publish();
                        shared = true;
                    }
                    const uint32_t from_idx = __shfl_sync(0xFFFFFFFFu, idx, st.from >= 0 ? st.from : (int)lane_id());
                    if (st.from >= 0) start(from_idx, st.subtree, __uint_as_float(st.near));
                } else if (feed.drained && idle == 0xFFFFFFFFu) {
                    break;
                }
            }
        }
        // lanes that took a branch above or below come together before the next
        // (8 bounces 2.05 -> 1.97 ms)
        if (SHARE) __syncwarp();
#pragma unroll
        for (uint32_t sub = 0; sub < kStepsPerTurn; sub++) if (busy && !(next & kWideLeaf)) {
            constexpr int kChildren = WIDE ? 4 : 2;
            uint32_t c[kChildren], hits;
            float t0[kChildren], t1[kChildren];
            if constexpr (WIDE) {
                hits = wide_hits(S.wide_nodes, next, r, wr, reach, c, t0, t1);
            } else {
                hits = binary_hits(S, node_offset, next, r, reach, c, t0, t1);
                for (float &t : t0) t = maxr(t, next_near);
            }
            bump<COUNT>(w.mesh_nodes, kChildren);
            // the nearest hit child is next, the others go on the stack
            float near = INFINITY;
            next = kNone;
#pragma unroll
            for (int s = 0; s < kChildren; s++)
                if (hits >> s & 1u) {
                    const bool nearer = t0[s] < near;
                    const uint32_t other = nearer ? next : c[s];
                    const float far = nearer ? near : t0[s];
                    next = nearer ? c[s] : next;
                    near = nearer ? t0[s] : near;
                    if (other != kNone) stack[top++] = make_uint2(other, __float_as_uint(far));
                }
            if (!WIDE) next_near = near;
            advance();
        }
        if (SHARE) __syncwarp();
        if (leaf_round(waiting != kNone, busy && !(next & kWideLeaf)) && waiting != kNone) {
            // MeshTracer::hitTriangles (mesh_tracer.h:23-49) with the leaf's far clip
            const float4 *leaf = WIDE ? S.wide_leaves + 8 * (size_t)(waiting & ~kWideLeaf)
                                      : S.mesh_nodes + 2 * (size_t)(waiting & ~kWideLeaf);
            float4 na, nb;
            load_node(leaf, 0, na, nb);
            float ln, lf;
            waiting = kNone;
            if (WIDE ? wide_leaf_box(r, wr, na, nb, ln, lf) : hit_node(r, na, nb, ln, lf)) {
                if (!WIDE) ln = maxr(ln, waiting_near);
                const float gb = key_reach(A.masks[slot]);
                const float before = lc;
                const uint32_t count = node_leaf_count(nb), first = node_first(nb);
                for (uint32_t i = 0; i < count; i++) {
                    bump<COUNT>(w.triangles);
                    const float4 *t4 = leaf_triangle<WIDE>(S, leaf, tri_offset + first, i);
                    float4 a = __ldg(t4), b = __ldg(t4 + 1), c = __ldg(t4 + 2);
                    float3 pp = xyz(a), nn = f3(a.w, b.x, b.y);
                    float tt; float3 pos; bool bh;
                    if (!hit_plane(r, pp, nn, tt, pos, bh)) continue;
                    float3 q = pos - pp;
                    float ux = b.z * q.x + c.x * q.y + c.z * q.z;
                    float uy = b.w * q.x + c.y * q.y + c.w * q.z;
                    if (ux < 0 || uy < 0 || (ux + uy) > 1 || tt >= lf || tt > gb) continue;
                    if (tt >= lc) {
                        unsure |= found && tt <= lc_near;
                        continue;
                    }
                    unsure |= (found && lc <= ln) || (shared && tt <= ln);
                    lc = tt;
                    lc_near = maxr(ln, tt);
                    bu = ux;
                    bv = uy;
                    behind = bh;
                    tri = first + i;
                    found = true;
                }
                if (SHARE && shared && lc < before) publish();
                reach = slack(fminf(lc_near, gb));
            }
            advance();
        }
        if (SHARE) __syncwarp();
        if (busy && next == kNone && waiting == kNone && top == bottom) {
            float4 *p = A.pairs + 4 * (size_t)idx;
            const float4 result = make_float4(lc, bu, bv, __uint_as_float(tri | ((uint32_t)behind << 31)));
            if (!SHARE || !shared) {
                // publishes and waits for no answer (waiting: 225 -> 284 us for the first round's launch)
                if (found && !unsure) {
                    p[2] = result;
                    p[3].w = maxr(lc_near, box_near);
                    atomicMin(A.masks + slot, key());
                }
            } else if (found && !unsure) {
                const unsigned long long held = __ldcg(A.masks + slot);
                const bool best = held == key();
                // not the nearest, but where the order of the visits decides
                unsure = !best && held && lc <= key_reach(held);
                uint32_t record = idx;
                if (best && piece) {
                    // a part's hit gets a record of its own behind the candidates
                    record = feed.n + atomicAdd(A.pair_count + 3, 1u);
                    unsure = record >= cap;
                }
                if (best && !unsure) {
                    float4 *o = A.pairs + 4 * (size_t)record;
                    const float4 p1 = p[1], p3 = p[3];
                    if (piece) o[1] = p1;
                    o[2] = result;
                    o[3] = make_float4(p3.x, p3.y, p3.z, maxr(lc_near, box_near));
                }
            }
            // two hits so close together that the order of the visits decides
            // between them: the ray is traced whole, once, in the reference's
            // order (k_extend_overflow)
            if (unsure && atomicMin(A.masks + slot, 0ull))
                reinterpret_cast<uint32_t *>(A.shadow_rays)[atomicAdd(A.pair_count + 2, 1u)] = slot;
            busy = false;
        }
    }
    flush_stage<COUNT>(A.counters, w);
}

template <bool COUNT, bool WIDE>
__global__ void __launch_bounds__(kMeshBlock, SLIM_EXTEND_MESH_BLOCKS) k_extend_mesh(DevScene S, DevFrame F, QueueArgs A) {
    chain_wait();
    const uint32_t cap = A.pair_capacity * 3u / 4u;
    Feed feed(min(*A.pair_count, cap));
    if (feed.sparse()) extend_walks<COUNT, true, WIDE>(S, A, feed, cap);
    else extend_walks<COUNT, false, WIDE>(S, A, feed, cap);
}

// The candidate holding its ray's minimum (distance, k) writes the hit
// record with the attributes MeshTracer::trace fills in.
template <bool COUNT, bool BATCH>
__global__ void __launch_bounds__(256) k_extend_resolve(DevScene S0, DevFrame F0, QueueArgs A) {
    chain_wait();
    const uint32_t cap = A.pair_capacity * 3u / 4u;
    const uint32_t n = min(min(*A.pair_count, cap) + A.pair_count[3], cap);
    Work w = {};
    for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += gridDim.x * blockDim.x) {
        const float4 *p = A.pairs + 4 * (size_t)idx;
        const float4 p3 = p[3];
        if (signbit(p3.w)) continue;
        const float4 p1 = p[1], p2 = p[2];
        const uint32_t slot = __float_as_uint(p1.w);
        const unsigned long long best = A.masks[slot];
        const bool winner = best == hit_key(p2.x, p3.w, __float_as_uint(p3.z));
        // the hit that is not the nearest: another candidate's here, or the best
        // implicit one
        float other = p2.x;
        if (winner) {
            other = INFINITY;
            if ((best & 31u) && __float_as_int(A.hits[2 * (size_t)A.hit_stride + slot].x) >= 0) other = A.hits[slot].w;
        }
        if (best && other <= key_reach(best) && other < INFINITY) {
            // so close to the nearest that the order of the visits decides
            if (atomicExch(A.masks + slot, 0ull))
                reinterpret_cast<uint32_t *>(A.shadow_rays)[atomicAdd(A.pair_count + 2, 1u)] = slot;
            continue;
        }
        if (!winner) continue;
        uint32_t pid = 0;
        if (BATCH) pid = __float_as_uint(A.rays_in[2 * (size_t)slot + 1].w);
        const DevScene &S = scene_of<BATCH>(S0, A, pid);
        const DevMesh &m = S.meshes[__float_as_uint(p3.y)];
        Hit h;
        h.distance = p2.x;
        h.u = p2.y;
        h.v = p2.z;
        const uint32_t tb = __float_as_uint(p2.w);
        h.id = tb & 0x7FFFFFFFu;
        h.from_behind = (tb >> 31) != 0;
        const float4 *t4 = S.tri_hot + 3 * (size_t)(m.tri_offset + h.id);
        const float4 a = __ldg(t4), b = __ldg(t4 + 1);
        h.normal = f3(a.w, b.x, b.y);
        h.position = f3(0, 0, 0);
        mesh_hit_attributes<COUNT>(S, m, h, w);
        h.NdotRd = -(dot(h.normal, xyz(p1)));
        store_hit(A.hits, A.hit_stride, slot, (int)__float_as_uint(p3.x), h);
    }
    flush_stage<COUNT>(A.counters, w);
}

// ---- fused tail: the rest of every queued path in one thread ------------------
//
// Late rounds hold few paths whose traversals are long, so each round's
// kernels wait on a handful of slow rays and the frame pays that wait once
// per remaining bounce.  From the tail depth on, one kernel walks every
// remaining path to its end -- the reference's per-pixel loop
// (ray_tracer.h:42-107) from the queued ray on, closest hits and shadow rays
// traced inline -- so the wait is paid once.  Per path the arithmetic is
// k_extend / k_shade's, in the same order: the frame is unchanged.
template <bool COUNT, bool BATCH>
__global__ void __launch_bounds__(128) k_finish_paths(DevScene S0, DevFrame F0, QueueArgs A) {
    chain_wait();
    const uint32_t n = queue_size(A);
    uint32_t stack[kStackCapacity], mesh_stack[kStackCapacity];
    uint32_t err = 0;
    Work w = {};
    for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < n; slot += gridDim.x * blockDim.x) {
        float3 o, d;
        uint32_t path, pid;
        load_ray(F0, A, slot, o, d, path, pid);
        const DevScene &S = scene_of<BATCH>(S0, A, pid);
        const DevFrame &F = frame_of<BATCH>(F0, A, pid);
        const SlimRayTracerSettings &st = F.settings;
        const float scaling = cone_scaling<BATCH>(F, pid);
        float4 pc = A.path_color[path];
        float3 color = xyz(pc), throughput = xyz(A.path_throughput[path]);
        const float depth = pc.w;
        Ray ray;
        reset(ray, o, d);
        for (uint32_t level = A.depth;; level++) {
            Hit hit;
            float3 current = f3(0, 0, 0), next_throughput = f3(0, 0, 0);
            bool bounce = false;
            int g = scene_trace<COUNT>(S, n, ray, hit, false, INFINITY, stack, mesh_stack, err, w);
            float hit_distance = INFINITY;
            if (g >= 0) {
                hit_distance = hit.distance;
                Geo geo = load_geo(S, (uint32_t)g);
                Mat m = load_mat(S, geo.material);
                if ((m.flags & SLIM_MATERIAL_IS_EMISSIVE) && geo.type == SLIM_GEOMETRY_QUAD && !hit.from_behind) {
                    current = m.emission;
                } else {
                    Surface s;
                    prepare_for_shading<COUNT>(S, geo, m, ray, hit, scaling, s, w);
                    hit_distance = hit.distance;
                    for (uint32_t i = 0; i < S.light_count; i++) {
                        LightRec l = load_light(S, i);
                        if (!is_facing_light(s, l)) continue;
                        if (l.flags & SLIM_LIGHT_IS_SHADOWING) {
                            Ray sr;
                            sr.o = s.P;
                            sr.d = s.L;
                            Hit sh;
                            bump<COUNT>(w.shadow);
                            if (scene_trace<COUNT>(S, n, sr, sh, true, s.Ld, stack, mesh_stack, err, w) >= 0) continue;
                        }
                        add_light(s, m, l, current);
                    }
                    if (S.flags & SLIM_SCENE_HAD_EMISSIVE_QUADS) shade_from_emissive_quads(S, g, s, m, current);
                    if (st.skybox_irradiance_texture_id >= 0 && st.skybox_radiance_texture_id >= 0) {
                        s.L = s.N;
                        s.NdotL = 1.0f;
                        float3 D = texture_sample_cube<COUNT>(S, (uint32_t)st.skybox_irradiance_texture_id, s.N.x, s.N.y, s.N.z, w);
                        float3 Sp = texture_sample_cube<COUNT>(S, (uint32_t)st.skybox_radiance_texture_id, s.R.x, s.R.y, s.R.z, w);
                        radiance_fraction(s, m);
                        current = mul_add(D, s.Fd, mul_add(s.Fs, Sp, current));
                    }
                    if ((m.flags & (SLIM_MATERIAL_IS_REFLECTIVE | SLIM_MATERIAL_IS_REFRACTIVE)) && level < st.max_depth) {
                        float3 Fr = schlick_fresnel(clamp01(dot(s.N, s.R)), m.reflectivity);
                        next_throughput = s.refracted ? one_minus(Fr) : Fr;
                        bounce = true;
                        reset(ray, hit.position, s.RF);
                        bump<COUNT>(w.bounce);
                    }
                }
            } else if (st.skybox_color_texture_id >= 0) {
                current = texture_sample_cube<COUNT>(S, (uint32_t)st.skybox_color_texture_id, ray.d.x, ray.d.y, ray.d.z, w);
            }
            if (level != A.skip_glow_depth) add_glow(S, ray, hit_distance, current);
            color = mul_add(current, throughput, color);
            throughput = throughput * next_throughput;
            if (!bounce) break;
        }
        if (A.sink) A.sink[path] = make_float4(color.x, color.y, color.z, 0.0f);
        else write_pixel<BATCH>(F, pid, color, depth);
    }
    if (err) atomicOr(F0.error_flags, err);
    flush_stage<COUNT>(A.counters, w);
}

// ---- radiance-cache vertex ---------------------------------------------------
// The network's inputs at a shaded surface: position in the scene box mapped
// to [0,1]^3 (longest side, from the scene BVH root), roughness, ray
// direction, shading normal, albedo x albedo map.
SLIM_D void query_features(const DevScene &S, const Mat &m, const Ray &ray, const Surface &s, float4 f[4]) {
    float4 r0 = make_float4(0, 0, 0, 1), r1 = make_float4(1, 1, 0, 0);
    if (S.scene_node_count) { r0 = S.scene_nodes[0]; r1 = S.scene_nodes[1]; }
    const float ext = fmaxf(fmaxf(r0.w - r0.x, r1.x - r0.y), r1.y - r0.z);
    const float inv = ext > 0.0f ? 1.0f / ext : 1.0f;
    float3 p = (s.P - f3(r0.x, r0.y, r0.z)) * inv;
    float3 al = m.albedo * s.albedo_from_map;
    f[0] = make_float4(p.x, p.y, p.z, m.roughness);
    f[1] = make_float4(ray.d.x, ray.d.y, ray.d.z, 0.0f);
    f[2] = make_float4(s.N.x, s.N.y, s.N.z, 0.0f);
    f[3] = make_float4(al.x, al.y, al.z, 0.0f);
}

// The path has reached the vertex the cache answers at.  Misses and emissive
// quads finish it exactly as k_shade does; every other hit turns it into a
// query: the segment's glow is added to the path colour now, the surface's
// features (position in the scene box, roughness, direction, shading normal,
// albedo) go to the network, and the path waits in path_color /
// path_throughput for the answer.  Returns true for a query.
template <bool COUNT, bool BATCH>
SLIM_D bool cache_vertex(const DevScene &S, const DevFrame &F, const QueueArgs &A, uint32_t slot, uint32_t path,
                         uint32_t pid, float3 o, float3 d, float4 f[4], Work &w, float4 &q_color, float4 &q_through) {
    const SlimRayTracerSettings &st = F.settings;
    Ray ray;
    reset(ray, scale_add(d, kTraceOffset, o), d);
    Hit hit;
    int g = load_hit(A.hits, A.hit_stride, slot, hit);
    float4 pc = A.path_color[path];
    float3 color = xyz(pc), throughput = xyz(A.path_throughput[path]);
    float3 current = f3(0, 0, 0);
    float hit_distance = INFINITY;
    bool query = false;
    if (g >= 0) {
        hit_distance = hit.distance;
        Geo geo = load_geo(S, (uint32_t)g);
        Mat m = load_mat(S, geo.material);
        if ((m.flags & SLIM_MATERIAL_IS_EMISSIVE) && geo.type == SLIM_GEOMETRY_QUAD && !hit.from_behind) {
            current = m.emission;
        } else {
            Surface s;
            prepare_for_shading<COUNT>(S, geo, m, ray, hit, cone_scaling<BATCH>(F, pid), s, w);
            hit_distance = hit.distance;
            query = true;
            query_features(S, m, ray, s, f);
        }
    } else if (st.skybox_color_texture_id >= 0) {
        current = texture_sample_cube<COUNT>(S, (uint32_t)st.skybox_color_texture_id, ray.d.x, ray.d.y, ray.d.z, w);
    }
    add_glow(S, ray, hit_distance, current);
    color = mul_add(current, throughput, color);
    q_color = make_float4(color.x, color.y, color.z, pc.w);
    q_through = make_float4(throughput.x, throughput.y, throughput.z, 0.0f);
    if (query) A.path_color[path] = q_color;
    else if (A.sink) A.sink[path] = make_float4(color.x, color.y, color.z, 0.0f);   // a self-training path ends
    else write_pixel<BATCH>(F, pid, color, pc.w);
    return query;
}

// `hits`: the round's hit planes (stride entries each), whose record of
// `slot` the query keeps (null: none kept).
SLIM_D void append_query(const CacheArgs &C, uint32_t q, const float4 f[4], float3 o, float3 d, uint32_t path,
                         uint32_t pid, float4 q_color, float4 q_through, const float4 *hits = nullptr,
                         uint32_t stride = 0, uint32_t slot = 0) {
    if (C.q_hit && hits) {
        float4 *h = C.q_hit + 3 * (size_t)q;
        h[0] = hits[slot]; h[1] = hits[(size_t)stride + slot]; h[2] = hits[2 * (size_t)stride + slot];
    }
    float4 *p = C.features + 4 * (size_t)q;
    p[0] = f[0]; p[1] = f[1]; p[2] = f[2]; p[3] = f[3];
    C.aux[2 * (size_t)q] = make_float4(o.x, o.y, o.z, __uint_as_float(path));
    C.aux[2 * (size_t)q + 1] = make_float4(d.x, d.y, d.z, __uint_as_float(pid));
    if (C.q_color) {
        C.q_color[q] = q_color;
        C.q_through[q] = q_through;
    }
}

// ---- shade: colour of this segment, next bounce, finished paths --------
// Capped at 64 registers (4 blocks per SM): latency-bound, the extra warps pay
// for the spills (mesh 1080p 1.138 ms, textures 1080p 393 us; 3 blocks at 80
// registers 1.143 and 400; 2 at 128 1.146 and 406).
#ifndef SLIM_SHADE_BLOCKS
#define SLIM_SHADE_BLOCKS 4
#endif
template <bool COUNT, bool BATCH>
__global__ void __launch_bounds__(256, SLIM_SHADE_BLOCKS) k_shade(DevScene S0, DevFrame F0, QueueArgs A) {
    chain_wait();
    uint32_t n = queue_size(A);
    if (A.slot_end && A.slot_end < n) n = A.slot_end;
    const uint32_t first = A.slot_begin;
    Work w = {};
    uint32_t stride = gridDim.x * blockDim.x;
    uint32_t rounds = n > first ? (n - first + stride - 1) / stride : 0;
    for (uint32_t r = 0, slot = first + blockIdx.x * blockDim.x + threadIdx.x; r < rounds; r++, slot += stride) {
        bool live = slot < n;
        bool bounce = false, query = false;
        uint32_t path = 0, pid = 0;
        float3 o = f3(0, 0, 0), d = f3(0, 0, 0);
        float3 bo = f3(0, 0, 0), bd = f3(0, 0, 0);
        float4 feat[4], qc = make_float4(0, 0, 0, 0), qt = make_float4(0, 0, 0, 0);
        if (live) {
            load_ray(F0, A, slot, o, d, path, pid);
            const DevScene &S = scene_of<BATCH>(S0, A, pid);
            const DevFrame &F = frame_of<BATCH>(F0, A, pid);
            const SlimRayTracerSettings &st = F.settings;
            if (at_cache_vertex<BATCH>(F, A)) {
                query = cache_vertex<COUNT, BATCH>(S, F, A, slot, path, pid, o, d, feat, w, qc, qt);
            } else {
                Ray ray;
                reset(ray, scale_add(d, kTraceOffset, o), d);
                Hit hit;
                int g = load_hit(A.hits, A.hit_stride, slot, hit);
                float4 pc = A.depth == 1 ? make_float4(0, 0, 0, INFINITY) : A.path_color[path];
                float3 color = xyz(pc), throughput = A.depth == 1 ? f3(1, 1, 1) : xyz(A.path_throughput[path]);
                float depth = pc.w;
                float3 current = f3(0, 0, 0), next_throughput = f3(0, 0, 0);
                float hit_distance = INFINITY;
                if (g >= 0) {
                    hit_distance = hit.distance;
                    Geo geo = load_geo(S, (uint32_t)g);
                    Mat m = load_mat(S, geo.material);
                    if ((m.flags & SLIM_MATERIAL_IS_EMISSIVE) && geo.type == SLIM_GEOMETRY_QUAD && !hit.from_behind) {
                        current = m.emission;
                    } else {
                        Surface s;
                        prepare_for_shading<COUNT>(S, geo, m, ray, hit, cone_scaling<BATCH>(F, pid), s, w);
                        hit_distance = hit.distance;
                        if (A.depth == 1) depth = depth_at(F.projection, hit.position);
                        unsigned long long occluded = A.masks[slot];
                        for (uint32_t i = 0; i < S.light_count; i++) {
                            LightRec l = load_light(S, i);
                            if (!is_facing_light(s, l)) continue;
                            if ((l.flags & SLIM_LIGHT_IS_SHADOWING) && ((occluded >> i) & 1ull)) continue;
                            add_light(s, m, l, current);
                        }
                        if (S.flags & SLIM_SCENE_HAD_EMISSIVE_QUADS) shade_from_emissive_quads(S, g, s, m, current);
                        if (st.skybox_irradiance_texture_id >= 0 && st.skybox_radiance_texture_id >= 0) {
                            s.L = s.N;
                            s.NdotL = 1.0f;
                            float3 D = texture_sample_cube<COUNT>(S, (uint32_t)st.skybox_irradiance_texture_id, s.N.x, s.N.y, s.N.z, w);
                            float3 Sp = texture_sample_cube<COUNT>(S, (uint32_t)st.skybox_radiance_texture_id, s.R.x, s.R.y, s.R.z, w);
                            radiance_fraction(s, m);
                            current = mul_add(D, s.Fd, mul_add(s.Fs, Sp, current));
                        }
                        if ((m.flags & (SLIM_MATERIAL_IS_REFLECTIVE | SLIM_MATERIAL_IS_REFRACTIVE)) && A.depth < st.max_depth) {
                            float3 Fr = schlick_fresnel(clamp01(dot(s.N, s.R)), m.reflectivity);
                            next_throughput = s.refracted ? one_minus(Fr) : Fr;
                            bounce = true;
                            bo = hit.position;
                            bd = s.RF;
                            reset(ray, bo, bd);
                        }
                    }
                } else if (st.skybox_color_texture_id >= 0) {
                    current = texture_sample_cube<COUNT>(S, (uint32_t)st.skybox_color_texture_id, ray.d.x, ray.d.y, ray.d.z, w);
                }
                if (A.depth != A.skip_glow_depth) add_glow(S, ray, hit_distance, current);
                color = mul_add(current, throughput, color);
                throughput = throughput * next_throughput;
                if (bounce) {
                    A.path_color[path] = make_float4(color.x, color.y, color.z, depth);
                    A.path_throughput[path] = make_float4(throughput.x, throughput.y, throughput.z, 0.0f);
                } else if (A.sink) {
                    A.sink[path] = make_float4(color.x, color.y, color.z, 0.0f);
                } else {
                    write_pixel<BATCH>(F, pid, color, depth, BATCH || !A.early_depth);
                }
            }
        }
        uint32_t q = warp_append(A.count_out, bounce);
        if (bounce) {
            bump<COUNT>(w.bounce);
            A.rays_out[2 * (size_t)q] = make_float4(bo.x, bo.y, bo.z, __uint_as_float(path));
            A.rays_out[2 * (size_t)q + 1] = make_float4(bd.x, bd.y, bd.z, __uint_as_float(pid));
        }
        if (BATCH) {
            uint32_t cq = warp_append(A.cache.count, query);
            if (query) append_query(A.cache, cq, feat, o, d, path, pid, qc, qt);
        }
    }
    flush_stage<COUNT>(A.counters, w);
}

// ---- radiance cache ----------------------------------------------------------
// Single-request frames: the round at the cache depth runs this instead of
// shadows and shading.
template <bool COUNT>
__global__ void __launch_bounds__(256) k_cache_gather(DevScene S, DevFrame F, QueueArgs A, CacheArgs C) {
    chain_wait();
    uint32_t n = queue_size(A);
    Work w = {};
    uint32_t stride = gridDim.x * blockDim.x;
    uint32_t rounds = (n + stride - 1) / stride;
    for (uint32_t r = 0, slot = blockIdx.x * blockDim.x + threadIdx.x; r < rounds; r++, slot += stride) {
        bool query = false;
        uint32_t path = 0, pid = 0;
        float3 o = f3(0, 0, 0), d = f3(0, 0, 0);
        float4 feat[4], qc = make_float4(0, 0, 0, 0), qt = make_float4(0, 0, 0, 0);
        if (slot < n) {
            load_ray(F, A, slot, o, d, path, pid);
            query = cache_vertex<COUNT, false>(S, F, A, slot, path, pid, o, d, feat, w, qc, qt);
        }
        uint32_t q = warp_append(C.count, query);
        if (query) append_query(C, q, feat, o, d, path, pid, qc, qt, A.hits, A.hit_stride, slot);
    }
    flush_stage<COUNT>(A.counters, w);
}

// Training paths: query j of the frame's training set restarts from the
// query's ray with zero colour and unit throughput in its own slot j.  With
// more queries than training paths the set is stratified: j takes query
// floor((j + u) * queries / capacity), u = frac(0.618034 * frame) (a
// golden-ratio sequence, so consecutive frames train on different queries).
__global__ void k_cache_select(CacheArgs C, float4 *rays, uint32_t *ray_count, float4 *hits, uint32_t hit_stride) {
    const uint32_t nq = *C.count, cap = C.train_capacity;
    const uint32_t n = nq < cap ? nq : cap;
    const double f = (double)*C.frame_counter * 0.6180339887498949;
    const double u = f - floor(f);
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        uint32_t idx = j;
        if (nq > cap) {
            idx = (uint32_t)(((double)j + u) * (double)nq / (double)cap);
            if (idx >= nq) idx = nq - 1;
        }
        if (C.t_features) {
            const float4 *f = C.features + 4 * (size_t)idx;
            float4 *t = C.t_features + 4 * (size_t)j;
            t[0] = f[0]; t[1] = f[1]; t[2] = f[2]; t[3] = f[3];
        }
        if (C.q_hit && hits) {   // the query's hit: the training path's first round needs no extend
            const float4 *h = C.q_hit + 3 * (size_t)idx;
            hits[j] = h[0];
            hits[(size_t)hit_stride + j] = h[1];
            hits[2 * (size_t)hit_stride + j] = h[2];
        }
        float4 a = C.aux[2 * (size_t)idx], b = C.aux[2 * (size_t)idx + 1];
        rays[2 * (size_t)j] = make_float4(a.x, a.y, a.z, __uint_as_float(j));
        rays[2 * (size_t)j + 1] = b;
        C.t_color[j] = make_float4(0.0f, 0.0f, 0.0f, INFINITY);
        C.t_through[j] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *C.train_count = n;
        *ray_count = n;
    }
}

// Self-training targets: a training path that reached its cache vertex
// (query q of the self-training set) ends in the cache's answer there:
// target = colour so far + throughput * radiance.  Paths that ended earlier
// already wrote their targets.
__global__ void k_cache_train_targets(const float4 *aux, const uint32_t *count, const float4 *radiance,
                                      const float4 *t_color, const float4 *t_through, float4 *t_targets) {
    const uint32_t nq = *count;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x) {
        uint32_t path = __float_as_uint(aux[2 * (size_t)q].w);
        float3 c = mul_add(xyz(radiance[q]), xyz(t_through[path]), xyz(t_color[path]));
        t_targets[path] = make_float4(c.x, c.y, c.z, 0.0f);
    }
}

// Waiting paths take the cache's answer: colour += throughput * radiance,
// then tone mapping and the canvas write of k_shade.
template <bool BATCH>
__global__ void k_cache_resolve(DevFrame F0, QueueArgs A, const float4 *path_color, const float4 *path_throughput) {
    const CacheArgs &C = A.cache;
    const uint32_t nq = *C.count;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(C.frame_counter, 1u);
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x) {
        uint32_t path = __float_as_uint(C.aux[2 * (size_t)q].w);
        uint32_t pid = __float_as_uint(C.aux[2 * (size_t)q + 1].w);
        float4 pc = C.q_color ? C.q_color[q] : path_color[path];
        float3 thr = xyz(C.q_color ? C.q_through[q] : path_throughput[path]);
        float3 L = f3(0, 0, 0);
        if (C.mode == SLIM_CACHE_ON) L = xyz(C.radiance[q]);
        else if (C.mode == SLIM_CACHE_EXACT) L = xyz(C.t_targets[q]);
        write_pixel<BATCH>(frame_of<BATCH>(F0, A, pid), pid, mul_add(L, thr, xyz(pc)), pc.w);
    }
}

// ---- batched requests: primary rays of a wave --------------------------------
// tiles[t] = (request, first pixel, pixel count, first slot), slots ascending.
__global__ void k_batch_generate(QueueArgs A, const uint4 *__restrict__ tiles, uint32_t tile_count, float4 *rays,
                                 uint32_t *ray_count, uint32_t wave_samples, unsigned long long *counters) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < wave_samples; s += gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = tile_count;          // last tile with first slot <= s
        while (hi - lo > 1) {
            uint32_t mid = (lo + hi) >> 1;
            if (__ldg(&tiles[mid].w) <= s) lo = mid; else hi = mid;
        }
        uint4 t = tiles[lo];
        const DevFrame &F = A.frames[t.x];
        const uint2 xy = xy_of_slot(F.width, F.height, t.y + (s - t.w));
        const uint32_t pixel = xy.y * F.width + xy.x;
        float3 o, d;
        primary_ray(F, xy.x, xy.y, o, d);
        rays[2 * (size_t)s] = make_float4(o.x, o.y, o.z, __uint_as_float(s));
        rays[2 * (size_t)s + 1] = make_float4(d.x, d.y, d.z, __uint_as_float((t.x << kBatchPixelBits) | pixel));
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *ray_count = wave_samples;
        if (counters) atomicAdd(counters, (unsigned long long)wave_samples);   // primary rays
    }
}

// ---- frame orchestration ------------------------------------------------------
struct RoundLaunch {
    const DevScene *S;
    const DevFrame *F;
    const WavefrontBuffers *B;
    int block, sms;
    cudaStream_t stream;
    StageTimer *timer;
    unsigned long long *counters;
    uint32_t bound;      // queue capacity (one ray per path slot)
    uint32_t lights;     // most lights of any scene in the round
    bool split_extend;   // closest hits as scene candidates + the persistent mesh pass
    bool share_sms = false;  // leave a block's room per SM (overlapped cache training runs beside)
    cudaEvent_t pixel_wait = nullptr;  // kernels that write pixels wait for it (a download in flight)
    const FrameDownload *depth_download = nullptr;  // first round: the depths download after shadow_gen
    const FrameDownload *pixel_download = nullptr;  // first round: each shade chunk's rows download after it
    // Chained launches: a round's kernels follow one another on their stream,
    // most of them for a few microseconds, and the gap between the end of one
    // and the start of the next counts as much as they do.  A chained kernel is
    // set up while the one before it drains and waits in chain_wait instead
    // (light meshes at 637x359, 4 bounces 589 -> 515 us, mesh 1080p depth 8
    // 2.147 -> 1.997 ms, depth 2 1.135 -> 1.103 ms, textures 1080p 389 -> 377
    // us; signalled from the start of each kernel instead of from its end, the
    // waiting blocks keep the other band off the SMs: 2.050 and 1.124 ms).
    // The first launch of a frame is not chained, so that the scene it reads
    // through the read-only path is complete; neither are launches that wait for
    // an event of another stream or are captured into a graph.  (An event
    // recorded between two launches of the stream changes nothing: it marks the
    // end of the first, and the second writes nothing before that.)  A launch's
    // error is the last error, which each round checks.
    bool chain = false;
    template <typename... P, typename... X>
    void launch(bool chained, void (*kernel)(P...), uint32_t grid, int threads, const X &...args) const {
        cudaLaunchAttribute serial{};
        serial.id = cudaLaunchAttributeProgrammaticStreamSerialization;
        serial.val.programmaticStreamSerializationAllowed = 1;
        cudaLaunchConfig_t config{};
        config.gridDim = dim3(grid);
        config.blockDim = dim3((uint32_t)threads);
        config.stream = stream;
        config.attrs = &serial;
        config.numAttrs = chain && chained ? 1 : 0;
        cudaLaunchKernelEx(&config, kernel, args...);
        count_launch();
    }
    unsigned long long *stage(int st) const { return counters ? counters + kCountersPerStage * st : nullptr; }
    uint32_t grid(const void *kernel, uint32_t work) const { return grid_for(kernel, work, block); }
    // the persistent mesh kernels run 128-thread blocks (kMeshBlock)
    uint32_t mesh_grid(const void *kernel, uint32_t work) const { return grid_for(kernel, work, kMeshBlock); }
    uint32_t grid_for(const void *kernel, uint32_t work, int block) const {
        int per_sm = 1;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0);
        if (share_sms && per_sm > 1) per_sm--;
        uint32_t g = (uint32_t)(sms * (per_sm > 0 ? per_sm : 1));
        uint32_t need = (work + block - 1) / block;
        return need < g ? (need ? need : 1) : g;
    }
};

// One bounce round over the queue `in` (primary rays at depth 1 of a single
// frame): extend, then shadows and shading -- or, at a single frame's cache
// depth, the cache gather.  Leaves `in` at the round's output queue.
// Paths still bouncing at depth >= kTailDepth finish in the fused tail kernel
// when the scene has no meshes: textures at 1080p, depth 8, 394 us, with the
// tail from depth 2 393 and from 4 419.  With meshes the rounds stay: one thread
// per remaining path would walk mesh BVHs and every light's shadow ray serially
// (1080p, 8 bounces, 2.88 against 1.99 ms; light meshes at 637x359 1.28 against
// 0.69).
constexpr uint32_t kTailDepth = 3;

// The rest of the paths queued in `in` (depth `depth` on) in one fused kernel.
template <bool COUNT, bool BATCH>
cudaError_t tail_round(const RoundLaunch &L, QueueArgs &A, uint32_t in, uint32_t depth) {
    const WavefrontBuffers &B = *L.B;
    A.depth = depth;
    A.rays_in = B.rays[in];
    A.count_in = A.count_out;
    if (L.pixel_wait) {
        cudaError_t r = cudaStreamWaitEvent(L.stream, L.pixel_wait, 0);
        if (r != cudaSuccess) return r;
    }
    A.counters = L.stage(STAGE_TAIL);
    if (L.timer) L.timer->begin(STAGE_TAIL, L.stream);
    RoundLaunch T = L;
    T.block = 128;
    L.launch(!L.pixel_wait, k_finish_paths<COUNT, BATCH>, T.grid((const void *)k_finish_paths<COUNT, BATCH>, L.bound),
             T.block, *L.S, *L.F, A);
    if (L.timer) L.timer->end(STAGE_TAIL, L.stream);
    return cudaGetLastError();
}

template <bool COUNT, bool BATCH>
cudaError_t trace_round(const RoundLaunch &L, QueueArgs &A, const CacheArgs &CA, uint32_t &in, uint32_t depth,
                        bool primary, bool gather, bool hits_given = false) {
    const WavefrontBuffers &B = *L.B;
    const DevScene &S = *L.S;
    const DevFrame &F = *L.F;
    cudaStream_t stream = L.stream;
    StageTimer *timer = L.timer;
    uint32_t out = in ^ 1u;
    A.depth = depth;
    uint32_t *const counts = A.round_counts;
    A.round_counts += kRoundWords;
    A.rays_in = primary ? nullptr : B.rays[in];
    A.count_in = primary ? nullptr : A.count_out;
    A.rays_out = B.rays[out];
    A.count_out = counts;
    cudaError_t r;
    A.counters = L.stage(STAGE_EXTEND);
    if (timer) timer->begin(STAGE_EXTEND, stream);
    if (hits_given) {
        // the queued rays' hit records are in place already (training paths
        // that start at their cache vertex)
    } else if (L.split_extend && B.pair_capacity >= 4) {
        A.pair_count = counts + 1;
        A.pair_cursor = counts + 2;
        L.launch(!primary, k_extend_scene<COUNT, BATCH>,
                 L.grid((const void *)k_extend_scene<COUNT, BATCH>, L.bound), L.block, S, F, A);
        const auto extend_mesh = S.binary_walks ? k_extend_mesh<COUNT, false> : k_extend_mesh<COUNT, true>;
        L.launch(true, extend_mesh, L.mesh_grid((const void *)extend_mesh, B.pair_capacity), kMeshBlock, S, F, A);
        L.launch(true, k_extend_resolve<COUNT, BATCH>,
                 L.grid((const void *)k_extend_resolve<COUNT, BATCH>, B.pair_capacity), L.block, S, F, A);
        L.launch(true, k_extend_overflow<COUNT, BATCH>,
                 L.grid((const void *)k_extend_overflow<COUNT, BATCH>, L.bound), L.block, S, F, A);
    } else {
        L.launch(!primary, k_extend<COUNT, BATCH>,
                 L.grid((const void *)k_extend<COUNT, BATCH>, L.bound), L.block, S, F, A);
    }
    if (timer) timer->end(STAGE_EXTEND, stream);
    if (gather) {
        A.counters = L.stage(STAGE_CACHE);
        if (timer) timer->begin(STAGE_CACHE, stream);
        L.launch(true, k_cache_gather<COUNT>, L.grid((const void *)k_cache_gather<COUNT>, L.bound), L.block, S, F, A, CA);
        if (timer) timer->end(STAGE_CACHE, stream);
        in = out;
        return cudaGetLastError();
    }
    // Shadow rays in light batches that fit the shadow queue.
    uint32_t per_batch = B.shadow_capacity / (L.bound ? L.bound : 1);
    if (per_batch < 1) per_batch = 1;
    for (uint32_t l0 = 0; l0 < L.lights; l0 += per_batch) {
        A.light_begin = l0;
        A.light_end = l0 + per_batch < L.lights ? l0 + per_batch : L.lights;
        if (l0 && (r = cudaMemsetAsync(counts + 5, 0, 3 * sizeof(uint32_t), stream)) != cudaSuccess) return r;
        A.shadow_count = counts + 5;
        A.counters = L.stage(STAGE_SHADOW_GEN);
        if (timer) timer->begin(STAGE_SHADOW_GEN, stream);
        L.launch(true, k_shadow_gen<COUNT, BATCH>, L.grid((const void *)k_shadow_gen<COUNT, BATCH>, L.bound), L.block, S, F, A);
        if (timer) timer->end(STAGE_SHADOW_GEN, stream);
        if (l0 == 0 && A.early_depth && L.depth_download) {
            const FrameDownload *dl = L.depth_download;
            if ((r = cudaEventRecord(dl->depths_done, stream)) != cudaSuccess) return r;
            if ((r = cudaStreamWaitEvent(dl->copy_stream, dl->depths_done, 0)) != cudaSuccess) return r;
            if ((r = cudaMemcpyAsync(dl->host_depths, dl->dev_depths, dl->depth_bytes, cudaMemcpyDeviceToHost,
                                     dl->copy_stream)) != cudaSuccess)
                return r;
        }
        // Scene arrays without meshes (split_extend is false exactly then)
        // append no (shadow ray, instance) pairs: no mesh pass (config 3: 0.021
        // ms of a 0.56 ms whole-frame pass).
        A.pair_count = counts + 6;
        A.pair_cursor = counts + 7;
        A.counters = L.stage(STAGE_SHADOW);
        if (timer) timer->begin(STAGE_SHADOW, stream);
        L.launch(true, k_shadow_scene<COUNT, BATCH>,
                 L.grid((const void *)k_shadow_scene<COUNT, BATCH>, L.bound * (A.light_end - A.light_begin)), L.block, S, F, A);
        if (timer) timer->end(STAGE_SHADOW, stream);
        if (!L.split_extend) continue;
        A.counters = L.stage(STAGE_SHADOW_MESH);
        if (timer) timer->begin(STAGE_SHADOW_MESH, stream);
        const auto shadow_mesh = S.binary_walks ? k_shadow_mesh<COUNT, false> : k_shadow_mesh<COUNT, true>;
        L.launch(true, shadow_mesh, L.mesh_grid((const void *)shadow_mesh, B.pair_capacity), kMeshBlock, S, F, A);
        if (timer) timer->end(STAGE_SHADOW_MESH, stream);
    }
    if (L.pixel_wait && (r = cudaStreamWaitEvent(stream, L.pixel_wait, 0)) != cudaSuccess) return r;
    A.counters = L.stage(STAGE_SHADE);
    if (timer) timer->begin(STAGE_SHADE, stream);
    // A downloaded frame's first round shades its primary paths (slot =
    // sample, in row order) in chunks of whole 4-row tiles; each chunk's rows
    // start crossing PCIe while the next chunk shades.
    const FrameDownload *dl = L.pixel_download;
    const uint32_t chunks = dl ? kPixelChunks : 1u, tiles = (F.rows + 3) / 4;
    for (uint32_t c = 0; c < chunks; c++) {
        const uint32_t r0 = 4 * (tiles * c / chunks), r1 = c + 1 == chunks ? F.rows : 4 * (tiles * (c + 1) / chunks);
        if (dl) {
            A.slot_begin = r0 * F.width;
            A.slot_end = r1 * F.width;
            if (r1 == r0) continue;
        }
        L.launch(!dl && !L.pixel_wait, k_shade<COUNT, BATCH>,
                 L.grid((const void *)k_shade<COUNT, BATCH>, dl ? A.slot_end - A.slot_begin : L.bound), L.block, S, F, A);
        if (dl) {
            if ((r = cudaEventRecord(dl->pixels_done[c], stream)) != cudaSuccess) return r;
            if ((r = cudaStreamWaitEvent(dl->copy_stream, dl->pixels_done[c], 0)) != cudaSuccess) return r;
            if ((r = cudaMemcpyAsync((char *)dl->host_pixels + r0 * dl->pixel_row_bytes,
                                     (const char *)dl->dev_pixels + r0 * dl->pixel_row_bytes,
                                     (r1 - r0) * dl->pixel_row_bytes, cudaMemcpyDeviceToHost, dl->copy_stream)) != cudaSuccess)
                return r;
        }
    }
    A.slot_begin = A.slot_end = 0;
    if (timer) timer->end(STAGE_SHADE, stream);
    in = out;
    return cudaGetLastError();
}

CacheArgs cache_args(const CacheFrame *cache) {
    CacheArgs CA{};
    if (!cache) return CA;
    CA.features = cache->features;
    CA.aux = cache->aux;
    CA.radiance = cache->radiance;
    CA.count = cache->counts;
    CA.train_count = cache->counts + 1;
    CA.train_capacity = cache->train_capacity;
    CA.t_features = cache->mode == SLIM_CACHE_ON ? cache->t_features : nullptr;
    CA.t_targets = cache->t_targets;
    CA.t_color = cache->t_color;
    CA.t_through = cache->t_through;
    CA.frame_counter = cache->frame_counter;
    CA.mode = cache->mode;
    CA.q_color = cache->q_color;
    CA.q_through = cache->q_through;
    CA.q_hit = cache->q_hit;
    return CA;
}

// The training paths queued in `in` (from the cache vertex on; A sinks
// their radiance into the training targets): traced to max_depth, or -- with
// a training suffix, in single-request frames -- `train_suffix` bounces on,
// where the paths still going query the cache (with the training's current
// weights, `weights`) and their targets take its answer.
template <bool COUNT, bool BATCH>
cudaError_t trace_training(const RoundLaunch &L, QueueArgs &A, const CacheArgs &CA, uint32_t in,
                           const CacheFrame *cache, uint32_t max_depth, const uint8_t *weights) {
    cudaError_t e;
    const uint32_t K = cache->depth;
    const bool short_paths = !BATCH && weights && cache->train_suffix && cache->s_count &&
                             K + cache->train_suffix <= max_depth;
    // the selection copied every training path's hit at the cache vertex
    const bool hits_given = !BATCH && cache->q_hit;
    if (!short_paths) {
        if (!L.split_extend && !hits_given) return tail_round<COUNT, BATCH>(L, A, in, K);
        for (uint32_t depth = K; depth <= max_depth; depth++) {
            if (!L.split_extend && depth >= kTailDepth && depth > K) return tail_round<COUNT, BATCH>(L, A, in, depth);
            if ((e = trace_round<COUNT, BATCH>(L, A, CA, in, depth, false, false, hits_given && depth == K)) != cudaSuccess)
                return e;
        }
        return cudaSuccess;
    }
    const uint32_t last = K + cache->train_suffix;
    CacheArgs SC = CA;
    SC.features = cache->s_features;
    SC.aux = cache->s_aux;
    SC.count = cache->s_count;
    SC.q_color = SC.q_through = SC.q_hit = nullptr;   // the frame's own query records stay untouched
    for (uint32_t depth = K; depth < last; depth++)
        if ((e = trace_round<COUNT, BATCH>(L, A, CA, in, depth, false, false, hits_given && depth == K)) != cudaSuccess)
            return e;
    if ((e = cudaMemsetAsync(cache->s_count, 0, sizeof(uint32_t), L.stream)) != cudaSuccess) return e;
    if ((e = trace_round<COUNT, BATCH>(L, A, SC, in, last, false, true)) != cudaSuccess) return e;
    if ((e = nrc::launch_infer(cache->s_features, cache->s_count, 0, cache->train_capacity, cache->s_radiance, weights,
                               L.F->error_flags, L.stream)) != cudaSuccess)
        return e;
    uint32_t g = (cache->train_capacity + 255) / 256;
    if (g > (uint32_t)(L.sms * 4)) g = (uint32_t)(L.sms * 4);
    k_cache_train_targets<<<g ? g : 1, 256, 0, L.stream>>>(cache->s_aux, cache->s_count, cache->s_radiance,
                                                            cache->t_color, cache->t_through, cache->t_targets);
    count_launch();
    return cudaGetLastError();
}

// The Adam steps over a frame's training set, as many as a full set takes; a
// step past the parts of the set as it is changes nothing.
cudaError_t train_steps(const CacheFrame *cache, cudaStream_t stream) {
    const uint32_t n = cache->batch < cache->train_capacity ? cache->batch : cache->train_capacity;
    for (uint32_t off = 0; off < cache->train_capacity; off += n) {
        const cudaError_t e = cache->trainer->step(cache->t_features, cache->t_targets, n, cache->counts + 1, off, stream);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// After the queries of a frame (or wave) are gathered: the training paths
// traced on (to max_depth, or a few bounces into the cache's own answers),
// the Adam steps, the network's answers, and the waiting paths resolved.
template <bool COUNT, bool BATCH>
cudaError_t cache_phase(const RoundLaunch &L, QueueArgs &A, const CacheArgs &CA, uint32_t &in, const CacheFrame *cache,
                        uint32_t max_depth) {
    const WavefrontBuffers &B = *L.B;
    cudaStream_t stream = L.stream;
    StageTimer *timer = L.timer;
    cudaError_t e;
    const int mode = cache->mode;
    const bool train = mode == SLIM_CACHE_ON && cache->trainer && cache->batch && cache->train_capacity;
    if (train && cache->train_stream && cache->train_queues && !BATCH) {
        // Overlapped training.  The previous frame's training has finished
        // once `trained` completes: take its weights for this frame's
        // queries, then hand this frame's training paths to the training
        // stream, which traces them with its own queues while this stream
        // answers the queries and the next frame's primary rays run.
        const WavefrontBuffers &TB = *cache->train_queues;
        cudaStream_t ts = cache->train_stream;
        if ((e = cudaStreamWaitEvent(stream, cache->trained, 0)) != cudaSuccess) return e;
        if ((e = cudaMemcpyAsync((void *)cache->weights, cache->train_weights, nrc::kImgBytes, cudaMemcpyDeviceToDevice,
                                 stream)) != cudaSuccess)
            return e;
        if ((e = cudaMemsetAsync(TB.queue_count, 0, counter_bytes(max_depth + 2), stream)) != cudaSuccess) return e;
        if (timer) timer->begin(STAGE_CACHE, stream);
        uint32_t g = (cache->train_capacity + 255) / 256;
        if (g > (uint32_t)(L.sms * 8)) g = (uint32_t)(L.sms * 8);
        k_cache_select<<<g ? g : 1, 256, 0, stream>>>(CA, TB.rays[0], TB.queue_count, TB.hits, TB.capacity);
        count_launch();
        if (timer) timer->end(STAGE_CACHE, stream);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        if ((e = cudaEventRecord(cache->selected, stream)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(ts, cache->selected, 0)) != cudaSuccess) return e;
        RoundLaunch TL{L.S, L.F, &TB, L.block, L.sms, ts, nullptr, nullptr, TB.capacity, L.lights, L.split_extend};
        QueueArgs TA = A;
        TA.hits = TB.hits;
        TA.hit_stride = TB.capacity;
        TA.shadow_rays = TB.shadow_rays;
        TA.masks = TB.shadow_mask;
        TA.pairs = TB.pairs;
        TA.count_out = TB.queue_count;
        TA.round_counts = TB.queue_count + kRoundWords;
        TA.pair_capacity = TB.pair_capacity;
        TA.path_color = cache->t_color;
        TA.path_throughput = cache->t_through;
        TA.sink = cache->t_targets;
        TA.skip_glow_depth = cache->depth;
        TA.samples = TB.capacity;
        if ((e = trace_training<false, false>(TL, TA, CA, 0, cache, max_depth, cache->train_weights)) != cudaSuccess)
            return e;
        if ((e = train_steps(cache, ts)) != cudaSuccess) return e;
        if ((e = cudaEventRecord(cache->trained, ts)) != cudaSuccess) return e;
    } else if (mode == SLIM_CACHE_EXACT || train) {
        if (timer) timer->begin(STAGE_CACHE, stream);
        uint32_t g = (cache->train_capacity + 255) / 256;
        if (g > (uint32_t)(L.sms * 8)) g = (uint32_t)(L.sms * 8);
        k_cache_select<<<g ? g : 1, 256, 0, stream>>>(CA, B.rays[in], B.queue_count + in, B.hits, B.capacity);
        count_launch();
        if (timer) timer->end(STAGE_CACHE, stream);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        QueueArgs main = A;
        A.count_out = B.queue_count + in;
        A.path_color = cache->t_color;
        A.path_throughput = cache->t_through;
        A.sink = cache->t_targets;
        A.skip_glow_depth = cache->depth;
        if ((e = trace_training<COUNT, BATCH>(L, A, CA, in, cache, max_depth,
                                              mode == SLIM_CACHE_ON ? cache->weights : nullptr)) != cudaSuccess)
            return e;
        main.round_counts = A.round_counts;
        A = main;
    }
    if (train && !(cache->train_stream && cache->train_queues && !BATCH)) {
        if (timer) timer->begin(STAGE_CACHE_TRAIN, stream);
        if ((e = train_steps(cache, stream)) != cudaSuccess) return e;
        if (timer) timer->end(STAGE_CACHE_TRAIN, stream);
    }
    if (mode == SLIM_CACHE_ON) {
        if (timer) timer->begin(STAGE_CACHE_QUERY, stream);
        e = nrc::launch_infer(cache->features, cache->counts, 0, L.bound, cache->radiance, cache->weights,
                              L.F->error_flags, stream);
        if (timer) timer->end(STAGE_CACHE_QUERY, stream);
        if (e != cudaSuccess) return e;
    }
    if (timer) timer->begin(STAGE_CACHE, stream);
    A.cache = CA;
    k_cache_resolve<BATCH><<<L.grid((const void *)k_cache_resolve<BATCH>, L.bound), L.block, 0, stream>>>(
        *L.F, A, B.path_color, B.path_throughput);
    count_launch();
    if (timer) timer->end(STAGE_CACHE, stream);
    return cudaGetLastError();
}

template <bool COUNT>
cudaError_t run_frame(const DevScene &S, const DevFrame &F, const WavefrontBuffers &B, int block, cudaStream_t stream,
                      StageTimer *timer, const CacheFrame *cache, const FrameDownload *dl) {
    uint32_t samples = F.width * F.rows;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    RoundLaunch L{&S, &F, &B, block <= 0 ? 256 : block, sms, stream, timer, F.counters, samples, S.light_count,
                  S.mesh_count > 0};
    // the cache's overlapped training runs beside this frame: leave it room
    // (config 4: 3.50 -> 3.37 ms per frame)
    L.share_sms = cache && cache->train_stream && cache->mode == SLIM_CACHE_ON && !cache->train_suffix;
    cudaError_t e = cudaMemsetAsync(B.queue_count, 0, counter_bytes(2 * F.settings.max_depth + 4), stream);
    if (e != cudaSuccess) return e;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    const bool known = cudaStreamIsCapturing(stream, &capture) == cudaSuccess;
    if (!known) cudaGetLastError();
    L.chain = known && capture == cudaStreamCaptureStatusNone && !timer;
    QueueArgs A{};
    A.hits = B.hits;
    A.hit_stride = B.capacity;
    A.shadow_rays = B.shadow_rays;
    A.masks = B.shadow_mask;
    A.pairs = B.pairs;
    A.round_counts = B.queue_count + kRoundWords;
    A.pair_capacity = B.pair_capacity;
    A.path_color = B.path_color;
    A.path_throughput = B.path_throughput;
    A.samples = samples;
    const uint32_t max_depth = F.settings.max_depth;
    const bool use_cache = cache && cache->mode != SLIM_CACHE_OFF && cache->depth >= 2 && cache->depth <= max_depth;
    CacheArgs CA = use_cache ? cache_args(cache) : CacheArgs{};
    const int part = use_cache ? cache->part : kCachePartWhole;
    uint32_t in = 0;
    if (part == kCachePartPhase) {   // the bands have gathered every query of the frame
        A.cache = CA;
        return cache_phase<COUNT, false>(L, A, CA, in, cache, max_depth);
    }
    // Only the query count starts over: the training count belongs to the
    // training set, which the overlapped training stream may still be using;
    // the selection that replaces the set rewrites it.  (A banded frame
    // clears it once, before its bands.)
    if (use_cache && part == kCachePartWhole &&
        (e = cudaMemsetAsync(cache->counts, 0, sizeof(uint32_t), stream)) != cudaSuccess)
        return e;
    const uint32_t last = use_cache ? cache->depth : max_depth;
    DevFrame late = F;   // the frame as the rounds after a download see it
    for (uint32_t depth = 1; depth <= last; depth++) {
        if (!L.split_extend && depth >= kTailDepth && !(use_cache && depth == last)) {
            if ((e = tail_round<COUNT, false>(L, A, in, depth)) != cudaSuccess) return e;
            break;
        }
        // the depths are final after the first round's shadow_gen (which
        // needs a light to run): they download while the shadows are traced
        const bool early_depth = depth == 1 && dl && !use_cache && L.lights > 0;
        A.early_depth = early_depth;
        L.depth_download = early_depth ? dl : nullptr;
        // every path that ends at its first hit writes its pixel in this
        // round's shading: the rows go to the host chunk by chunk
        L.pixel_download = depth == 1 && !use_cache ? dl : nullptr;
        if ((e = trace_round<COUNT, false>(L, A, CA, in, depth, depth == 1, use_cache && depth == last)) != cudaSuccess)
            return e;
        A.early_depth = 0;
        L.depth_download = L.pixel_download = nullptr;
        if (depth == 1 && dl && !use_cache) {
            // the copy stream is past the round's last shade chunk: later
            // pixels go to the host canvas directly once the copies landed
            if (!early_depth && (e = cudaMemcpyAsync(dl->host_depths, dl->dev_depths, dl->depth_bytes,
                                                     cudaMemcpyDeviceToHost, dl->copy_stream)) != cudaSuccess)
                return e;
            if ((e = cudaEventRecord(dl->copied, dl->copy_stream)) != cudaSuccess) return e;
            late.pixels = dl->mapped_pixels;
            late.depths = dl->mapped_depths;
            L.F = &late;
            L.pixel_wait = dl->copied;
        }
    }
    if (!use_cache || part == kCachePartGather) return cudaSuccess;
    A.cache = CA;
    return cache_phase<COUNT, false>(L, A, CA, in, cache, max_depth);
}

// Batched requests: every wave is a full multi-request frame over its slots.
template <bool COUNT>
cudaError_t run_batch(const BatchFrame &BF, const WavefrontBuffers &B0, int block, cudaStream_t stream0,
                      StageTimer *timer) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const CacheFrame *cache = BF.cache;
    CacheArgs CA = cache_args(cache);
    cudaError_t e;
    const bool two_lanes = BF.lane_stream && BF.lane_queues;
    if (two_lanes) {
        if ((e = cudaEventRecord(BF.lane_fork, stream0)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(BF.lane_stream, BF.lane_fork, 0)) != cudaSuccess) return e;
    }
    uint32_t next_lane = 0;
    if (BF.p_count && BF.p_total) {
        // the persistent launch takes the second lane; the waves (the cache
        // requests') all stay on the first
        cudaStream_t ps = two_lanes ? BF.lane_stream : stream0;
        if (timer) timer->begin(STAGE_FUSED, ps);
        if ((e = launch_batch_persistent(BF.scenes, BF.frames, BF.p_requests, BF.p_prefix, BF.p_count, BF.p_total,
                                         BF.p_cursor, BF.frame.error_flags, BF.frame.counters, ps)) != cudaSuccess)
            return e;
        if (timer) timer->end(STAGE_FUSED, ps);
    }
    const bool one_lane_waves = BF.p_count && BF.p_total;
    for (uint32_t wi = 0; wi < BF.wave_count; wi++) {
        const BatchWave &wave = BF.waves[wi];
        uint32_t lane = 0;
        if (two_lanes && !one_lane_waves && !(cache && wave.cache_paths)) {
            lane = next_lane;
            next_lane ^= 1u;
        }
        const WavefrontBuffers &B = lane ? *BF.lane_queues : B0;
        const cudaStream_t stream = lane ? BF.lane_stream : stream0;
        RoundLaunch L{&BF.shared, &BF.frame, &B, block <= 0 ? 256 : block, sms, stream, timer, BF.frame.counters,
                      B.capacity, wave.max_lights, BF.shared.mesh_count > 0};
        if ((e = cudaMemsetAsync(B.queue_count, 0, counter_bytes(2 * wave.max_depth + 4), stream)) != cudaSuccess) return e;
        const bool use_cache = cache && wave.cache_paths;
        if (use_cache && (e = cudaMemsetAsync(cache->counts, 0, sizeof(uint32_t), stream)) != cudaSuccess)
            return e;
        QueueArgs A{};
        A.hits = B.hits;
        A.hit_stride = B.capacity;
        A.shadow_rays = B.shadow_rays;
        A.masks = B.shadow_mask;
        A.pairs = B.pairs;
        A.count_out = B.queue_count;
        A.round_counts = B.queue_count + kRoundWords;
        A.pair_capacity = B.pair_capacity;
        A.path_color = B.path_color;
        A.path_throughput = B.path_throughput;
        A.samples = wave.samples;
        A.scenes = BF.scenes;
        A.frames = BF.frames;
        A.cache = CA;
        if (timer) timer->begin(STAGE_EXTEND, stream);
        uint32_t g = (wave.samples + 255) / 256;
        if (g > (uint32_t)(sms * 8)) g = (uint32_t)(sms * 8);
        k_batch_generate<<<g ? g : 1, 256, 0, stream>>>(A, BF.tiles + wave.first_tile, wave.tile_count, B.rays[0],
                                                         B.queue_count, wave.samples, L.stage(STAGE_EXTEND));
        count_launch();
        if (timer) timer->end(STAGE_EXTEND, stream);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        uint32_t in = 0;
        const uint32_t tail_from = cache && cache->depth >= kTailDepth ? cache->depth + 1 : kTailDepth;
        for (uint32_t depth = 1; depth <= wave.max_depth; depth++) {
            if (!L.split_extend && depth >= tail_from) {
                if ((e = tail_round<COUNT, true>(L, A, in, depth)) != cudaSuccess) return e;
                break;
            }
            if ((e = trace_round<COUNT, true>(L, A, CA, in, depth, false, false)) != cudaSuccess) return e;
        }
        if (use_cache && (e = cache_phase<COUNT, true>(L, A, CA, in, cache, wave.max_depth)) != cudaSuccess) return e;
    }
    if (two_lanes) {
        if ((e = cudaEventRecord(BF.lane_join, BF.lane_stream)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(stream0, BF.lane_join, 0)) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace dev

cudaError_t launch_render_wavefront(const DevScene &S, const DevFrame &F, const WavefrontBuffers &B, int block,
                                    cudaStream_t stream, StageTimer *timer, const CacheFrame *cache,
                                    const FrameDownload *download) {
    if (F.settings.render_mode != SLIM_RENDER_BEAUTY)   // a single primary hit: nothing to queue
        return launch_render_fused(S, F, block, stream, timer);
    if (F.settings.max_depth == 0) return launch_render_fused(S, F, block, stream, timer);
    if (F.counters) return dev::run_frame<true>(S, F, B, block, stream, timer, cache, download);
    return dev::run_frame<false>(S, F, B, block, stream, timer, cache, download);
}

cudaError_t launch_render_batch(const BatchFrame &BF, const WavefrontBuffers &B, int block, cudaStream_t stream,
                                StageTimer *timer) {
    if (BF.frame.counters) return dev::run_batch<true>(BF, B, block, stream, timer);
    return dev::run_batch<false>(BF, B, block, stream, timer);
}

}  // namespace slim
