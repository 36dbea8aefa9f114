// Device-resident scene and render parameters of the B200 path tracer.
//
// HBM layout (one allocation per array, all 16-byte aligned):
//   nodes         4-wide BVH nodes with byte-quantised boxes, 64 B each
//                 (two 32-byte sectors): the instance tree, then every
//                 mesh's tree
//   node_boxes / instance_boxes  float boxes, 32 B each
//   tris          leaf triangles of all meshes in node order, 64 B each:
//                 object-space vertices, local primitive index, padded box
//   entries       per instance, the ray's transform and the mesh's root (64 B)
//   shade_tris    the meshes' triangles as shading reads them, 96 B each
//   instances     InstanceGpu (object<->world transforms, material)
//   materials / code / scalars / vectors  closure programs and their
//                 parameter blocks (rebinding rewrites scalars/vectors)
//   baked / closures  the programs evaluated, as the kernels shade with them
//   emitters / distribution  emissive triangles and the flat light CDF
//   lights        analytic lights (psy_light_desc)
#pragma once

#include <cstdint>

#include "../../include/psycles_cuda.h"
#include "psy_light_tree.h"

namespace psy {

constexpr uint32_t kInvalidId = 0xffffffffu;

// Light flags the host derives at compile (src/luisa/path_tracer_scene.cpp:1787-1830):
// the effective use_mis (MIS only for lamps with a finite extent) and
// whether BSDF / camera rays can hit the lamp.
constexpr uint32_t kLightFlagUseMis = 1u << 30;
constexpr uint32_t kLightFlagForward = 1u << 31;

// Child links and traversal-stack entries: an inner node (global index), an
// instance to enter, the marker that returns to the world ray, the end of
// the traversal, or -- only as a child link -- a leaf triangle.  An empty
// child slot holds kInvalidId.
constexpr uint32_t kLinkInstance = 1u << 30, kLinkLeaf = 1u << 31;
constexpr uint32_t kLinkLeave = kLinkLeaf - 1u, kLinkDone = kLinkLeaf - 2u;
// Entries of the per-ray traversal stack.  Scene compile proves, from the
// built trees, that no ray can push more (see blas_stack_need /
// tlas_instance_depths in psy_host.cpp), rebuilding a mesh with median
// splits or rejecting the scene where needed; a debug build
// (-DPSY_STACK_CHECK=1) also counts pushes that would not fit on the device.
constexpr uint32_t kTraversalStackSize = 48u;
constexpr uint32_t kGgxETableSize = 32u * 32u, kGgxEavgTableSize = 32u;

// Four children of a wide BVH node in two 32-byte sectors, so one ray reads
// it with two 256-bit loads.  Child k's box is stored as one byte per plane:
// byte b stands for the float of bits 0x3f000000 | b << 16, a factor f of
// 0.5 + b / 256 below 1 and 1 + (b - 128) / 128 from there on, and for the
// plane base + span * f.  The host rounds the planes
// outward, with a margin for the rounding of the slab test (see quantise in
// psy_host.cpp).  Leaf children come first; their triangles follow one
// another, so slot k's is the first slot's plus k.
struct alignas(32) NodeGpu {
    float base[3], span[3];
    uint32_t lox, hix, loy, hiy, loz, hiz;  // byte k: child k
    uint32_t link[4];
};
static_assert(sizeof(NodeGpu) == 64, "a node is two 32-byte sectors");

// A padded float box: of a node as its parent's child (what its bytes there
// enclose; only closest_exact in psy_kernels.cu reads it), or of an instance in
// the world.
struct alignas(32) BoxGpu {
    float lo[3], hi[3];
    uint32_t slot;  // a node's place among its parent's children as built (leaves come first in NodeGpu)
    uint32_t pad;
};
static_assert(sizeof(BoxGpu) == 32, "a box is one 32-byte sector");

// A leaf triangle (object space) and its padded float box in two sectors.
struct alignas(32) TriGpu {
    float4 v0;        // w: local primitive index bits
    float4 v1, v2;    // w: box lo.x, lo.y
    float4 lo_z_hi;   // box lo.z, hi.x, hi.y, hi.z
};
static_assert(sizeof(TriGpu) == 64, "a triangle is two 32-byte sectors");

// What a ray needs to enter an instance, in two sectors.
struct alignas(32) EntryGpu {
    float w2o[12];
    uint32_t root;         // root node of the mesh
    uint32_t prim_offset;  // Cycles primitive id of local primitive 0
    uint32_t visibility;
    uint32_t material;  // as InstanceGpu::material
};
static_assert(sizeof(EntryGpu) == 64, "an instance entry is two 32-byte sectors");

// An instance as shading reads it: three sectors for the hit point, two for
// the object-space ray of a new origin.
struct alignas(32) InstanceGpu {
    float o2w[12];  // column-major c0, c1, c2, c3 (xyz each)
    float nrm[9];   // normal-to-world columns
    uint32_t prim_offset;  // Cycles primitive id of local primitive 0
    uint32_t smooth;
    uint32_t material;  // of the whole instance, with kMaterialTransparent; kInvalidId: per triangle
    float w2o[12];
    uint32_t mesh, visibility, pad[2];
};
static_assert(sizeof(InstanceGpu) == 160, "an instance is five 32-byte sectors");
// Set beside a material index whose program has transparent closures.
constexpr uint32_t kMaterialTransparent = 1u << 31;

// A triangle as shading reads it, in Cycles primitive order: three sectors
// instead of a gather through the index, position and normal arrays.
struct alignas(32) ShadeTriGpu {
    float p0[3], p1[3], p2[3];  // object space
    float n0[3], n1[3], n2[3];  // vertex normals (smooth meshes)
    float ng[3];                // normalised geometric normal
    uint32_t material;          // with kMaterialTransparent; kInvalidId: the instance's
    uint32_t pad[2];
};
static_assert(sizeof(ShadeTriGpu) == 96, "a shading triangle is three 32-byte sectors");

// A mesh while its triangle records are packed (k_pack_triangles).
struct alignas(16) MeshGpu {
    uint32_t tri_offset;  // first leaf triangle in `tris`, also the Cycles primitive id of local primitive 0
    uint32_t vertex_offset;    // into positions / normals (vertices)
    uint32_t index_offset;     // into indices (uint32 elements)
    uint32_t material_offset;  // into the triangle materials, kInvalid = instance material
    uint32_t smooth, pad[3];
};

struct alignas(16) MaterialGpu {
    uint32_t code_offset, code_count, root, scalar_offset;
    uint32_t vector_offset, emission_sampling, has_emission, has_transparent;
    uint32_t value_offset, value_count;
    uint32_t bump_correction;  // contract::Material::use_bump_map_correction
    uint32_t closure_first;    // first of the material's baked closures
};

// A material's closure program evaluated: nothing in it depends on the
// shading point (no textures or context values), so k_bake_materials walks
// it once when the scene is compiled or the material's parameters are
// edited, and shading reads the result.
struct alignas(16) BakedMaterialGpu {
    float4 emission;    // xyz: summed emission; w: bits of the first baked closure's index
    float4 extinction;  // xyz: summed transparent weight (a shadow ray's factor); w: bits of the closure count
    uint32_t runtime;   // the closures' runtime flags
    uint32_t emission_sampling, has_emission, bump_correction;
};
// A BSDF closure of the shading point's list, up to what its normal and side
// add (glossy normals, the IOR of a back face, MULTI_GGX's energy factors).
struct alignas(16) BakedClosureGpu {
    float4 weight;  // w: sample weight
    float4 color;   // w: op bits
    float4 params;  // roughness, IOR, IOR of a back face, F0
};

// Value instructions a material's program may hold (its stream is
// evaluated into a per-thread array of this many entries).
constexpr uint32_t kMaxValues = 64u;

struct alignas(16) EmitterGpu {
    float p0[3], p1[3], p2[3], ng[3];
    float area;
    uint32_t material, object, cycles_prim;
    uint32_t emission_sampling, pad0, pad1, pad2;
};

struct alignas(16) DistEntryGpu {
    float cumulative, selection_pdf;
    uint32_t kind, index;
};

// Per-lamp constants of analytic_light_sampling.h that depend on the lamp
// alone, computed once on the host with the kernels' float expressions
// (transcendentals in double, rounded once): the inverse of the spot axes
// (spot_light_to_local, :309-329) with cos(spot_angle / 2) and the smooth
// blend (:331-345), the spot spread cap (:355-376), point_eval_factor
// (:880-896), and the distant lamp's cone and eval factor (:84-108).
struct alignas(16) LampConstGpu {
    float4 spot_rx;  // xyz: first row of the inverse spot axes; w: cos(spot_angle / 2)
    float4 spot_ry;  // w: (1 - cos(spot_angle / 2)) * spot_smooth
    float4 spot_rz;  // w: one minus cosine of the spot's spread cone
    float4 factors;  // x: point eval factor, y: distant cone one minus cosine, z: distant eval factor
};

struct SceneView {
    const NodeGpu *nodes;  // the instance tree from node 0, then every mesh's tree
    const BoxGpu *node_boxes;      // one per node
    const BoxGpu *instance_boxes;  // one per instance
    const TriGpu *tris;
    const EntryGpu *entries;  // one per instance
    const InstanceGpu *instances;
    const ShadeTriGpu *shade_tris;
    const MaterialGpu *materials;
    const BakedMaterialGpu *baked;    // one per material
    const BakedClosureGpu *closures;
    const psy_closure_instruction *code;
    const psy_value_instruction *values;
    const float *scalars;
    const float *vectors;
    const EmitterGpu *emitters;
    const DistEntryGpu *distribution;
    // Cycles' GGX albedo tables (null unless a material has a MULTI_GGX glossy
    // closure): E, 32 rows of incoming cosine x 32 columns of roughness, and
    // its average over the cosine, 32 values of roughness
    const float *ggx_e;
    const float *ggx_eavg;
    const psy_light_desc *lights;
    uint32_t instance_count;
    uint32_t emitter_count;   // distribution entries - 1 (triangles + lights)
    uint32_t triangle_emitters;
    uint32_t light_count;
    // lamps a ray can hit (area lamps, finite point / spot disks) in light
    // order: bounding sphere (centre, radius^2) and light index
    const float4 *lamp_bounds;
    const LampConstGpu *lamp_consts;  // one per light
    float4 world_lo, world_hi;        // bounds of the instances (xyz)
    const uint32_t *lamp_ids;
    uint32_t lamp_count;
    float triangle_area_pdf;
    float light_selection_pdf;
    float background[3];
    uint32_t world_visibility;
    uint32_t any_transparent;
    uint32_t has_glossy;  // a material holds a glossy, glass or refraction closure (selects the shading variant)
    // many-light tree (empty when the scene has no emitter with energy)
    const LtNodeGpu *lt_nodes;
    const LtEmitterGpu *lt_emitters;
    const uint2 *lt_mapping;  // emitter id -> (tree emitter, leaf node)
    const uint4 *lt_lookup;   // sorted (object, primitive, emitter id)
    uint32_t lt_node_count, lt_emitter_count, lt_lookup_count, lt_root;
};

struct RenderParams {
    uint32_t full_w, full_h, win_x, win_y, win_w, win_h;
    uint32_t seed, transparent_background;
    float pass_alpha_threshold;
    uint32_t maximum, minimum, max_diffuse, max_glossy, max_transmission;
    uint32_t transparent_min, transparent_max, steps;
    float clamp_direct, clamp_indirect, inv_rr_threshold;
    uint32_t direct_mode, nee, use_light_tree;
    float cam[12];  // camera_to_world columns c0..c3
    float htan, vtan, shift_x, shift_y, near_clip, far_clip;
    uint32_t projection, aperture_blades, depth_of_field, pad_camera;  // PSY_CAMERA_*; DOF on / off
    float ortho_span, aperture_radius, focal_distance, aperture_ratio, aperture_rotation;
    const float4 *sobol;
    uint32_t sobol_size;
    const float *filter;  // 1024 entries
};

// Wavefront path state, structure of arrays over `capacity` paths.
// The per-path fields every bounce reads and writes share one 128-byte
// record per path, in four 32-byte sectors: ray origin and direction; the
// two state words; throughput and radiance; the hit and its primitive
// (whose sector's other 12 bytes the closest-hit kernel writes as zeros, so
// that it writes whole sectors, and the light tree's picks use).  The shading kernel takes its paths in
// material order, and one cache line per path then replaces a sector in
// each of eight arrays.
constexpr size_t kPathRecordBytes = 128u;
template <class T>
struct PathField {
    unsigned char *base;  // the field in path 0's record
    __host__ __device__ __forceinline__ T &operator[](size_t i) const {
        return *reinterpret_cast<T *>(base + i * kPathRecordBytes);
    }
};
constexpr size_t kRecRayO = 0u, kRecRayD = 16u, kRecSt = 32u, kRecSt2 = 48u, kRecTp = 64u, kRecRad = 80u,
                 kRecHit = 96u, kRecHitPrim = 112u;

struct PathBuffers {
    PathField<float4> ray_o;    // origin, tmin
    PathField<float4> ray_d;    // direction, tmax
    PathField<float4> tp;       // throughput, previous bsdf pdf
    PathField<float4> rad;      // radiance, transparency
    PathField<uint4> st;        // flag, cycles visibility, rng_offset, packed counters
    PathField<uint4> st2;       // transparent bounce | bits, source object, source prim, pixel
    uint32_t *sample;           // absolute sample index
    float4 *aov_n;              // first-surface normal
    float4 *aov_a;              // albedo
    float4 *mis_n;              // shading normal of the last non-transparent scatter (light-tree MIS)
    PathField<float4> hit;      // t, u, v, instance bits
    PathField<uint4> hit_prim;  // x: primitive (kInvalid on a miss); y, z, w: the light tree's pick (entry of the
                                // distribution or kInvalid), its pdf, the forward pdf
    float4 *rad_final;          // radiance and transparency of an ended path (the film reads these
                                // coalesced instead of a 16-byte field of each 128-byte record)
    float4 *sh_o;     // shadow origin, tmax
    float4 *sh_d;     // shadow direction, transparent depth bits
    float4 *sh_c;     // unshadowed contribution
    uint4 *sh_ids;    // source object, source prim, light object, light prim
    uint32_t *sh_path;
    uint32_t *queue_in;
    uint32_t *queue_out;
    uint32_t *ambiguous;  // paths whose closest hit depends on the order of visits
    uint32_t *counters;  // [0] in count, [1] out count, [2] shadow count, [3..4] fetch cursors, [kCounterMisses],
                         // [kCounterTail], [kCounterAmbiguous],
                         // [kCounterWaveGlossy] a batched wavefront's glossy flag
    uint32_t *job;       // batched wavefronts: the job of each path
    // shading-queue sort by material: per-queue-entry bucket, the sorted
    // queue, and kSortBuckets-word histogram / offset arrays
    uint32_t *sort_keys, *queue_sorted, *sort_hist, *sort_offsets;
};

constexpr uint32_t kSortBuckets = 2048u;
constexpr uint32_t kCounterMisses = 5u;  // misses at the front of a sorted shading queue
// 1 + the step from which the queue is k_tail's; 0 before that
constexpr uint32_t kCounterTail = 6u;
constexpr uint32_t kCounterAmbiguous = 7u;  // paths in PathBuffers::ambiguous
constexpr uint32_t kCounterWaveGlossy = 8u;
constexpr uint32_t kCounterWaveTree = 9u;  // a job of the batched wavefront uses its light tree
// sh_path top bit: the shadow ray's path has ended, its contribution goes to rad_final
constexpr uint32_t kShadowFinal = 0x80000000u;

// One job of a batched wavefront: a session's render parameters, its scene
// and its film.  Paths of many jobs share the path state; each path reads
// its job's record.
struct alignas(16) JobGpu {
    RenderParams p;
    SceneView s;
    float4 *combined, *normal, *albedo;
    uint32_t *sample_count;
};

// A block of paths of one job in a batched wavefront: samples
// [sample_base, sample_base + samples) over the job's `pixels` window
// pixels, laid out sample-major from path_begin.  film_begin is the item's
// first pixel in the batch-wide pixel numbering the film kernel walks.
struct BatchItem {
    uint32_t job, path_begin, pixels, samples, sample_base, film_begin, pad0, pad1;
};

// Packed counters of st.w: bounce | diffuse << 8 | glossy << 16 | transmission << 24.
// st2.x: transparent bounce (bits 0-7), previous_delta (8), primary_recorded
// (9), terminate_on_next_surface (10), terminate_after_transparent (11).
constexpr uint32_t kSt2Delta = 1u << 8, kSt2Primary = 1u << 9, kSt2TermNext = 1u << 10, kSt2TermAfter = 1u << 11;

}  // namespace psy
