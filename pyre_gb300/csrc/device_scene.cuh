// device_scene.cuh — scene layout in HBM and ray traversal (closest / any hit).
//
// Layout (all arrays device-resident, built once by pyre_scene_upload):
//   nodes               64-B trace nodes (see "binary traversal" below): every
//                       mesh BVH (collapsed from the reference BVH2), then the
//                       top-level BVH over instances
//   tris   float4[3*T]  per triangle slot, in BVH leaf order:
//                       (v0.xyz, original triangle id as bits),
//                       (e1.xyz, instance slot as bits, -1 where several instances use the mesh),
//                       (e2.xyz, 1 as bits in the last triangle of a leaf)
//                       with e1 = v1 - v0, e2 = v2 - v0 rounded exactly as
//                       moller_trumbore computes them (mesh.rs:153-157)
//   inst   DevInstance[] instances in top-level-leaf order
//   index  uint32[3*T]  mesh index buffers rebased to global vertex ids
//   slot_normals float4[3*T] per triangle slot, its three vertex normals (for shading)
//   normal float[3*V]   vertex normals (meshes without normals use e1 x e2)
#pragma once
#include <cuda_runtime.h>
#include "pyre_math.cuh"

#ifndef PYRE_WIDE_FIELDS
#define PYRE_WIDE_FIELDS 8  // fields of a wide node: 6 box planes, child, count
#endif

namespace pyre {

struct alignas(16) DevInstance {
    float lo[3];  // BLAS root box (the reference tests it first, bvh.rs:103-110)
    int32_t blas_root;  // device node index, -1 for an empty mesh
    float hi[3];
    int32_t has_motion;
    float off0[3];
    int32_t orig_id;    // index in Scene::primitives
    float off1[3];
    int32_t more;       // the top-level leaf holds the next slot too
    uint32_t material;
    uint32_t index_base;   // first index (3 per triangle) of the mesh in `index`
    int32_t normal_base;   // first vertex of the mesh's normals, -1 if none
    uint32_t hang;         // PYRE_HANG_*: how the binary traversal reaches it
};

// A static instance with a top-level leaf of its own: that leaf holds its root
// box, whose test is the reference's root test, and the traversal steps its root
// node next. DIRECT: no other instance uses the mesh, and the root hangs below
// the top level without any entry.
#define PYRE_HANG_ENTRY 0u   // moving, or in a leaf of several instances
#define PYRE_HANG_STATIC 1u
#define PYRE_HANG_DIRECT 2u

// A material and what the BSDF derives from it alone (make_material), 64 B.
struct alignas(64) DevMaterial {
    float base[3];
    uint32_t kind;
    float metallic, roughness, specular;
    float alpha;   // GGX alpha
    float kd[3];   // base (1 - metallic) / pi; Lambertian: albedo / pi
    float pd;      // probability of the diffuse lobe
    float f0[3];   // specular reflectance at normal incidence
    float ps;      // probability of the specular lobe
};

struct DevQuadLight {
    f3 p0, edge_u, edge_v, crs, normal, emission;
    float inv_cross_len_sq, area;
};

struct DevEnv {
    uint32_t width, height;
    float intensity;
    const float4* pixels;      // w*h, rgb + pad
    const float* marg_cdf;     // h+1
    const float* cond_cdf;     // h*(w+1)
    const float* marg_pdf;     // h: (cdf[b+1]-cdf[b])*h
    const float* cond_pdf;     // h*w
    const float2* marg_alias;  // h: (prob, alias as bits)
    const float2* cond_alias;  // h*w
};

struct DevScene {
    const float4* nodes;   // trace nodes, 4 float4 each; for the wide traversals the top level's GpuNodes
    const float4* tris;
    const DevInstance* inst;
    uint32_t n_inst;
    int32_t tlas_root;     // -1: no geometry
    const uint32_t* index;
    const float* normal;
    const float4* slot_normals;  // 3 per triangle slot: its vertex normals (xyz, 0)
    const DevMaterial* materials;
    uint32_t n_materials;
    const DevQuadLight* lights;
    uint32_t n_lights;
    int has_env;
    DevEnv env;
    int* error_flag;       // set to PYRE_ERR_OVERFLOW by a kernel that hit a limit
    // sub-scenes of a batch upload (one part for an ordinary scene)
    const int32_t* part_tlas;    // top-level root per part
    const uint32_t* part_light;  // (first light, light count) per part
    uint32_t n_parts;
    // wide BVH of the instances (traversals with WIDTH 4 or 8): wide nodes (8
    // fields x WIDTH floats each) and the wide root of each instance slot. The
    // top level stays binary; for these traversals `nodes` holds it alone, as
    // GpuNodes with instance entries
    const float4* wnodes;
    const int32_t* wroot;
};

struct TraceRay {
    f3 o, d;
    float tmin, tmax, time;
    uint32_t job;  // batched rendering: the ray's job (set and read by the ray source only)
};

struct TraceHit {
    float t, u, v;
    int32_t inst;  // instance slot (device order); -1 = no hit
    int32_t tri;   // triangle slot
    int32_t light; // quad light index when the closest hit is a light, else -1
};

#define PYRE_STACK 64
// lanes of a warp that may still be looking for a leaf when the leaf phase
// starts, for closest-hit and any-hit traversal: 12 / 16 / 20 gave 127.1 /
// 126.9 / 128.0 ms per 1080p studio frame and 2.88 / 2.90 / 3.00 ms on the
// closest-hit microbenchmark
#ifndef PYRE_LEAF_WAIT_CLOSEST
#define PYRE_LEAF_WAIT_CLOSEST 16
#endif
#ifndef PYRE_LEAF_WAIT_ANY
#define PYRE_LEAF_WAIT_ANY 16
#endif
// Node steps a lane takes between two warp votes of the inner phase (a vote, a
// ballot, a population count and an any, costs issue slots): 3 / 4 / 6 gave
// 127.5 / 126.9 / 126.6 ms per 1080p studio frame and 2.93 / 2.90 / 2.87 ms on
// the closest-hit microbenchmark. Wide BVHs, whose steps are longer, take 4:
// the microbenchmark gave 4.33 / 4.35 ms with 4 / 6 at width 4 and 6.21 / 6.32 at
// width 8, a 960x540 studio frame at 16 spp 14.74 / 14.78 and 19.43 / 19.70.
// Films are bit-identical for every setting.
#ifndef PYRE_STEPS_PER_VOTE
#define PYRE_STEPS_PER_VOTE 6
#endif
#define PYRE_STEPS_PER_VOTE_WIDE 4

// 32 B with one load (sm_100+; p is 32-B aligned): half the load instructions
// of 128-bit ones, and of the L1's data cycles where every lane reads a record of
// its own (46.4 against 77.3 cycles per 64-B record of 32 lanes).
__device__ __forceinline__ void ldg_256(const float4* p, float4& a, float4& b) {
    asm("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(p));
}

// 32-B path-state records with one streaming (evict-first) 256-bit load or
// store each; p must be 32-B aligned. The load stays where it is among the
// stores and barriers: k_wave_small reads back what it wrote a depth before.
__device__ __forceinline__ void ldcs_256(const float4* p, float4& a, float4& b) {
    asm volatile("ld.global.cs.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void stcs_256(float4* p, const float4& a, const float4& b) {
    asm volatile("st.global.cs.v8.f32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 :: "l"(p), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
}

// Rust-order slab test (bvh.rs:146-153): t1/t2 per axis, max of mins vs
// t_min, min of maxes vs t_max, hit iff tmin <= tmax. Returns the entry.
__device__ __forceinline__ bool slab(float lox, float hix, float loy, float hiy, float loz, float hiz,
                                     const f3& o, const f3& inv, float tmin_ray, float tmax_cur, float* entry) {
    float t1x = (lox - o.x) * inv.x, t2x = (hix - o.x) * inv.x;
    float t1y = (loy - o.y) * inv.y, t2y = (hiy - o.y) * inv.y;
    float t1z = (loz - o.z) * inv.z, t2z = (hiz - o.z) * inv.z;
    float tmin = fmaxf(fmaxf(fminf(t1x, t2x), fmaxf(fminf(t1y, t2y), fminf(t1z, t2z))), tmin_ray);
    float tmax = fminf(fminf(fmaxf(t1x, t2x), fminf(fmaxf(t1y, t2y), fmaxf(t1z, t2z))), tmax_cur);
    *entry = tmin;
    return tmin <= tmax;
}

// moller_trumbore, crates/pyre/src/geometry/mesh.rs:153-178, without the
// final t-range test (the caller applies it).
__device__ __forceinline__ bool mt_test(const f3& o, const f3& d, const float4& A, const float4& B, const float4& C,
                                        float* t_out, float* u_out, float* v_out) {
    const f3 v0 = mk3(A.x, A.y, A.z), e1 = mk3(B.x, B.y, B.z), e2 = mk3(C.x, C.y, C.z);
    const f3 h = cross3(d, e2);
    const float a = dot3(e1, h);
    if (fabsf(a) < 1e-8f) return false;
    const float f = __frcp_rn(a);
    const f3 s = o - v0;
    const float u = f * dot3(s, h);
    if (!(u >= 0.0f && u <= 1.0f)) return false;
    const f3 q = cross3(s, e1);
    const float v = f * dot3(d, q);
    if (v < 0.0f || u + v > 1.0f) return false;
    *t_out = f * dot3(e2, q);
    *u_out = u;
    *v_out = v;
    return true;
}

__device__ __forceinline__ f3 motion_offset(const DevInstance& I, float time) {
    // InstanceMotion::at (mesh.rs:53-55)
    return lerp3(mk3(I.off0[0], I.off0[1], I.off0[2]), mk3(I.off1[0], I.off1[1], I.off1[2]),
                 clampf_(time, 0.0f, 1.0f));
}

// Ray traversal, closest or any hit, equivalent to the instance scan of
// Scene::intersect / Scene::occluded (scene.rs:57-140) with the canonical tie
// rule. A warp loops over a queue of n rays: the lanes take rays from the
// queue through a shared work counter, and whenever at least `refill` lanes
// have finished their ray (or the warp has none), the idle lanes take new rays
// with one atomic for the warp, so the warp does not run on with a few long
// rays. A ray's traversal does not depend on which lane or warp runs it, so
// the results are the same as one ray per thread.
//
// Src supplies the rays and takes the results (kTmin / kTmax: the t range
// that idle lanes start with; kFixedTmin: every ray's t_min is kTmin):
//   uint32_t load(uint32_t j, TraceRay& r, int32_t& root)  ray j of the queue,
//            the top-level root to trace; returns the id passed to store
//   void store(uint32_t id, const TraceRay& r, TraceHit& h, bool found)
// All 32 lanes of the warp must call it with the same n and counter.
//
// ------------------------------------------------------- binary traversal --
// Trace node (64 B, 64-B aligned, two 256-bit loads): a GpuNode repacked by
// k_pack_nodes at upload so that the slab tests run on packed pairs of floats
//   q0 = (lo0.x, lo0.y)  q1 = (hi0.x, hi0.y)  q2 = (lo1.x, lo1.y)  q3 = (hi1.x, hi1.y)
//   q4 = (lo0.z, hi0.z)  q5 = (lo1.z, hi1.z)  q6 = (ref0, ref1)    q7 = (bias, counts)
// A child reference, which is also a stack entry:
//   >= 0                 interior node (of an instance BVH or the top level)
//   PYRE_REF_LEAF | s    triangles s, s + 1, ... up to the one marked last
//   PYRE_REF_INST | k    enter instance slot k, after its root-box test at the ray's time
//   PYRE_REF_STATIC | k  static instance k, whose root box is this child's: its root is stepped next
// A static instance whose mesh no other instance uses needs no entry: its
// root node hangs directly below the top level (same world space), and its
// triangle records carry its slot. A static one whose mesh others use too is an
// interior child in the visiting order (nearest first) and needs no second box
// test, only its slot noted. Treated like the other entries, it cost rays among
// 512 spheres, each with a second user of its mesh out of their way, 1.54 against
// 1.36 ms of closest hit and 1.24 against 1.15 of any hit (1.26 and 1.07 without
// those users; noting the slot within the step loop gave 1.34 and 1.14 but cost
// every other scene 1 to 3 %). `bias` gives the visiting order of two
// children that are both hit: child 1 first iff e1 < e0 + bias. It is 0 between
// interior children (nearest first) and +-inf where the order is fixed
// (triangles before interior nodes, interior nodes before instance entries,
// otherwise child 0 first). `counts` holds the leaf sizes (16 bits each).
#define PYRE_REF_LEAF ((int)0x80000000)
#define PYRE_REF_INST ((int)0xC0000000)
#define PYRE_REF_STATIC ((int)0xE0000000)
#define PYRE_REF_SLOT 0x3fffffff       // of a leaf
#define PYRE_REF_INST_SLOT 0x1fffffff  // of an instance entry
#define PYRE_REF_LEAVE (-3)  // stack entry below an entered instance: back to world space
#define PYRE_REF_DONE (-2)   // bottom of the stack
#define PYRE_REF_NONE (-1)   // idle lane / no postponed leaf
__device__ __forceinline__ bool ref_is_leaf(int r) { return r < PYRE_REF_INST; }
__device__ __forceinline__ bool ref_is_pending(int r) { return r < PYRE_REF_DONE; }
__device__ __forceinline__ bool ref_is_static(int r) { return r >= PYRE_REF_STATIC && r < PYRE_REF_LEAVE; }

typedef unsigned long long pair32;  // two floats in one 64-bit register pair
__device__ __forceinline__ pair32 pack2(float a, float b) {
    pair32 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(pair32 v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ pair32 add2(pair32 a, pair32 b) {
    pair32 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ pair32 mul2(pair32 a, pair32 b) {
    pair32 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void ldg_4x64(const void* p, pair32& a, pair32& b, pair32& c, pair32& d) {
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];" : "=l"(a), "=l"(b), "=l"(c), "=l"(d) : "l"(p));
}

// The address of q0..q3 of trace node n; q4..q7 sit at that address ^ 32. Nodes
// with bit 1 of their index set hold their halves swapped: otherwise the lanes
// of a warp, each at its own node, would all read offset 0 or 64 of a 128-B
// line with one load and 32 or 96 with the other, half of the L1's banks at a
// time. L1 data cycles bound the traversal once its instructions were halved:
// extend 55.6 against 58.2 ms and shadow 21.4 against 23.1 ms per 1080p studio
// frame, closest-hit queries 2.54 against 2.62 ms. (Random 64-B fetches by 32
// lanes from an L1-resident array: 35.6 against 46.4 cycles; four 128-bit loads
// 77.3.)
#define PYRE_NODE_SWAP(n) ((n) & 2u)
__device__ __forceinline__ uint64_t trace_node_half(const float4* nodes, uint32_t n) {
    return reinterpret_cast<uint64_t>(nodes) + ((uint64_t)n * 64u | (PYRE_NODE_SWAP(n) << 4));
}

// The slab test of `slab`, two planes per instruction: lo - o is lo + (-o) and
// the packed operations round like the scalar ones, so the entries and the
// decisions are the same bits.
__device__ __forceinline__ bool slab2(pair32 loxy, pair32 hixy, pair32 z, pair32 noxy, pair32 nozz, pair32 ixy,
                                      pair32 izz, float tmin_ray, float tmax_cur, float* entry) {
    float t1x, t1y, t2x, t2y, t1z, t2z;
    unpack2(mul2(add2(loxy, noxy), ixy), t1x, t1y);
    unpack2(mul2(add2(hixy, noxy), ixy), t2x, t2y);
    unpack2(mul2(add2(z, nozz), izz), t1z, t2z);
    const float tmin = fmaxf(fmaxf(fminf(t1x, t2x), fmaxf(fminf(t1y, t2y), fminf(t1z, t2z))), tmin_ray);
    const float tmax = fminf(fminf(fmaxf(t1x, t2x), fminf(fmaxf(t1y, t2y), fmaxf(t1z, t2z))), tmax_cur);
    *entry = tmin;
    return tmin <= tmax;
}

// trace_binary: the warp loop over the packed binary nodes. A lane's whole state is one reference: the node it steps next,
// the leaf or instance entry it waits with, DONE, or NONE (idle). The visiting
// order of a ray is that of the reference's boxes and depends on nothing but
// the ray: children nearest first, a node's leaves before its interior child,
// and a closest-hit lane tests a leaf before its next node step (an any-hit
// lane, whose result does not depend on the order, keeps stepping with one
// leaf postponed).
// What a ray needs only now and then sits in shared memory, one column per
// thread: its world origin (leaving an instance, quad lights), direction (leaf
// tests), time and the current hit. That leaves 10 resident blocks per SM
// their 48 registers.
//
// Bound by the L1's data cycles (three quarters of their peak) and load latency;
// issue slots are 60 % busy with 12 to 16 lanes. Against the loop it replaced
// (scalar slab tests; leaf ranges, tags and counts in registers; every
// instance behind an entry of its own), same bits: extend 61.4 against 81.0 ms
// and shadow 23.5 against 30.8 ms per 1080p studio frame (125.7 against 152.7 ms
// in all), closest hit 2.93 against 3.65 ms and any hit 0.40 against 0.50 ms on
// the ray cases, the Cornell preset at 800x600 and 16 spp 6.82 against 8.59 ms.
// A warp that needs rays takes a share of the queue: consecutive rays, which
// start close together, so that what one ray brought into L1 serves the next.
// A share is at most PYRE_SHARE rays and a 64th of what a warp gets on average,
// whole warps of it; below that a warp takes what its idle lanes need, and the
// last rays of the queue stay spread over all warps. On the 1080p studio frame
// (133 M camera rays) 118.6 ms against 119.8 without shares; the Cornell preset
// at 800x600 (7.7 M camera rays) 6.10 with a 32nd, 6.05 with a 64th, 6.04 without.
#ifndef PYRE_SHARE
#define PYRE_SHARE 128
#endif
// Bottom entries of a lane's stack kept in shared memory (entry-major, so a
// lane always uses its own bank), the rest in local memory, whose lines the
// nodes push out of L1 (26 % of the stack loads hit): 0 / 4 / 8 / 12 / 16
// entries gave 62.4 / 61.6 / 60.0 / 59.8 / 59.8 ms of extend per 1080p studio
// frame and 2.82 / 2.76 / 2.63 / 2.62 / 2.63 ms of closest-hit queries.
#ifndef PYRE_STACK_SHARED
#define PYRE_STACK_SHARED 12
#endif
// Shared memory of a block of at most 128 threads (a closest-hit kernel's, or
// an any-hit kernel's, which keeps no hit).
template <bool ANY>
struct TraceShared {
    int stack[PYRE_STACK_SHARED][128];  // bottom entries of the stacks
    float ray[8][128];                  // o, d, time, job
    int hit[ANY ? 1 : 4][128];          // u, v, instance slot, triangle slot
};
// Who traces a queue: warp `warp` of `warps` (all others of the grid stay
// out). With `deal`, the queue holds less than 32 rays for each of them and is
// dealt out evenly: a warp runs the union of its rays' steps, so the launch's
// time is that of its fullest warp, and no warp waits for the counter. Short
// queues (the viewer's, a large wave's last bounces) are bound by that latency.
struct TraceTeam {
    uint32_t warp, warps;
    bool deal;
};
__device__ __forceinline__ TraceTeam whole_grid(uint32_t n) {
    TraceTeam t;
    t.warps = gridDim.x * (blockDim.x >> 5);
    t.warp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    t.deal = n < 32u * t.warps;
    return t;
}

template <bool ANY, class Src>
__device__ __forceinline__ void trace_binary(const DevScene& S, const Src& src, uint32_t n, uint32_t* counter,
                                             int refill, const TraceTeam& team, int (*sstack)[128], float (*sray)[128],
                                             int (*shit)[128]) {
    constexpr int LEAF_WAIT = ANY ? PYRE_LEAF_WAIT_ANY : PYRE_LEAF_WAIT_CLOSEST;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lanes_below = (1u << lane) - 1u;
    // 64 nodes, as deep as before, plus the bottom, an instance's exit, and a
    // leaf's sibling waiting for the leaf
    constexpr int STACK = PYRE_STACK + 4;
    constexpr int SK = PYRE_STACK_SHARED;
    const int tid = threadIdx.x;
    int stack[STACK - SK + 1];  // + 1: the node that waits while a postponed leaf is tested
    int sp = 0;
    auto spush = [&](int v) {
        if (sp < SK) sstack[sp][tid] = v;
        else stack[sp - SK] = v;
        ++sp;
    };
    auto spop = [&]() -> int {
        --sp;
        return sp < SK ? sstack[sp][tid] : stack[sp - SK];
    };
    bool drained = false;         // warp-uniform: the counter has no rays left
    uint32_t next = 0, end = 0;   // warp-uniform: the rest of the warp's share of the queue
    if (team.deal) {
        const uint32_t slice = (n + team.warps - 1) / team.warps;
        next = min(team.warp * slice, n);
        end = min(next + slice, n);
        drained = true;
    }
    const uint32_t share = min((uint32_t)PYRE_SHARE, n / (team.warps * 64u) & ~31u);
    uint32_t id = 0;
    int node = PYRE_REF_NONE;
    int postponed = PYRE_REF_NONE;  // any hit: a leaf met while stepping on
    int inst = -1;                  // instance entered through an INST reference
    float tmin = Src::kTmin, best_t = 0.0f;
    pair32 noxy = 0, nozz = 0, ixy = 0, izz = 0;  // -origin and 1 / direction
    bool hit_any = false;

    while (true) {
        // ---- refill idle lanes from the queue
        if (!drained || next < end) {
            const unsigned idle = __ballot_sync(FULL, node == PYRE_REF_NONE);
            const int n_idle = __popc(idle);
            if (n_idle >= refill || n_idle == 32) {
                const uint32_t avail = end - next, rank = (uint32_t)__popc(idle & lanes_below);
                uint32_t j = next + rank, stop = end;
                next += min((uint32_t)n_idle, avail);
                if ((uint32_t)n_idle > avail && !drained) {  // the rest of the idle lanes start the warp's next share
                    const uint32_t need = (uint32_t)n_idle - avail, take = max(share, need);
                    uint32_t base = 0;
                    if (lane == 0) base = atomicAdd(counter, take);
                    base = __shfl_sync(FULL, base, 0);
                    if ((uint64_t)base + take >= (uint64_t)n) drained = true;
                    base = min(base, n);
                    end = min(base + take, n);
                    if (rank >= avail) { j = base + (rank - avail); stop = end; }
                    next = min(base + need, end);
                }
                if (node == PYRE_REF_NONE && j < stop) {
                    int32_t root;
                    TraceRay r;
                    id = src.load(j, r, root);
                    sray[0][tid] = r.o.x; sray[1][tid] = r.o.y; sray[2][tid] = r.o.z;
                    sray[3][tid] = r.d.x; sray[4][tid] = r.d.y; sray[5][tid] = r.d.z;
                    sray[6][tid] = r.time; sray[7][tid] = __uint_as_float(r.job);
                    noxy = pack2(-r.o.x, -r.o.y);
                    nozz = pack2(-r.o.z, -r.o.z);
                    const float iz = __frcp_rn(r.d.z);
                    ixy = pack2(__frcp_rn(r.d.x), __frcp_rn(r.d.y));
                    izz = pack2(iz, iz);
                    if (!Src::kFixedTmin) tmin = r.tmin;
                    best_t = r.tmax;
                    hit_any = false;
                    if (!ANY) { shit[0][tid] = 0; shit[ANY ? 0 : 1][tid] = 0; shit[ANY ? 0 : 2][tid] = -1; shit[ANY ? 0 : 3][tid] = -1; }
                    inst = -1;
                    sp = 0;
                    spush(PYRE_REF_DONE);
                    node = root < 0 ? PYRE_REF_DONE : root;
                }
            }
        }
        if (!__any_sync(FULL, node != PYRE_REF_NONE)) {
            if (drained && next == end) break;
            continue;
        }
        // ---- inner phase: step nodes until at most LEAF_WAIT lanes still
        // look for a leaf and some lane holds one
        while (true) {
            const bool seeks = node >= 0 && (!ANY || postponed == PYRE_REF_NONE);
            const int seeking = __popc(__ballot_sync(FULL, seeks));
            if (seeking == 0) break;
            if (seeking <= LEAF_WAIT &&
                __any_sync(FULL, ref_is_pending(node) || (ANY && postponed != PYRE_REF_NONE)))
                break;
#pragma unroll 1
            for (int step = 0; step < PYRE_STEPS_PER_VOTE; ++step) {
                if (node < 0) break;
                const uint64_t N = trace_node_half(S.nodes, (uint32_t)node);
                pair32 q0, q1, q2, q3, q4, q5, q6, q7;
                ldg_4x64(reinterpret_cast<const void*>(N), q0, q1, q2, q3);
                ldg_4x64(reinterpret_cast<const void*>(N ^ 32u), q4, q5, q6, q7);
                float e0, e1;
                const bool h0 = slab2(q0, q1, q4, noxy, nozz, ixy, izz, tmin, best_t, &e0);
                const bool h1 = slab2(q2, q3, q5, noxy, nozz, ixy, izz, tmin, best_t, &e1);
                const int r0 = (int)(uint32_t)q6, r1 = (int)(uint32_t)(q6 >> 32);
                if (h0 && h1) {
                    const bool swap = e1 < e0 + __uint_as_float((uint32_t)q7);
                    if (sp >= STACK) { atomicExch(S.error_flag, -5); node = PYRE_REF_DONE; break; }
                    spush(swap ? r0 : r1);
                    node = swap ? r1 : r0;
                } else if (h0 || h1) {
                    node = h0 ? r0 : r1;
                } else {
                    node = spop();
                }
                if (ANY && ref_is_leaf(node) && postponed == PYRE_REF_NONE) {
                    postponed = node;
                    node = spop();
                }
            }
        }
        // ---- leaf phase: the lanes that hold a leaf test its triangles
        if (ANY && postponed != PYRE_REF_NONE) {  // the postponed leaf first; the stack has room: its entry came off it
            spush(node);
            node = postponed;
            postponed = PYRE_REF_NONE;
        }
        if (ref_is_leaf(node)) {
            float ox, oy, oz, oz2;
            unpack2(noxy, ox, oy);
            unpack2(nozz, oz, oz2);
            const f3 o = mk3(-ox, -oy, -oz), d = mk3(sray[3][tid], sray[4][tid], sray[5][tid]);
            do {
                const int slot = node & PYRE_REF_SLOT;
                const float4 A = __ldg(S.tris + 3 * (size_t)slot), B = __ldg(S.tris + 3 * (size_t)slot + 1),
                             C = __ldg(S.tris + 3 * (size_t)slot + 2);
                float t, u, v;
                if (mt_test(o, d, A, B, C, &t, &u, &v) && t > tmin) {
                    if (ANY) {
                        if (t < best_t) { hit_any = true; node = PYRE_REF_DONE; break; }
                    } else {
                        const int own = __float_as_int(B.w);
                        const int at = own >= 0 ? own : inst;
                        bool better = t < best_t;
                        if (!better && t == best_t && shit[ANY ? 0 : 3][tid] >= 0) {
                            // a tie (rare): the lower Scene::primitives index, then the lower
                            // triangle id, wins; both are read back from the records
                            const int32_t cur = S.inst[at].orig_id, best = S.inst[shit[ANY ? 0 : 2][tid]].orig_id;
                            const uint32_t key = __float_as_uint(A.w);
                            const uint32_t best_key = __float_as_uint(__ldg(S.tris + 3 * (size_t)shit[ANY ? 0 : 3][tid]).w);
                            better = cur < best || (cur == best && key < best_key);
                        }
                        if (better) {
                            best_t = t;
                            shit[0][tid] = __float_as_int(u); shit[ANY ? 0 : 1][tid] = __float_as_int(v);
                            shit[ANY ? 0 : 2][tid] = at; shit[ANY ? 0 : 3][tid] = slot;
                        }
                    }
                }
                node = __float_as_uint(C.w) != 0u ? spop() : node + 1;
            } while (ref_is_leaf(node));
        }
        // ---- instance entries: the reference's root-box test at the ray's time
        if (ref_is_pending(node) && !ref_is_leaf(node)) {
            const f3 wo = mk3(sray[0][tid], sray[1][tid], sray[2][tid]);
            if (node == PYRE_REF_LEAVE) {
                noxy = pack2(-wo.x, -wo.y);
                nozz = pack2(-wo.z, -wo.z);
                inst = -1;
                node = spop();
            } else if (ref_is_static(node)) {
                inst = node & PYRE_REF_INST_SLOT;
                node = S.inst[inst].blas_root;
            } else {
                const int k = node & PYRE_REF_INST_SLOT;
                const DevInstance& I = S.inst[k];
                if (sp + 2 > STACK) { atomicExch(S.error_flag, -5); node = PYRE_REF_DONE; }
                else {
                    if (I.more) spush(PYRE_REF_INST | (k + 1));
                    f3 lo = wo;
                    if (I.has_motion) {
                        const f3 off = motion_offset(I, sray[6][tid]);
                        if (!is_zero3(off)) lo = wo - off;
                    }
                    float ix, iy, iz, iz2, e;
                    unpack2(ixy, ix, iy);
                    unpack2(izz, iz, iz2);
                    if (I.blas_root >= 0 && slab(I.lo[0], I.hi[0], I.lo[1], I.hi[1], I.lo[2], I.hi[2], lo,
                                                 mk3(ix, iy, iz), tmin, best_t, &e)) {
                        spush(PYRE_REF_LEAVE);
                        inst = k;
                        noxy = pack2(-lo.x, -lo.y);
                        nozz = pack2(-lo.z, -lo.z);
                        node = I.blas_root;
                    } else {
                        node = spop();
                    }
                }
            }
        }
        // ---- finished rays hand over their result; the lane becomes idle
        if (node == PYRE_REF_DONE) {
            TraceRay r;
            r.o = mk3(sray[0][tid], sray[1][tid], sray[2][tid]);
            r.d = mk3(sray[3][tid], sray[4][tid], sray[5][tid]);
            r.tmin = tmin;
            r.tmax = best_t;  // read only where nothing was hit: then the ray's own
            r.time = sray[6][tid];
            r.job = __float_as_uint(sray[7][tid]);
            TraceHit hit;
            hit.t = best_t;
            hit.light = -1;
            hit.u = hit.v = 0.0f;
            hit.inst = hit.tri = -1;
            bool found = hit_any;
            if (!ANY) {
                hit.u = __int_as_float(shit[0][tid]); hit.v = __int_as_float(shit[ANY ? 0 : 1][tid]);
                hit.inst = shit[ANY ? 0 : 2][tid]; hit.tri = shit[ANY ? 0 : 3][tid];
                found = hit.tri >= 0;
            }
            src.store(id, r, hit, found);
            node = PYRE_REF_NONE;
        }
    }
}


// --------------------------------------------------------- wide traversal --
// Instance BVHs of width 4 or 8 below a binary top level. Each lane keeps one
// tagged stack:
//   [0, 2^28)          node of an instance BVH
//   LEAF | n*W + k     leaf child k of wide node n
//   TOP | n            node of the top-level BVH
//   INST | slot        enter instance `slot` (root-box test, local origin)
//   INST | TOP | slot  enter static instance `slot`, whose root box the
//                      top-level step already tested
// A lane inside an instance leaves it (restores the world origin) when it
// reaches the next TOP or INST entry: those lie below the instance's nodes. A
// node step tests every child box, continues with the nearest hit child and
// pushes the others farthest first; leaf children are parked when they are
// reached (an any-hit lane keeps up to three parked triangle ranges, a
// closest-hit lane waits with its first) and tested by all lanes in lock step.
#define PYRE_TAG_LEAF (1 << 28)
#define PYRE_TAG_TOP (1 << 29)
#define PYRE_TAG_INST (1 << 30)
#define PYRE_NODE_NONE (-1)
// Compare-exchange of (entry distance, stack entry) pairs, ascending.
__device__ __forceinline__ void cmp_swap(float& ea, int& na, float& eb, int& nb) {
    const bool sw = eb < ea;
    const float e = sw ? eb : ea;
    const int m = sw ? nb : na;
    eb = sw ? ea : eb;
    nb = sw ? na : nb;
    ea = e;
    na = m;
}
template <int W>
__device__ __forceinline__ void sort_children(float (&e)[W], int (&c)[W]) {
    if (W == 4) {  // optimal 5-comparator network
        cmp_swap(e[0], c[0], e[1], c[1]); cmp_swap(e[2], c[2], e[3], c[3]);
        cmp_swap(e[0], c[0], e[2], c[2]); cmp_swap(e[1], c[1], e[3], c[3]);
        cmp_swap(e[1], c[1], e[2], c[2]);
    } else {  // optimal 19-comparator network for 8
        constexpr int net[19][2] = {{0, 2}, {1, 3}, {4, 6}, {5, 7}, {0, 4}, {1, 5}, {2, 6}, {3, 7}, {0, 1}, {2, 3},
                                    {4, 5}, {6, 7}, {2, 4}, {3, 5}, {1, 4}, {3, 6}, {1, 2}, {3, 4}, {5, 6}};
#pragma unroll
        for (int q = 0; q < 19; ++q) cmp_swap(e[net[q][0]], c[net[q][0]], e[net[q][1]], c[net[q][1]]);
    }
}

template <bool ANY, int WIDTH, class Src>
__device__ __forceinline__ void trace_wide(const DevScene& S, const Src& src, uint32_t n, uint32_t* counter,
                                             int refill) {
    // A lane stops stepping nodes once it holds STOP parked leaves. A
    // closest-hit lane stops at its first: its leaves are then tested before its next node step, so
    // the boxes it culls with its current closest distance, and its hit, do
    // not depend on the other lanes of its warp. Where two triangles are hit
    // at distances a rounding apart, a box whose rounded entry lies between
    // them is culled or not depending on when the nearer hit was recorded;
    // with speculative steps that point moved with the warp, and about one
    // pixel in 10^6 of 1024^2 Cornell views changed from run to run. Any hit
    // culls with the ray's own fixed t_max, so its lanes keep stepping.
    static_assert(WIDTH > 2, "binary BVHs are traced by trace_binary");
    constexpr int STOP = ANY ? 3 : 1;
    constexpr int LEAF_WAIT = ANY ? PYRE_LEAF_WAIT_ANY : PYRE_LEAF_WAIT_CLOSEST;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lanes_below = (1u << lane) - 1u;
    bool drained = false;   // warp-uniform: the queue has no rays left
    bool active = false;    // the lane holds a ray
    uint32_t id = 0;
    TraceRay r;
    r.o = splat3(0.0f); r.d = mk3(0.0f, 0.0f, 1.0f); r.time = 0.0f; r.job = 0;
    r.tmin = Src::kTmin; r.tmax = Src::kTmax;  // a source whose rays share one range makes it a constant
    TraceHit hit;
    hit.inst = -1; hit.tri = -1; hit.light = -1; hit.t = 0.0f; hit.u = 0.0f; hit.v = 0.0f;
    f3 inv = splat3(0.0f);
    float best_t = 0.0f;
    bool found = false;
    bool hit_any = false;    // any-hit: the ray is occluded
    bool exhausted = true;   // no node left to step
    // an 8-wide step can push 7 entries, so the 8-wide stack is deeper
    constexpr int STACK = WIDTH == 8 ? 96 : PYRE_STACK;
    // Any-hit traversal keeps the bottom 8 stack entries of each lane in
    // shared memory (entry-major, so a lane always uses its own bank), the
    // rest in local memory: the shadow stage is 4 % faster on the 1080p frame
    // (4 or 12 entries are slower than 8).
    // Closest hit keeps the whole stack in local memory; with the same short
    // stack it was 0.6 % slower (4 entries), 2 % (8) and 4 % (16).
    constexpr int SK = ANY ? 8 : 0;
    __shared__ int sstack[SK > 0 ? SK : 1][128];  // traversal blocks have at most 128 threads
    int stack[STACK - SK];
    int sp = 0;
    auto spush = [&](int v) {
        if (SK > 0 && sp < SK) sstack[sp][threadIdx.x] = v;
        else stack[sp - SK] = v;
        ++sp;
    };
    auto spop = [&]() -> int {
        --sp;
        return (SK > 0 && sp < SK) ? sstack[sp][threadIdx.x] : stack[sp - SK];
    };
    int node = PYRE_NODE_NONE;
    int inst = -1;
    f3 o = r.o;
    constexpr int PR = ANY ? 3 : 2;
    int ls[PR], lc[PR];
#pragma unroll
    for (int q = 0; q < PR; ++q) { ls[q] = 0; lc[q] = 0; }
    int parked = 0;

    while (true) {
        // ---- refill idle lanes from the queue
        if (!drained) {
            const unsigned idle = __ballot_sync(FULL, !active);
            const int n_idle = __popc(idle);
            if (n_idle >= refill || n_idle == 32) {
                const int leader = __ffs(idle) - 1;
                uint32_t base = 0;
                if (lane == leader) base = atomicAdd(counter, (uint32_t)n_idle);
                base = __shfl_sync(FULL, base, leader);
                if ((uint64_t)base + (uint64_t)n_idle >= (uint64_t)n) drained = true;
                const uint32_t j = base + (uint32_t)__popc(idle & lanes_below);
                if (!active && j < n) {
                    int32_t root;
                    id = src.load(j, r, root);
                    active = true;
                    inv = mk3(__frcp_rn(r.d.x), __frcp_rn(r.d.y), __frcp_rn(r.d.z));
                    hit.inst = -1; hit.tri = -1;
                    hit.u = 0.0f; hit.v = 0.0f;
                    best_t = r.tmax;
                    found = false;
                    hit_any = false;
                    exhausted = root < 0;
                    sp = 0;
                    node = exhausted ? PYRE_NODE_NONE : (root | PYRE_TAG_TOP);
                    inst = -1;
                    o = r.o;
                    parked = 0;
#pragma unroll
                    for (int q = 0; q < PR; ++q) lc[q] = 0;
                }
            }
        }
        if (!__any_sync(FULL, active)) {
            if (drained) break;
            continue;
        }
        // ---- inner phase: step nodes until at most LEAF_WAIT lanes still
        // look for a leaf. Those lanes sit out the leaf phase and resume after
        // it; the others do not idle until the slowest lane reaches its first
        // leaf. The phase also runs while no lane holds a leaf to test, so each
        // round makes progress.
        while (true) {
            const int seeking = __popc(__ballot_sync(FULL, active && !exhausted && !hit_any && parked == 0));
            if (seeking == 0) break;
            if (seeking <= LEAF_WAIT && __any_sync(FULL, active && !hit_any && parked > 0)) break;
            // each lane takes up to PYRE_STEPS_PER_VOTE_WIDE node steps between the warp's votes
#pragma unroll 1
            for (int step = 0; step < PYRE_STEPS_PER_VOTE_WIDE; ++step) {
                if (!active || exhausted || hit_any || parked >= STOP) break;
                if (node == PYRE_NODE_NONE) {
                    if (sp == 0) { exhausted = true; continue; }
                    node = spop();
                }
                // a top-level entry reached inside an instance: the instance's
                // BVH is done, so the lane leaves it (once its parked leaves,
                // which belong to the instance, are tested)
                if (node & (PYRE_TAG_TOP | PYRE_TAG_INST)) {  // a top-level node or an instance entry
                    if (inst >= 0) {
                        if (ANY && parked) { spush(node); node = PYRE_NODE_NONE; parked = STOP; continue; }
                        inst = -1;
                        o = r.o;
                    }
                    if ((node & (PYRE_TAG_INST | PYRE_TAG_TOP)) == (PYRE_TAG_INST | PYRE_TAG_TOP)) {
                        // a static instance whose root box the top-level step
                        // tested: enter it and step its root node in this step
                        // (the lane is at the top level, so o is the world origin)
                        const int k = node & ~(PYRE_TAG_INST | PYRE_TAG_TOP);
                        node = __ldg(S.wroot + k);
                        if (node < 0) { node = PYRE_NODE_NONE; continue; }
                        inst = k;
                    } else if (node & PYRE_TAG_INST) {
                        if (ANY && parked) { spush(node); node = PYRE_NODE_NONE; parked = STOP; continue; }
                        const int k = node & ~PYRE_TAG_INST;
                        node = PYRE_NODE_NONE;
                        const DevInstance& I = S.inst[k];
                        const int root = S.wroot[k];
                        if (root < 0) continue;
                        f3 lo = r.o;
                        if (I.has_motion) {
                            f3 off = motion_offset(I, r.time);
                            if (!is_zero3(off)) lo = r.o - off;
                        }
                        float e;
                        if (!slab(I.lo[0], I.hi[0], I.lo[1], I.hi[1], I.lo[2], I.hi[2], lo, inv, r.tmin, best_t, &e))
                            continue;
                        inst = k;
                        o = lo;
                        node = root;
                        continue;
                    }
                }
                if (!(node & PYRE_TAG_TOP)) {
                    if (node & PYRE_TAG_LEAF) {  // park a leaf child of a wide node
                        const uint32_t ref = (uint32_t)(node & ~PYRE_TAG_LEAF);
                        const int32_t* NI = reinterpret_cast<const int32_t*>(S.wnodes) +
                                            (size_t)(ref / WIDTH) * (PYRE_WIDE_FIELDS * WIDTH) + ref % WIDTH;
                        ls[parked] = __ldg(NI + 6 * WIDTH);
                        lc[parked] = __ldg(NI + 7 * WIDTH);
                        ++parked;
                        node = PYRE_NODE_NONE;
                        continue;
                    }
                    constexpr int Q = WIDTH / 4;  // float4 rows per field
                    const float4* N = S.wnodes + (size_t)node * (2 * WIDTH);
                    float e[WIDTH];
                    int ent[WIDTH];
    #pragma unroll
                    for (int q = 0; q < Q; ++q) {
                        const float4 lx = __ldg(N + 0 * Q + q), hx = __ldg(N + 1 * Q + q), ly = __ldg(N + 2 * Q + q),
                                     hy = __ldg(N + 3 * Q + q), lz = __ldg(N + 4 * Q + q), hz = __ldg(N + 5 * Q + q);
                        const int4 ch = __ldg(reinterpret_cast<const int4*>(N + 6 * Q + q));
                        const int4 ct = __ldg(reinterpret_cast<const int4*>(N + 7 * Q + q));
                        const float LX[4] = {lx.x, lx.y, lx.z, lx.w}, HX[4] = {hx.x, hx.y, hx.z, hx.w};
                        const float LY[4] = {ly.x, ly.y, ly.z, ly.w}, HY[4] = {hy.x, hy.y, hy.z, hy.w};
                        const float LZ[4] = {lz.x, lz.y, lz.z, lz.w}, HZ[4] = {hz.x, hz.y, hz.z, hz.w};
                        const int CH[4] = {ch.x, ch.y, ch.z, ch.w}, CT[4] = {ct.x, ct.y, ct.z, ct.w};
    #pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            float ek;
                            const bool h = CH[k] >= 0 && slab(LX[k], HX[k], LY[k], HY[k], LZ[k], HZ[k], o, inv, r.tmin,
                                                              best_t, &ek);
                            e[4 * q + k] = h ? ek : __int_as_float(0x7f800000);
                            ent[4 * q + k] = !h ? PYRE_NODE_NONE
                                                : (CT[k] > 0 ? (PYRE_TAG_LEAF | (node * WIDTH + 4 * q + k)) : CH[k]);
                        }
                    }
                    sort_children<WIDTH>(e, ent);
                    int nh = 0;
    #pragma unroll
                    for (int k = 1; k < WIDTH; ++k) nh += ent[k] != PYRE_NODE_NONE ? 1 : 0;
                    if (sp + nh > STACK) { atomicExch(S.error_flag, -5); exhausted = true; sp = 0; continue; }
    #pragma unroll
                    for (int k = WIDTH - 1; k >= 1; --k)
                        if (ent[k] != PYRE_NODE_NONE) spush(ent[k]);
                    node = ent[0];
                    continue;
                }
                const float4* N = S.nodes + 4 * (size_t)(node & ~PYRE_TAG_TOP);
                float4 na, nb, nc, ndf;
                ldg_256(N, na, nb);
                ldg_256(N + 2, nc, ndf);
                const int4 nd = make_int4(__float_as_int(ndf.x), __float_as_int(ndf.y), __float_as_int(ndf.z),
                                          __float_as_int(ndf.w));
                float e0, e1;
                const bool h0 = nd.x >= 0 && slab(na.x, na.y, na.z, na.w, nc.x, nc.y, o, inv, r.tmin, best_t, &e0);
                const bool h1 = nd.y >= 0 && slab(nb.x, nb.y, nb.z, nb.w, nc.z, nc.w, o, inv, r.tmin, best_t, &e1);
                node = PYRE_NODE_NONE;
                const bool leaf0 = nd.z > 0, leaf1 = nd.w > 0;
                // a leaf queues its instances
                const int need = (h0 && leaf0 ? nd.z : 0) + (h1 && leaf1 ? nd.w : 0) + 1;
                if (sp + need > STACK) { atomicExch(S.error_flag, -5); exhausted = true; sp = 0; continue; }
                if (h1 && leaf1)
                    for (int k = nd.w - 1; k >= 0; --k) spush(PYRE_TAG_INST | (nd.y + k));
                if (h0 && leaf0)
                    for (int k = nd.z - 1; k >= 0; --k) spush(PYRE_TAG_INST | (nd.x + k));
                const int tag = PYRE_TAG_TOP;
                const bool g0 = h0 && !leaf0, g1 = h1 && !leaf1;
                if (g0 && g1) {
                    const bool first0 = e0 <= e1;
                    if (sp >= STACK) { atomicExch(S.error_flag, -5); exhausted = true; sp = 0; continue; }
                    spush((first0 ? nd.y : nd.x) | tag);
                    node = (first0 ? nd.x : nd.y) | tag;
                } else if (g0) {
                    node = nd.x | tag;
                } else if (g1) {
                    node = nd.y | tag;
                }
            }
        }
        // ---- leaf phase: all lanes test their parked triangles together
        const bool testing = active && !hit_any;
        const int c0 = testing ? lc[0] : 0, c1 = testing ? lc[1] : 0, c2 = (PR > 2 && testing) ? lc[PR - 1] : 0;
        const int total = parked == 0 ? 0 : c0 + (parked > 1 ? c1 : 0) + (PR > 2 && parked > 2 ? c2 : 0);
        const int kmax = __reduce_max_sync(FULL, total);
        for (int k = 0; k < kmax; ++k) {
            if (k >= total || hit_any) continue;
            const int slot = k < c0 ? ls[0] + k : (k < c0 + c1 ? ls[1] + (k - c0) : ls[PR - 1] + (k - c0 - c1));
            const float4 A = __ldg(S.tris + 3 * (size_t)slot), B = __ldg(S.tris + 3 * (size_t)slot + 1),
                         C = __ldg(S.tris + 3 * (size_t)slot + 2);
            float t, u, v;
            if (!mt_test(o, r.d, A, B, C, &t, &u, &v)) continue;
            if (!(t > r.tmin && t < r.tmax)) continue;
            if (ANY) { found = true; hit_any = true; continue; }
            bool better = t < best_t;
            if (!better && t == best_t && found) {
                // a tie (rare): the lower Scene::primitives index, then the lower
                // triangle id, wins; both are read back from the records
                const int32_t cur = S.inst[inst].orig_id, best = S.inst[hit.inst].orig_id;
                const uint32_t key = __float_as_uint(A.w);
                const uint32_t best_key = __float_as_uint(__ldg(S.tris + 3 * (size_t)hit.tri).w);
                better = cur < best || (cur == best && key < best_key);
            }
            if (better) {
                best_t = t;
                found = true;
                hit.u = u; hit.v = v;
                hit.inst = inst; hit.tri = slot;
            }
        }
        parked = 0;
#pragma unroll
        for (int q = 0; q < PR; ++q) lc[q] = 0;
        // ---- finished rays hand over their result; the lane becomes idle
        if (active && (exhausted || hit_any)) {
            hit.t = best_t;
            hit.light = -1;
            src.store(id, r, hit, found);
            active = false;
        }
    }
}

// DiffuseAreaQuadLight::intersect_plane (light.rs:86-107).
__device__ __forceinline__ bool quad_intersect(const DevQuadLight& L, const f3& o, const f3& d, float tmin, float tmax,
                                               float* t_out, f3* p_out) {
    float denom = dot3(d, L.normal);
    if (fabsf(denom) < 1e-9f) return false;
    float t = dot3(L.p0 - o, L.normal) / denom;
    if (t < tmin || t > tmax) return false;
    f3 p = o + t * d;
    f3 dd = p - L.p0;
    float alpha = dot3(cross3(dd, L.edge_v), L.crs) * L.inv_cross_len_sq;
    if (!(alpha >= 0.0f && alpha <= 1.0f)) return false;
    float beta = dot3(cross3(L.edge_u, dd), L.crs) * L.inv_cross_len_sq;
    if (!(beta >= 0.0f && beta <= 1.0f)) return false;
    *t_out = t;
    *p_out = p;
    return true;
}

// The traversal of one width (trace_binary for 2, trace_wide for 4 and 8).
template <bool ANY, int WIDTH, class Src>
__device__ __forceinline__ void trace_stream(const DevScene& S, const Src& src, uint32_t n, uint32_t* counter,
                                             int refill) {
    if constexpr (WIDTH == 2) {
        __shared__ TraceShared<ANY> sh;
        trace_binary<ANY>(S, src, n, counter, refill, whole_grid(n), sh.stack, sh.ray, sh.hit);
    } else trace_wide<ANY, WIDTH>(S, src, n, counter, refill);
}

// Quad lights after primitives with strict `<` (scene.rs:78-94): lights
// [light_first, light_first + light_count) can replace the closest hit.
__device__ __forceinline__ void hit_quad_lights(const DevScene& S, const TraceRay& r, uint32_t light_first,
                                                uint32_t light_count, TraceHit* hit) {
    float best = hit->inst >= 0 ? hit->t : r.tmax;
    for (uint32_t l = light_first; l < light_first + light_count; ++l) {
        float t; f3 p;
        if (quad_intersect(S.lights[l], r.o, r.d, r.tmin, best, &t, &p) && t < best) {
            best = t;
            hit->t = t; hit->light = (int32_t)l;
        }
    }
}

}  // namespace pyre
