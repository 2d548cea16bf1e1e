// bvh_device.cu — the reference's SAH-binned BVH build on the GPU.
//
// Produces, for each mesh, the same node array and primitive order as
// Bvh::build (crates/pyre/src/geometry/bvh.rs:45-64,180-409; restated on the
// host in bvh_host.cpp): 12 bins on the longest centroid axis, cost
// 1 + 2 (nL AL + nR AR) / A, leaves of at most 8 primitives, the midpoint and
// equal-count fallbacks, depth-first pre-order with the left child next.
//
// The recursion becomes a breadth-first loop over levels; every level
// processes all open nodes of more than 32 primitives, of all meshes, at once:
//   box      each position's node of this level, and the nodes' primitive and
//            centroid bounds (warp-segmented reductions, then order-preserving
//            integer atomics: min and max are exact, so the result does not
//            depend on the order)
//   bin      12-bin counts and boxes per node
//   decide   the prefix/suffix sweeps and SAH costs in the reference's order,
//            leaf or partition position
//   scan / sums / tables / scatter
//            the reference's in-place partition (two pointers, swap from the
//            end) computed in parallel from its closed form: with mid the
//            number of primitives left of the split, the k-th right-side
//            primitive of [start, mid) moves to l(k-1) - 1 and the k-th
//            left-side primitive of [mid, end) counted from the end (at l(k))
//            takes its place (l(0) = end); a right-side primitive at mid moves
//            to l(K) - 1 (K such pairs); any other right-side primitive at
//            q >= mid moves to q - 1
//   finish   node records, the equal-count fallback, the next level's nodes
// Ranges of at most 32 primitives are finished by one warp each (small).
// Depth-first indices follow from one scan of the leaf starts (BNode), and the
// emit kernels write the reference layout or the 64-byte device nodes.
//
// The host launches several levels before it asks how many nodes are open, and
// all arrays share one allocation (BuildWorkspace). Bound by launches: a
// level is 8 kernels of 3 to 20 us. From and to host arrays, 300,007 triangles
// take 1.82 ms and 1.3 M 5.2 ms; 13 kernels and a synchronisation per level down
// to single primitives, with some 35 allocations per build, took 7.6 and 17.4.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "bvh_host.h"
#include "internal.h"

// ------------------------------------------------------------------ types --
namespace pyre {
namespace {

constexpr int kBins = 12;
constexpr uint32_t kMaxLeaf = 8;
constexpr uint32_t kSmall = 32;   // ranges of at most this many primitives are finished by one warp (k_small)
constexpr int kScanBlock = 1024;  // threads of the scan kernels, 4 elements each
constexpr int kScanLog2 = 12;     // 4 * kScanBlock elements per block
constexpr int kCounters = 64;     // task counts of consecutive levels, a ring
enum : int { MODE_LEAF = 0, MODE_BIN = 1, MODE_PART = 2, MODE_SPLIT = 3 };

// float <-> unsigned with the same order (for atomicMin / atomicMax)
__device__ __forceinline__ uint32_t ord(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float unord(uint32_t o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
constexpr uint32_t kOrdInf = 0xFF800000u, kOrdNegInf = 0x007FFFFFu;
__device__ __forceinline__ float comp4(float4 v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }
__device__ __forceinline__ int32_t to_i32(float f) {  // Rust `as i32`
    if (f != f) return 0;
    if (f >= 2147483647.0f) return 2147483647;
    if (f <= -2147483648.0f) return (int32_t)0x80000000;
    return (int32_t)f;
}

// An open node: the primitives at positions [start, end) of the order.
struct Task {
    uint32_t start, end;
    uint32_t node;   // node id
    uint32_t mesh;
    uint32_t lefts;  // left steps on the path from the mesh's root (see BNode)
};

struct TaskAcc {
    uint32_t lo[3], hi[3], clo[3], chi[3];
    uint32_t bins[kBins][7];  // count, lo, hi
};
constexpr uint32_t kAccWords = sizeof(TaskAcc) / 4;
__device__ __forceinline__ uint32_t acc_init_word(uint32_t k) {  // word k of an empty TaskAcc
    if (k < 12) return (k / 3) & 1 ? kOrdNegInf : kOrdInf;
    const uint32_t q = (k - 12) % 7;
    return q == 0 ? 0u : (q <= 3 ? kOrdInf : kOrdNegInf);
}

struct TaskState {
    int mode, axis;
    float cmin, scale, extent, split;
    uint32_t mid;                    // first position of the right child
    int32_t left_task, right_task;   // of the next level; -1 for a range that k_small finishes
    uint32_t leaf_count;
};

// A node, ids in no order. A binary tree over n leaves has n - 1 interior
// nodes, so with L(v) the leaves of the mesh that start before v's first
// position, the depth-first index of v is 2 L(v) + lefts(v), and its index
// among the interior nodes L(v) + lefts(v): a left step adds one (the parent),
// a right step the left subtree, 2 n - 1 nodes and the parent. One scan of the
// leaf starts replaces passes over the tree.
struct BNode {
    float lo[3], hi[3];
    uint32_t start, count;   // leaf: positions [start, start + count)
    int32_t left, right;     // interior: node ids; -1 for a leaf
    uint32_t axis, mesh;     // mesh: kNoMesh marks an unused id
    uint32_t mid, lefts;     // interior: first position of the right child
};
constexpr uint32_t kNoMesh = 0xffffffffu;

__device__ __forceinline__ float area(float lx, float ly, float lz, float hx, float hy, float hz) {
    const float dx = hx - lx, dy = hy - ly, dz = hz - lz;
    return 2.0f * (dx * dy + dx * dz + dy * dz);
}

// bvh.rs:189-211: leaves of one primitive or of coincident centroids; the
// binning axis and scale otherwise.
__device__ __forceinline__ TaskState prepare(uint32_t n, float clx, float cly, float clz, float chx, float chy,
                                             float chz) {
    TaskState s{};
    const float dx = chx - clx, dy = chy - cly, dz = chz - clz;
    const int axis = (dx >= dy && dx >= dz) ? 0 : (dy >= dz ? 1 : 2);
    const float extent = axis == 0 ? dx : (axis == 1 ? dy : dz);
    if (n == 1) {
        s.mode = MODE_LEAF; s.leaf_count = 1;
    } else if (extent < 1e-9f) {
        s.mode = MODE_LEAF; s.leaf_count = min(n, 65535u);
    } else {
        s.mode = MODE_BIN;
        s.axis = axis;
        s.extent = extent;
        s.cmin = axis == 0 ? clx : (axis == 1 ? cly : clz);
        s.scale = (float)kBins / extent;
    }
    return s;
}
__device__ __forceinline__ TaskState prepare(const Task& T, const TaskAcc& a) {
    return prepare(T.end - T.start, unord(a.clo[0]), unord(a.clo[1]), unord(a.clo[2]), unord(a.chi[0]),
                   unord(a.chi[1]), unord(a.chi[2]));
}
__device__ __forceinline__ int bin_of(float c, const TaskState& s) {
    return min(max(to_i32((c - s.cmin) * s.scale), 0), kBins - 1);
}
__device__ __forceinline__ float split_cost(uint32_t ln, float la, uint32_t rn, float ra, float parent_area) {
    return 1.0f + 2.0f * ((float)ln * la + (float)rn * ra) / parent_area;
}
// bvh.rs:306-321: leaf test and partition position, from the cheapest boundary.
__device__ __forceinline__ void decide(TaskState& s, uint32_t n, float best, int best_i) {
    if (!isfinite(best)) {
        s.mode = MODE_PART;
        s.split = s.cmin + 0.5f * s.extent;
    } else if (n <= kMaxLeaf && best >= 2.0f * (float)n) {
        s.mode = MODE_LEAF;
        s.leaf_count = n;
    } else {
        s.mode = MODE_PART;
        s.split = s.cmin + (float)(best_i + 1) * s.extent / (float)kBins;
    }
}

// Per-triangle bounds and centroid (mesh.rs:32-40, as triangle_bounds).
__global__ void k_tri_bounds(const float* __restrict__ pos, const uint32_t* __restrict__ idx, uint32_t n,
                             float4* blo, float4* bhi, float4* cen) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const uint32_t i0 = idx[3 * (size_t)t], i1 = idx[3 * (size_t)t + 1], i2 = idx[3 * (size_t)t + 2];
        const f3 a = mk3(pos[3 * (size_t)i0], pos[3 * (size_t)i0 + 1], pos[3 * (size_t)i0 + 2]);
        const f3 b = mk3(pos[3 * (size_t)i1], pos[3 * (size_t)i1 + 1], pos[3 * (size_t)i1 + 2]);
        const f3 c = mk3(pos[3 * (size_t)i2], pos[3 * (size_t)i2 + 1], pos[3 * (size_t)i2 + 2]);
        const f3 lo = vmin3(vmin3(a, b), c), hi = vmax3(vmax3(a, b), c);
        const f3 m = (a + b + c) / 3.0f;
        blo[t] = make_float4(lo.x, lo.y, lo.z, 0.0f);
        bhi[t] = make_float4(hi.x, hi.y, hi.z, 0.0f);
        cen[t] = make_float4(m.x, m.y, m.z, 0.0f);
    }
}

__device__ __forceinline__ void init_acc(TaskAcc& a) {
    for (uint32_t k = 0; k < kAccWords; ++k) reinterpret_cast<uint32_t*>(&a)[k] = acc_init_word(k);
}

// Level 0: the order, each position's mesh and task, and the root tasks: root
// m is node m; meshes of at most kSmall primitives go to the small list.
__global__ void k_init(const uint32_t* __restrict__ mesh_prim_base, uint32_t n_meshes, uint32_t n, uint32_t* prim_mesh,
                       int32_t* pos_task, uint32_t* idx, Task* tasks, TaskAcc* acc, Task* small, uint32_t* counters) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = n_meshes - 1;  // last mesh whose base is <= p
        while (lo < hi) {
            const uint32_t mid = (lo + hi + 1) / 2;
            if (mesh_prim_base[mid] <= p) lo = mid; else hi = mid - 1;
        }
        prim_mesh[p] = lo;
        idx[p] = p;
        const uint32_t base = mesh_prim_base[lo], end = lo + 1 < n_meshes ? mesh_prim_base[lo + 1] : n;
        const bool is_small = end - base <= kSmall;
        pos_task[p] = is_small ? -1 : (int32_t)lo;
        if (p == base) {
            const Task T{base, end, lo, lo, 0u};
            tasks[lo] = T;  // a task per mesh at level 0; those in the small list are holes there
            if (is_small) small[atomicAdd(&counters[kCounters], 1u)] = T;
            else init_acc(acc[lo]);
        }
    }
}

// Reduces v over the lanes of `peers` and lets its first lane apply the atomic.
__device__ __forceinline__ void seg_min(unsigned peers, bool leader, uint32_t* dst, uint32_t v) {
    v = __reduce_min_sync(peers, v);
    if (leader) atomicMin(dst, v);
}
__device__ __forceinline__ void seg_max(unsigned peers, bool leader, uint32_t* dst, uint32_t v) {
    v = __reduce_max_sync(peers, v);
    if (leader) atomicMax(dst, v);
}

// k_box and k_bin: a block takes kChunk consecutive positions, whole warps per
// round (every lane takes part in the warp-collective operations). The task of
// the block's first position is summed in shared memory and added once per
// block, other tasks directly: at the top levels all positions belong to a few
// tasks, and one atomic per warp and value queued on those addresses (k_bin
// 0.14 against 0.02 ms at the root of 300,007 triangles).
constexpr uint32_t kChunk = 512;
#define WARP_ROUNDS(wb, n)                                                                                     \
    for (uint32_t wb = blockIdx.x * kChunk + (threadIdx.x & ~31u), wb##_end = min((n), (blockIdx.x + 1) * kChunk); \
         wb < wb##_end; wb += blockDim.x)

// Moves each position to its task of this level (prev: the states of the
// level above, null at level 0) and gathers the tasks' bounds.
__global__ void k_box(int32_t* __restrict__ pos_task, const TaskState* __restrict__ prev,
                      const uint32_t* __restrict__ idx, const float4* __restrict__ blo, const float4* __restrict__ bhi,
                      const float4* __restrict__ cen, uint32_t n, TaskAcc* acc) {
    __shared__ uint32_t sum[12];
    __shared__ int32_t first;
    const int lane = threadIdx.x & 31;
    auto moved = [&](uint32_t p) -> int32_t {
        int32_t t = pos_task[p];
        if (prev && t >= 0) {
            const TaskState& s = prev[t];
            t = s.mode != MODE_SPLIT ? -1 : (p < s.mid ? s.left_task : s.right_task);
        }
        return t;
    };
    if (threadIdx.x < 12) sum[threadIdx.x] = (threadIdx.x / 3) & 1 ? kOrdNegInf : kOrdInf;  // lo, hi, clo, chi
    if (threadIdx.x == 0) first = moved(blockIdx.x * kChunk);
    __syncthreads();
    const int32_t t0 = first;
    WARP_ROUNDS(wb, n) {
        const uint32_t p = wb + lane;
        int32_t t = -1;
        if (p < n) {
            t = moved(p);
            if (prev) pos_task[p] = t;
        }
        const unsigned peers = __match_any_sync(0xffffffffu, t);
        if (t < 0) continue;
        const bool leader = lane == __ffs(peers) - 1;
        const uint32_t prim = idx[p];
        const float4 lo = blo[prim], hi = bhi[prim], c = cen[prim];
        uint32_t* a = t == t0 ? sum : reinterpret_cast<uint32_t*>(acc + t);  // lo, hi, clo, chi: 12 consecutive words
        seg_min(peers, leader, a + 0, ord(lo.x)); seg_min(peers, leader, a + 1, ord(lo.y));
        seg_min(peers, leader, a + 2, ord(lo.z));
        seg_max(peers, leader, a + 3, ord(hi.x)); seg_max(peers, leader, a + 4, ord(hi.y));
        seg_max(peers, leader, a + 5, ord(hi.z));
        seg_min(peers, leader, a + 6, ord(c.x)); seg_min(peers, leader, a + 7, ord(c.y));
        seg_min(peers, leader, a + 8, ord(c.z));
        seg_max(peers, leader, a + 9, ord(c.x)); seg_max(peers, leader, a + 10, ord(c.y));
        seg_max(peers, leader, a + 11, ord(c.z));
    }
    __syncthreads();
    if (t0 >= 0 && threadIdx.x < 12) {
        uint32_t* a = reinterpret_cast<uint32_t*>(acc + t0) + threadIdx.x;
        if ((threadIdx.x / 3) & 1) atomicMax(a, sum[threadIdx.x]);
        else atomicMin(a, sum[threadIdx.x]);
    }
}

__global__ void k_bin(const int32_t* __restrict__ pos_task, const Task* __restrict__ tasks,
                      const uint32_t* __restrict__ idx, const float4* __restrict__ blo, const float4* __restrict__ bhi,
                      const float4* __restrict__ cen, uint32_t n, TaskAcc* acc) {
    __shared__ uint32_t sum[kBins * 7];  // per bin: count, lo, hi
    const int lane = threadIdx.x & 31;
    for (uint32_t k = threadIdx.x; k < kBins * 7; k += blockDim.x)
        sum[k] = k % 7 == 0 ? 0u : (k % 7 <= 3 ? kOrdInf : kOrdNegInf);
    __syncthreads();
    const int32_t t0 = pos_task[blockIdx.x * kChunk];
    WARP_ROUNDS(wb, n) {
        const uint32_t p = wb + lane;
        int32_t t = p < n ? pos_task[p] : -1;
        int b = 0;
        uint32_t prim = 0;
        if (t >= 0) {
            const TaskState s = prepare(tasks[t], acc[t]);
            if (s.mode != MODE_BIN) t = -1;
            else {
                prim = idx[p];
                b = bin_of(comp4(cen[prim], s.axis), s);
            }
        }
        const long long key = t < 0 ? -1ll : (long long)t * kBins + b;
        const unsigned peers = __match_any_sync(0xffffffffu, key);
        if (t < 0) continue;
        const bool leader = lane == __ffs(peers) - 1;
        uint32_t* a = t == t0 ? sum + 7 * b : acc[t].bins[b];
        if (leader) atomicAdd(a, (uint32_t)__popc(peers));
        const float4 lo = blo[prim], hi = bhi[prim];
        seg_min(peers, leader, a + 1, ord(lo.x)); seg_min(peers, leader, a + 2, ord(lo.y));
        seg_min(peers, leader, a + 3, ord(lo.z));
        seg_max(peers, leader, a + 4, ord(hi.x)); seg_max(peers, leader, a + 5, ord(hi.y));
        seg_max(peers, leader, a + 6, ord(hi.z));
    }
    __syncthreads();
    if (t0 >= 0 && threadIdx.x < kBins * 7 && sum[threadIdx.x / 7 * 7]) {
        uint32_t* a = &acc[t0].bins[0][0] + threadIdx.x;
        const uint32_t v = sum[threadIdx.x], k = threadIdx.x % 7;
        if (k == 0) atomicAdd(a, v);
        else if (k <= 3) atomicMin(a, v);
        else atomicMax(a, v);
    }
}

// bvh.rs:236-321: sweeps, costs, leaf test, partition position.
__global__ void k_decide(const Task* __restrict__ tasks, const TaskAcc* __restrict__ acc,
                         const uint32_t* __restrict__ n_tasks, TaskState* st) {
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < *n_tasks; t += gridDim.x * blockDim.x) {
        const Task T = tasks[t];
        const TaskAcc& a = acc[t];
        const uint32_t n = T.end - T.start;
        if (n <= kSmall) { st[t].mode = MODE_LEAF; st[t].leaf_count = 0; continue; }  // a hole of level 0
        TaskState s = prepare(T, a);
        if (s.mode == MODE_BIN) {
            uint32_t ln[kBins - 1], rn[kBins - 1];
            float la[kBins - 1], ra[kBins - 1];
            uint32_t c = 0;
            float lx = INFINITY, ly = INFINITY, lz = INFINITY, hx = -INFINITY, hy = -INFINITY, hz = -INFINITY;
            for (int i = 0; i < kBins - 1; ++i) {
                c += a.bins[i][0];
                lx = fminf(lx, unord(a.bins[i][1])); ly = fminf(ly, unord(a.bins[i][2]));
                lz = fminf(lz, unord(a.bins[i][3]));
                hx = fmaxf(hx, unord(a.bins[i][4])); hy = fmaxf(hy, unord(a.bins[i][5]));
                hz = fmaxf(hz, unord(a.bins[i][6]));
                ln[i] = c;
                la[i] = area(lx, ly, lz, hx, hy, hz);
            }
            c = 0;
            lx = ly = lz = INFINITY; hx = hy = hz = -INFINITY;
            for (int i = kBins - 2; i >= 0; --i) {
                c += a.bins[i + 1][0];
                lx = fminf(lx, unord(a.bins[i + 1][1])); ly = fminf(ly, unord(a.bins[i + 1][2]));
                lz = fminf(lz, unord(a.bins[i + 1][3]));
                hx = fmaxf(hx, unord(a.bins[i + 1][4])); hy = fmaxf(hy, unord(a.bins[i + 1][5]));
                hz = fmaxf(hz, unord(a.bins[i + 1][6]));
                rn[i] = c;
                ra[i] = area(lx, ly, lz, hx, hy, hz);
            }
            const float parent_area = fmaxf(area(unord(a.lo[0]), unord(a.lo[1]), unord(a.lo[2]), unord(a.hi[0]),
                                                 unord(a.hi[1]), unord(a.hi[2])),
                                            1e-9f);
            float best = INFINITY;
            int best_i = 0;
            for (int i = 0; i < kBins - 1; ++i) {
                if (ln[i] == 0 || rn[i] == 0) continue;
                const float cost = split_cost(ln[i], la[i], rn[i], ra[i], parent_area);
                if (cost < best) { best = cost; best_i = i; }
            }
            decide(s, n, best, best_i);
        }
        st[t] = s;
    }
}

// Exclusive scan within a block of kScanBlock threads.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* warp_tot, uint32_t* total) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) warp_tot[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < (blockDim.x >> 5) ? warp_tot[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= (uint32_t)o) w += y;
        }
        warp_tot[lane] = w;
    }
    __syncthreads();
    const uint32_t r = (warp ? warp_tot[warp - 1] : 0u) + x - v;
    if (total) *total = warp_tot[(blockDim.x >> 5) - 1];
    __syncthreads();
    return r;
}

// The partition flags (1: left of the split) and their exclusive scan within
// blocks of 4 * kScanBlock positions; k_scan_sums scans the block sums.
// With `st` null the flags are given (the leaf starts).
__global__ void __launch_bounds__(kScanBlock) k_scan_local(const int32_t* __restrict__ pos_task,
                                                           const uint32_t* __restrict__ idx,
                                                           const float4* __restrict__ cen,
                                                           const TaskState* __restrict__ st, uint32_t n, uint32_t* flag,
                                                           uint32_t* out, uint32_t* block_sum) {
    __shared__ uint32_t warp_tot[32];
    __shared__ uint32_t tot;
    const uint64_t base = (uint64_t)blockIdx.x * 4 * kScanBlock + 4 * (uint64_t)threadIdx.x;
    uint32_t v[4], s = 0;
    for (int k = 0; k < 4; ++k) {
        uint32_t f = 0;
        if (base + k < n) {
            const uint32_t p = (uint32_t)(base + k);
            if (!st) f = flag[p];
            else {
                const int32_t t = pos_task[p];
                if (t >= 0 && st[t].mode == MODE_PART) f = comp4(cen[idx[p]], st[t].axis) < st[t].split ? 1u : 0u;
                flag[p] = f;
            }
        }
        v[k] = f;
        s += f;
    }
    uint32_t off = block_excl_scan(s, warp_tot, threadIdx.x == 0 ? &tot : nullptr);
    __syncthreads();
    for (int k = 0; k < 4; ++k) {
        if (base + k < n) out[base + k] = off;
        off += v[k];
    }
    if (threadIdx.x == 0) block_sum[blockIdx.x] = tot;
}

// Block sums to block offsets, and one more entry: the total.
__global__ void __launch_bounds__(kScanBlock) k_scan_sums(uint32_t* block_sum, uint32_t n_blocks) {
    __shared__ uint32_t warp_tot[32];
    __shared__ uint32_t tot;
    uint32_t carry = 0;
    for (uint32_t b0 = 0; b0 < n_blocks; b0 += kScanBlock) {
        const uint32_t i = b0 + threadIdx.x;
        const uint32_t v = i < n_blocks ? block_sum[i] : 0u;
        const uint32_t e = block_excl_scan(v, warp_tot, threadIdx.x == 0 ? &tot : nullptr);
        __syncthreads();
        if (i < n_blocks) block_sum[i] = carry + e;
        carry += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) block_sum[n_blocks] = carry;
}

// The scan of k_scan_local and k_scan_sums at position p of [0, n].
struct Scan {
    const uint32_t* local;
    const uint32_t* block;
    uint32_t n, n_blocks;
    __device__ __forceinline__ uint32_t operator()(uint32_t p) const {
        return p < n ? local[p] + block[p >> kScanLog2] : block[n_blocks];
    }
};

// Rank tables of the partition: front[start + k - 1] = position of the k-th
// right-side primitive of [start, mid); back[start + r - 1] = position of the
// r-th left-side primitive of [mid, end) counted from the end.
__global__ void k_tables(const int32_t* __restrict__ pos_task, const Task* __restrict__ tasks,
                         const TaskState* __restrict__ st, const uint32_t* __restrict__ flag, Scan pre, uint32_t n,
                         uint32_t* front, uint32_t* back) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const int32_t t = pos_task[p];
        if (t < 0 || st[t].mode != MODE_PART) continue;
        const Task T = tasks[t];
        const uint32_t p0 = pre(T.start), Lb = pre(p) - p0, Lt = pre(T.end) - p0;
        const uint32_t mid = T.start + Lt;
        if (p < mid) {
            if (!flag[p]) front[T.start + (p - T.start - Lb)] = p;
        } else if (flag[p]) {
            back[T.start + (Lt - Lb) - 1] = p;
        }
    }
}

__global__ void k_scatter(const int32_t* __restrict__ pos_task, const Task* __restrict__ tasks,
                          const TaskState* __restrict__ st, const uint32_t* __restrict__ flag, Scan pre,
                          const uint32_t* __restrict__ front, const uint32_t* __restrict__ back,
                          const uint32_t* __restrict__ idx, uint32_t n, uint32_t* idx_next) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const int32_t t = pos_task[p];
        uint32_t dst = p;
        if (t >= 0 && st[t].mode == MODE_PART) {
            const Task T = tasks[t];
            const uint32_t p0 = pre(T.start), Lb = pre(p) - p0, Lt = pre(T.end) - p0;
            const uint32_t mid = T.start + Lt;
            const uint32_t K = (mid - T.start) - (pre(mid) - p0);  // right-side primitives left of mid
            auto l_of = [&](uint32_t k) { return k == 0 ? T.end : back[T.start + k - 1]; };
            if (p < mid) {
                if (!flag[p]) dst = l_of(p - T.start - Lb) - 1;  // k-th: l(k - 1) - 1
            } else if (flag[p]) {
                dst = front[T.start + (Lt - Lb) - 1];
            } else {
                dst = p == mid ? l_of(K) - 1 : p - 1;
            }
        }
        idx_next[dst] = idx[p];
    }
}

// Node records and the open ranges below them: tasks of the next level, or
// entries of the small list. counters: task counts by level (a ring), then the
// length of the small list and the number of node ids.
__global__ void k_finish(const Task* __restrict__ tasks, const TaskAcc* __restrict__ acc, uint32_t level, Scan pre,
                         TaskState* st, BNode* nodes, Task* next, TaskAcc* next_acc, Task* small, uint32_t* leaf_start,
                         uint32_t* counters) {
    const uint32_t n_tasks = counters[level % kCounters];
    if (blockIdx.x == 0 && threadIdx.x == 0) counters[(level + 2) % kCounters] = 0;
    const unsigned FULL = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    uint32_t empty[kAccWords / 32];  // the lane's words of an empty TaskAcc
    static_assert(kAccWords % 32 == 0, "a warp writes whole rows of a TaskAcc");
#pragma unroll
    for (uint32_t k = 0; k < kAccWords / 32; ++k) empty[k] = acc_init_word(lane + 32 * k);
    // one atomic per warp: `*counter += step` for each lane of `take`, the lane's first number returned
    auto draw = [&](uint32_t* counter, bool take, uint32_t step) -> uint32_t {
        const unsigned m = __ballot_sync(FULL, take);
        uint32_t base = 0;
        if (m && lane == 0) base = atomicAdd(counter, step * (uint32_t)__popc(m));
        return __shfl_sync(FULL, base, 0) + step * (uint32_t)__popc(m & below);
    };
    for (uint32_t t0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); t0 < n_tasks; t0 += gridDim.x * blockDim.x) {
        const uint32_t t = t0 + lane;
        Task T{};
        if (t < n_tasks) T = tasks[t];
        const uint32_t n = T.end - T.start;
        const bool live = n > kSmall;  // not a hole of level 0
        TaskState s{};
        BNode nd{};
        uint32_t mid = 0;
        if (live) {
            s = st[t];
            const TaskAcc& a = acc[t];
            for (int k = 0; k < 3; ++k) { nd.lo[k] = unord(a.lo[k]); nd.hi[k] = unord(a.hi[k]); }
            nd.mesh = T.mesh;
            nd.lefts = T.lefts;
            nd.start = T.start;
            if (s.mode == MODE_PART) {
                mid = T.start + (pre(T.end) - pre(T.start));
                if (mid == T.start || mid == T.end) mid = T.start + n / 2;  // n > kMaxLeaf here
                s.mode = MODE_SPLIT;
                s.mid = mid;
            }
        }
        const bool split = s.mode == MODE_SPLIT;
        const uint32_t nn = draw(&counters[kCounters + 1], split, 2u);
        const Task kid[2] = {{T.start, mid, nn, T.mesh, T.lefts + 1}, {mid, T.end, nn + 1, T.mesh, T.lefts}};
        int32_t id[2] = {-1, -1};
        for (int c = 0; c < 2; ++c) {
            const bool big = split && kid[c].end - kid[c].start > kSmall;
            const uint32_t at_next = draw(&counters[(level + 1) % kCounters], big, 1u);
            const uint32_t at_small = draw(&counters[kCounters], split && !big, 1u);
            if (big) {
                id[c] = (int32_t)at_next;
                next[at_next] = kid[c];
            } else if (split) {
                small[at_small] = kid[c];
            }
        }
        if (live) {
            if (split) {
                s.left_task = id[0]; s.right_task = id[1];
                nd.left = (int32_t)nn; nd.right = (int32_t)nn + 1; nd.axis = (uint32_t)s.axis; nd.mid = mid;
            } else {
                nd.count = s.leaf_count; nd.left = nd.right = -1;
                leaf_start[T.start] = 1;
            }
            nodes[T.node] = nd;
            st[t] = s;
        }
        // the children's accumulators, a warp per record
        for (int c = 0; c < 2; ++c)
            for (unsigned todo = __ballot_sync(FULL, id[c] >= 0); todo; todo &= todo - 1) {
                uint32_t* w = reinterpret_cast<uint32_t*>(next_acc + __shfl_sync(FULL, id[c], __ffs(todo) - 1));
#pragma unroll
                for (uint32_t k = 0; k < kAccWords / 32; ++k) w[lane + 32 * k] = empty[k];
            }
    }
}

// One warp finishes a range of at most 32 primitives, a lane per primitive:
// the same decisions as the level kernels, with the bounds by warp reductions,
// the eleven candidate boundaries one per lane over the primitives in shared
// memory, and the partition's closed form on ballots. Below 32 primitives a
// level costs the device as much as one of the whole mesh, and there are eight
// or more of them.
__global__ void __launch_bounds__(128) k_small(const Task* __restrict__ small, const uint32_t* __restrict__ counters_in,
                                               const float4* __restrict__ blo, const float4* __restrict__ bhi,
                                               const float4* __restrict__ cen, uint32_t* idx, BNode* nodes,
                                               uint32_t* leaf_start, uint32_t* counters) {
    const unsigned FULL = 0xffffffffu;
    __shared__ float box[4][7][32];          // bounds and bin of the warp's primitives, in their order
    __shared__ uint32_t tab[4][2][32];       // front and back tables of a partition
    __shared__ uint32_t perm[4][32];
    __shared__ uint4 todo[4][32];            // (first, last, node, lefts) of the open ranges
    const uint32_t w = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t n_small = counters_in[kCounters];
    for (uint32_t task = blockIdx.x * 4 + w; task < n_small; task += gridDim.x * 4) {
        const Task T = small[task];
        const uint32_t n_all = T.end - T.start;
        uint32_t prim = 0;
        float4 lo = make_float4(0, 0, 0, 0), hi = lo, c = lo;
        if ((uint32_t)lane < n_all) {
            prim = idx[T.start + lane];
            lo = blo[prim]; hi = bhi[prim]; c = cen[prim];
        }
        uint32_t ids = 0;  // node ids of the subtree below its root
        if (lane == 0) ids = atomicAdd(&counters[kCounters + 1], 2u * n_all - 2u);
        ids = __shfl_sync(FULL, ids, 0);
        int n_open = 1;
        if (lane == 0) todo[w][0] = make_uint4(0, n_all, T.node, T.lefts);
        __syncwarp();
        while (n_open > 0) {
            const uint4 r = todo[w][--n_open];
            __syncwarp();
            const uint32_t a = r.x, b = r.y, n = b - a;
            const bool in = (uint32_t)lane >= a && (uint32_t)lane < b;
            auto rmin = [&](float v) { return unord(__reduce_min_sync(FULL, in ? ord(v) : kOrdInf)); };
            auto rmax = [&](float v) { return unord(__reduce_max_sync(FULL, in ? ord(v) : kOrdNegInf)); };
            BNode nd;
            nd.lo[0] = rmin(lo.x); nd.lo[1] = rmin(lo.y); nd.lo[2] = rmin(lo.z);
            nd.hi[0] = rmax(hi.x); nd.hi[1] = rmax(hi.y); nd.hi[2] = rmax(hi.z);
            const float clx = rmin(c.x), cly = rmin(c.y), clz = rmin(c.z), chx = rmax(c.x), chy = rmax(c.y), chz = rmax(c.z);
            TaskState s = prepare(n, clx, cly, clz, chx, chy, chz);
            uint32_t mid = 0;
            if (s.mode == MODE_BIN) {
                const int bin = in ? bin_of(comp4(c, s.axis), s) : 0;
                box[w][0][lane] = lo.x; box[w][1][lane] = lo.y; box[w][2][lane] = lo.z;
                box[w][3][lane] = hi.x; box[w][4][lane] = hi.y; box[w][5][lane] = hi.z;
                box[w][6][lane] = __int_as_float(bin);
                __syncwarp();
                // boundary `lane`: bins 0 .. lane on the left
                uint32_t ln = 0, rn = 0;
                float l[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
                float q[6] = {INFINITY, INFINITY, INFINITY, -INFINITY, -INFINITY, -INFINITY};
                for (uint32_t j = a; j < b; ++j) {
                    const bool left = __float_as_int(box[w][6][j]) <= lane;
                    ln += left ? 1u : 0u;
                    rn += left ? 0u : 1u;
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const float v = box[w][k][j], u = box[w][3 + k][j];
                        l[k] = fminf(l[k], left ? v : INFINITY); l[3 + k] = fmaxf(l[3 + k], left ? u : -INFINITY);
                        q[k] = fminf(q[k], left ? INFINITY : v); q[3 + k] = fmaxf(q[3 + k], left ? -INFINITY : u);
                    }
                }
                const float parent_area =
                    fmaxf(area(nd.lo[0], nd.lo[1], nd.lo[2], nd.hi[0], nd.hi[1], nd.hi[2]), 1e-9f);
                float cost = INFINITY;
                if (lane < kBins - 1 && ln && rn)
                    cost = split_cost(ln, area(l[0], l[1], l[2], l[3], l[4], l[5]), rn,
                                      area(q[0], q[1], q[2], q[3], q[4], q[5]), parent_area);
                if (!(cost < INFINITY)) cost = INFINITY;  // NaN is never chosen
                const float best = unord(__reduce_min_sync(FULL, ord(cost)));
                const int best_i = __ffs(__ballot_sync(FULL, cost == best)) - 1;  // the first of equals
                decide(s, n, best, best_i);
            }
            if (s.mode == MODE_PART) {
                // the partition (k_tables, k_scatter) on the warp's ballots
                const bool flag = in && comp4(c, s.axis) < s.split;
                const unsigned F = __ballot_sync(FULL, flag);
                const uint32_t p = (uint32_t)lane;
                const unsigned below = (1u << lane) - 1u;
                const uint32_t Lt = __popc(F), Lb = __popc(F & below);  // F holds lanes of [a, b) only
                mid = a + Lt;
                if (in && p < mid && !flag) tab[w][0][p - a - Lb] = p;
                if (in && p >= mid && flag) tab[w][1][Lt - Lb - 1] = p;
                __syncwarp();
                const uint32_t K = Lt - __popc(F & (mid < 32u ? (1u << mid) - 1u : FULL));
                auto l_of = [&](uint32_t k) { return k == 0 ? b : tab[w][1][k - 1]; };
                uint32_t dst = p;
                if (in) {
                    if (p < mid) {
                        if (!flag) dst = l_of(p - a - Lb) - 1;
                    } else if (flag) {
                        dst = tab[w][0][Lt - Lb - 1];
                    } else {
                        dst = p == mid ? l_of(K) - 1 : p - 1;
                    }
                }
                perm[w][dst] = p;
                __syncwarp();
                const int src = (int)perm[w][lane];
                prim = __shfl_sync(FULL, prim, src);
                lo.x = __shfl_sync(FULL, lo.x, src); lo.y = __shfl_sync(FULL, lo.y, src); lo.z = __shfl_sync(FULL, lo.z, src);
                hi.x = __shfl_sync(FULL, hi.x, src); hi.y = __shfl_sync(FULL, hi.y, src); hi.z = __shfl_sync(FULL, hi.z, src);
                c.x = __shfl_sync(FULL, c.x, src); c.y = __shfl_sync(FULL, c.y, src); c.z = __shfl_sync(FULL, c.z, src);
                __syncwarp();
                if (mid == a || mid == b) {
                    if (n <= kMaxLeaf) { s.mode = MODE_LEAF; s.leaf_count = n; }
                    else mid = a + n / 2;
                }
            }
            nd.mesh = T.mesh;
            nd.lefts = r.w;
            nd.start = T.start + a;
            if (s.mode == MODE_LEAF) {
                nd.count = s.leaf_count; nd.left = nd.right = -1; nd.axis = 0; nd.mid = 0;
                if (lane == 0) leaf_start[nd.start] = 1;
            } else {
                nd.count = 0; nd.left = (int32_t)ids; nd.right = (int32_t)ids + 1; nd.axis = (uint32_t)s.axis;
                nd.mid = T.start + mid;
                if (lane == 0) {
                    todo[w][n_open] = make_uint4(a, mid, ids, r.w + 1);
                    todo[w][n_open + 1] = make_uint4(mid, b, ids + 1, r.w);
                }
                n_open += 2;
                ids += 2;
            }
            if (lane == 0) nodes[r.z] = nd;
            __syncwarp();
        }
        if ((uint32_t)lane < n_all) idx[T.start + lane] = prim;
        __syncwarp();
    }
}

// The reference layout of every node (pyre_bvh2_node) into its mesh's range.
__global__ void k_emit_ref(const BNode* __restrict__ nodes, const uint32_t* __restrict__ counters, Scan leaves,
                           const uint32_t* __restrict__ mesh_prim_base, pyre_bvh2_node* out) {
    const uint32_t n_nodes = counters[kCounters + 1];
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n_nodes; v += gridDim.x * blockDim.x) {
        const BNode& nd = nodes[v];
        if (nd.mesh == kNoMesh) continue;
        const uint32_t first = mesh_prim_base[nd.mesh], l0 = leaves(first);
        pyre_bvh2_node r;
        for (int k = 0; k < 3; ++k) { r.bounds_min[k] = nd.lo[k]; r.bounds_max[k] = nd.hi[k]; }
        if (nd.left < 0) {
            r.offset = nd.start - first;
            r.n_primitives = (uint16_t)nd.count;
            r.axis = 0;
        } else {
            r.offset = 2 * (leaves(nd.mid) - l0) + nd.lefts;  // the right child's index
            r.n_primitives = 0;
            r.axis = (uint8_t)nd.axis;
        }
        r.pad = 0;
        out[2 * (leaves(nd.start) - l0) + nd.lefts] = r;  // one mesh per call
    }
}

__global__ void k_emit_prims(const uint32_t* __restrict__ idx, uint32_t n, const uint32_t* __restrict__ prim_mesh,
                             const uint32_t* __restrict__ mesh_prim_base, uint32_t* out) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x)
        out[p] = idx[p] - mesh_prim_base[prim_mesh[p]];
}

// Leaves of each mesh (from the leaf scan).
__global__ void k_mesh_leaves(Scan leaves, const uint32_t* __restrict__ mesh_prim_base, uint32_t n_meshes, uint32_t n,
                              uint32_t* out) {
    for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < n_meshes; m += gridDim.x * blockDim.x)
        out[m] = leaves(m + 1 < n_meshes ? mesh_prim_base[m + 1] : n) - leaves(mesh_prim_base[m]);
}

// 64-byte device nodes (GpuNode, bvh_host.h) of every mesh: the interior nodes
// in depth-first order from node_base[m] on; a mesh whose root is a leaf gets
// one node holding that leaf and an empty slot, as collapse_bvh2 does.
// Leaf children point at triangle slots, which are the build's positions.
__global__ void k_emit_gpu(const BNode* __restrict__ nodes, const uint32_t* __restrict__ counters, uint32_t n_meshes,
                           Scan leaves, const uint32_t* __restrict__ mesh_prim_base,
                           const uint32_t* __restrict__ node_base, GpuNode* out) {
    const uint32_t n_nodes = counters[kCounters + 1];
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n_nodes; v += gridDim.x * blockDim.x) {
        const BNode& nd = nodes[v];
        if (nd.mesh == kNoMesh) continue;
        const bool root = v < n_meshes;
        if (nd.left < 0 && !root) continue;
        const uint32_t l0 = leaves(mesh_prim_base[nd.mesh]);
        GpuNode g;
        auto put = [&](int s, const BNode& c) {
            float* xy = s == 0 ? g.a : g.b;
            xy[0] = c.lo[0]; xy[1] = c.hi[0]; xy[2] = c.lo[1]; xy[3] = c.hi[1];
            g.c[2 * s] = c.lo[2]; g.c[2 * s + 1] = c.hi[2];
        };
        if (nd.left < 0) {  // a root leaf
            put(0, nd);
            g.d[0] = (int32_t)nd.start; g.d[2] = (int32_t)nd.count;
            g.b[0] = INFINITY; g.b[1] = -INFINITY; g.b[2] = INFINITY; g.b[3] = -INFINITY;
            g.c[2] = INFINITY; g.c[3] = -INFINITY;
            g.d[1] = -1; g.d[3] = 0;
            out[node_base[nd.mesh]] = g;
            continue;
        }
        const int32_t kid[2] = {nd.left, nd.right};
        for (int s = 0; s < 2; ++s) {
            const BNode& c = nodes[kid[s]];
            put(s, c);
            if (c.left < 0) { g.d[s] = (int32_t)c.start; g.d[2 + s] = (int32_t)c.count; }
            else { g.d[s] = (int32_t)(node_base[nd.mesh] + (leaves(c.start) - l0) + c.lefts); g.d[2 + s] = 0; }
        }
        out[node_base[nd.mesh] + (leaves(nd.start) - l0) + nd.lefts] = g;
    }
}

// Triangle records in slot (= build position) order: (v0, local triangle id),
// e1 = v1 - v0, e2 = v2 - v0 (as pyre_scene_upload lays them out).
__global__ void k_emit_tris(const uint32_t* __restrict__ idx, uint32_t n, const uint32_t* __restrict__ prim_mesh,
                            const uint32_t* __restrict__ mesh_prim_base, const float* __restrict__ pos,
                            const uint32_t* __restrict__ vidx, float4* tris) {
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        const uint32_t t = idx[p];
        const uint32_t local = t - mesh_prim_base[prim_mesh[p]];
        const uint32_t i0 = vidx[3 * (size_t)t], i1 = vidx[3 * (size_t)t + 1], i2 = vidx[3 * (size_t)t + 2];
        const float* p0 = pos + 3 * (size_t)i0;
        const float* p1 = pos + 3 * (size_t)i1;
        const float* p2 = pos + 3 * (size_t)i2;
        tris[3 * (size_t)p] = make_float4(p0[0], p0[1], p0[2], __uint_as_float(local));
        tris[3 * (size_t)p + 1] = make_float4(p1[0] - p0[0], p1[1] - p0[1], p1[2] - p0[2], 0.0f);
        tris[3 * (size_t)p + 2] = make_float4(p2[0] - p0[0], p2[1] - p0[1], p2[2] - p0[2], 0.0f);
    }
}

int blocks_for(uint64_t n, int block = 256) { return (int)std::max<uint64_t>(1, std::min<uint64_t>((n + block - 1) / block, 1u << 20)); }

// The build's arrays, carved from one allocation of the context (base null: only the size).
struct Arena {
    char* base;
    size_t off = 0;
    template <typename T>
    T* take(size_t count) {
        off = (off + 255) & ~(size_t)255;
        T* p = reinterpret_cast<T*>(base ? base + off : nullptr);
        off += count * sizeof(T);
        return p;
    }
};

}  // namespace

// The build of M meshes (all non-empty; primitives of mesh m at
// [prim_base[m], prim_base[m + 1]) of the bound arrays). Results stay on the
// device: nodes by id (root m is node m), the leaf scan, the primitive order.
struct DeviceBvh {
    uint32_t n_prims = 0, n_meshes = 0;
    float4 *blo, *bhi, *cen;
    uint32_t *idx, *idx2, *flag, *pre, *front, *back, *prim_mesh, *block_sum, *leaf_start, *counters, *mesh_prim_base, *mesh_leaves;
    int32_t* pos_task;
    Task *tasks[2], *small;
    TaskAcc* acc[2];
    TaskState* st[2];
    BNode* nodes;

    uint32_t scan_blocks() const { return std::max(1u, (n_prims + 4 * kScanBlock - 1) / (4 * kScanBlock)); }
    uint32_t max_tasks() const { return std::max(n_meshes, n_prims / (kSmall + 1) + 1); }
    Scan scan() const { return Scan{pre, block_sum, n_prims, scan_blocks()}; }
    void carve(Arena& a) {
        const size_t N = n_prims, T = max_tasks();
        blo = a.take<float4>(N); bhi = a.take<float4>(N); cen = a.take<float4>(N);
        idx = a.take<uint32_t>(N); idx2 = a.take<uint32_t>(N); flag = a.take<uint32_t>(N); pre = a.take<uint32_t>(N);
        front = a.take<uint32_t>(N); back = a.take<uint32_t>(N); prim_mesh = a.take<uint32_t>(N);
        block_sum = a.take<uint32_t>(scan_blocks() + 1);
        leaf_start = a.take<uint32_t>(N);
        counters = a.take<uint32_t>(kCounters + 2);
        mesh_prim_base = a.take<uint32_t>(n_meshes);
        mesh_leaves = a.take<uint32_t>(n_meshes);
        pos_task = a.take<int32_t>(N);
        for (int k = 0; k < 2; ++k) { tasks[k] = a.take<Task>(T); acc[k] = a.take<TaskAcc>(T); st[k] = a.take<TaskState>(T); }
        small = a.take<Task>(N);
        nodes = a.take<BNode>(2 * N);
    }
};

// The context's build workspace for one build: given back at the end of the
// call where it holds more than `keep` bytes. A mesh that is rebuilt call after
// call keeps its arrays, about 330 B per triangle (300,007 triangles 1.82 against
// 2.02 ms with an allocation per build, 1.3 M 5.22 against 5.63); those of larger
// builds do not outlive the call. A scene upload leaves what it found, or 16 MiB:
// a scene that small is uploaded in 0.76 ms, 0.87 with an allocation.
constexpr size_t kKeepBuild = (size_t)512 << 20, kKeepUpload = (size_t)16 << 20;
struct BuildWorkspace {
    pyre_ctx* ctx;
    size_t keep;
    BuildWorkspace(pyre_ctx* c, size_t k) : ctx(c), keep(k) { ctx->building = true; }
    ~BuildWorkspace() {
        ctx->building = false;
        Workspace& ws = ctx->build_ws;
        if (ws.bytes <= keep) return;
        cudaFree(ws.ptr);
        ws = Workspace{};
    }
};

#define DTRY(expr)                                                            \
    do {                                                                      \
        cudaError_t _e = (expr);                                              \
        if (_e != cudaSuccess) return cuda_check(ctx, _e, #expr);             \
    } while (0)

static int build_device_bvh(pyre_ctx* ctx, DeviceBvh& B, const std::vector<uint32_t>& prim_base) {
    cudaStream_t st = ctx->stream;
    const uint32_t N = B.n_prims, M = B.n_meshes;
    DTRY(cudaMemcpyAsync(B.mesh_prim_base, prim_base.data(), M * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
    uint32_t* host = (uint32_t*)ctx->h_stage;  // pinned
    std::memset(host, 0, (kCounters + 2) * sizeof(uint32_t));
    host[0] = M;               // tasks of level 0
    host[kCounters + 1] = M;   // node ids: the roots
    DTRY(cudaMemcpyAsync(B.counters, host, (kCounters + 2) * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
    DTRY(cudaMemsetAsync(B.nodes, 0xff, 2 * (size_t)N * sizeof(BNode), st));  // mesh = kNoMesh
    DTRY(cudaMemsetAsync(B.leaf_start, 0, N * sizeof(uint32_t), st));
    k_init<<<blocks_for(N), 256, 0, st>>>(B.mesh_prim_base, M, N, B.prim_mesh, B.pos_task, B.idx, B.tasks[0], B.acc[0],
                                          B.small, B.counters);
    // levels in batches: as many as an even split takes, then a few at a time
    uint32_t level = 0, batch = 2;
    for (uint32_t n = N / M; n > kSmall; n /= 2) ++batch;
    const Scan pre = B.scan();
    const int pb = blocks_for(N), cb = (int)(((uint64_t)N + kChunk - 1) / kChunk);
    bool any = false;
    for (uint32_t m = 0; m < M; ++m) any = any || (m + 1 < M ? prim_base[m + 1] : N) - prim_base[m] > kSmall;
    while (any) {
        for (uint32_t k = 0; k < batch; ++k, ++level) {
            const int a = level & 1, b = a ^ 1;
            const uint64_t bound = std::min<uint64_t>(B.max_tasks(), (uint64_t)M << std::min(level, 31u));
            const int tb = blocks_for(bound, 32);
            k_box<<<cb, 256, 0, st>>>(B.pos_task, level ? B.st[b] : nullptr, B.idx, B.blo, B.bhi, B.cen, N, B.acc[a]);
            k_bin<<<cb, 256, 0, st>>>(B.pos_task, B.tasks[a], B.idx, B.blo, B.bhi, B.cen, N, B.acc[a]);
            k_decide<<<tb, 32, 0, st>>>(B.tasks[a], B.acc[a], B.counters + level % kCounters, B.st[a]);
            k_scan_local<<<B.scan_blocks(), kScanBlock, 0, st>>>(B.pos_task, B.idx, B.cen, B.st[a], N, B.flag, B.pre,
                                                                 B.block_sum);
            k_scan_sums<<<1, kScanBlock, 0, st>>>(B.block_sum, B.scan_blocks());
            k_tables<<<pb, 256, 0, st>>>(B.pos_task, B.tasks[a], B.st[a], B.flag, pre, N, B.front, B.back);
            k_scatter<<<pb, 256, 0, st>>>(B.pos_task, B.tasks[a], B.st[a], B.flag, pre, B.front, B.back, B.idx, N,
                                          B.idx2);
            std::swap(B.idx, B.idx2);
            k_finish<<<tb, 32, 0, st>>>(B.tasks[a], B.acc[a], level, pre, B.st[a], B.nodes, B.tasks[b], B.acc[b],
                                         B.small, B.leaf_start, B.counters);
        }
        DTRY(cudaMemcpyAsync(host, B.counters + level % kCounters, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        DTRY(cudaStreamSynchronize(st));
        DTRY(cudaGetLastError());
        if (host[0] == 0) break;
        batch = 3;
    }
    k_small<<<blocks_for(std::max(1u, N / 12), 4), 128, 0, st>>>(B.small, B.counters, B.blo, B.bhi, B.cen, B.idx,
                                                                 B.nodes, B.leaf_start, B.counters);
    k_scan_local<<<B.scan_blocks(), kScanBlock, 0, st>>>(nullptr, nullptr, nullptr, nullptr, N, B.leaf_start, B.pre,
                                                         B.block_sum);
    k_scan_sums<<<1, kScanBlock, 0, st>>>(B.block_sum, B.scan_blocks());
    k_mesh_leaves<<<blocks_for(M), 256, 0, st>>>(pre, B.mesh_prim_base, M, N, B.mesh_leaves);
    DTRY(cudaGetLastError());
    return PYRE_OK;
}

// Whether every index is below n_vertices (the maximum is found without an exit in the loop, which vectorizes).
static bool indices_valid(const uint32_t* indices, uint64_t n, uint32_t n_vertices) {
    uint32_t top = 0;
    for (uint64_t i = 0; i < n; ++i) top = std::max(top, indices[i]);
    return n == 0 || top < n_vertices;
}

int device_build_blas(pyre_ctx* ctx, const pyre_scene_desc* desc, const std::vector<uint32_t>& mesh_ids,
                      DeviceBlas* out) {
    cudaStream_t st = ctx->stream;
    const uint32_t M = (uint32_t)mesh_ids.size();
    std::vector<uint32_t> prim_base(M);
    uint64_t n_tri = 0, n_vert = 0;
    for (uint32_t k = 0; k < M; ++k) {
        prim_base[k] = (uint32_t)n_tri;
        n_tri += desc->meshes[mesh_ids[k]].n_triangles;
        n_vert += desc->meshes[mesh_ids[k]].n_vertices;
    }
    if (n_tri >= (1ull << 31) || 3 * n_vert >= (1ull << 32))
        return set_error(ctx, PYRE_ERR_UNSUPPORTED, "scene too large for the device BVH build");
    // all meshes' vertices, and their indices rebased to the concatenation
    std::vector<uint32_t> vidx(3 * n_tri);
    std::vector<float> pos(3 * n_vert);
    uint64_t vb = 0, tb = 0;
    for (uint32_t k = 0; k < M; ++k) {
        const pyre_mesh_desc& md = desc->meshes[mesh_ids[k]];
        std::memcpy(pos.data() + 3 * vb, md.positions, 3 * (size_t)md.n_vertices * sizeof(float));
        for (uint64_t i = 0; i < 3ull * md.n_triangles; ++i) vidx[3 * tb + i] = (uint32_t)(vb + md.indices[i]);
        vb += md.n_vertices;
        tb += md.n_triangles;
    }
    DeviceBvh B;
    B.n_prims = (uint32_t)n_tri;
    B.n_meshes = M;
    float* d_pos = nullptr;
    uint32_t *d_vidx = nullptr, *d_node_base = nullptr;
    auto layout = [&](char* base) {
        Arena a{base};
        B.carve(a);
        d_pos = a.take<float>(pos.size());
        d_vidx = a.take<uint32_t>(vidx.size());
        d_node_base = a.take<uint32_t>(M);
        return a.off;
    };
    const BuildWorkspace arrays(ctx, std::max(kKeepUpload, ctx->build_ws.bytes));
    int rc = ensure_workspace(ctx, ctx->build_ws, layout(nullptr));
    if (rc) return rc;
    layout((char*)ctx->build_ws.ptr);
    DTRY(cudaMemcpyAsync(d_pos, pos.data(), pos.size() * sizeof(float), cudaMemcpyHostToDevice, st));
    DTRY(cudaMemcpyAsync(d_vidx, vidx.data(), vidx.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
    k_tri_bounds<<<blocks_for(n_tri), 256, 0, st>>>(d_pos, d_vidx, (uint32_t)n_tri, B.blo, B.bhi, B.cen);
    rc = build_device_bvh(ctx, B, prim_base);
    if (rc) return rc;
    std::vector<uint32_t> mesh_leaves(M);
    std::vector<BNode> roots(M);
    DTRY(cudaMemcpyAsync(mesh_leaves.data(), B.mesh_leaves, M * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    DTRY(cudaMemcpyAsync(roots.data(), B.nodes, M * sizeof(BNode), cudaMemcpyDeviceToHost, st));
    DTRY(cudaStreamSynchronize(st));
    DTRY(cudaGetLastError());
    // node bases: interior nodes of each mesh (one node for a leaf root)
    std::vector<uint32_t> node_base(M);
    uint64_t total = 0;
    for (uint32_t k = 0; k < M; ++k) {
        node_base[k] = (uint32_t)total;
        total += std::max(mesh_leaves[k] - 1, 1u);
    }
    DTRY(cudaMemcpyAsync(d_node_base, node_base.data(), M * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
    GpuNode* d_nodes = nullptr;
    float4* d_tris = nullptr;
    DTRY(device_alloc(ctx, (void**)&d_nodes, std::max<uint64_t>(total, 1) * sizeof(GpuNode)));
    cudaError_t e = device_alloc(ctx, (void**)&d_tris, 3 * n_tri * sizeof(float4));
    if (e != cudaSuccess) { cudaFree(d_nodes); return cuda_check(ctx, e, "cudaMalloc(triangles)"); }
    k_emit_gpu<<<blocks_for(2 * n_tri), 256, 0, st>>>(B.nodes, B.counters, M, B.scan(), B.mesh_prim_base, d_node_base,
                                                      d_nodes);
    k_emit_tris<<<blocks_for(n_tri), 256, 0, st>>>(B.idx, (uint32_t)n_tri, B.prim_mesh, B.mesh_prim_base, d_pos, d_vidx,
                                                    d_tris);
    e = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) { cudaFree(d_nodes); cudaFree(d_tris); return cuda_check(ctx, e, "device BVH emit"); }
    out->nodes = d_nodes;
    out->n_nodes = total;
    out->tris = d_tris;
    out->root.assign(M, 0);
    out->box.assign(M, Aabb{});
    for (uint32_t k = 0; k < M; ++k) {
        out->root[k] = (int32_t)node_base[k];
        out->box[k].lo = mk3(roots[k].lo[0], roots[k].lo[1], roots[k].lo[2]);
        out->box[k].hi = mk3(roots[k].hi[0], roots[k].hi[1], roots[k].hi[2]);
    }
    return PYRE_OK;
}

}  // namespace pyre

using namespace pyre;

extern "C" int pyre_bvh_build_device(pyre_ctx* ctx, const float* positions, uint32_t n_vertices,
                                     const uint32_t* indices, uint32_t n_triangles, pyre_bvh2_node* nodes_out,
                                     uint32_t* prim_indices_out, uint32_t* n_nodes_out) {
    NvtxRange nvtx("pyre_bvh_build_device");
    if (!ctx || !positions || !indices || !nodes_out || !prim_indices_out || !n_nodes_out)
        return set_error(ctx, PYRE_ERR_INVALID, "pyre_bvh_build_device: NULL argument");
    if (!indices_valid(indices, 3ull * n_triangles, n_vertices)) return set_error(ctx, PYRE_ERR_INVALID, "index out of range");
    *n_nodes_out = 0;
    if (n_triangles == 0) return PYRE_OK;
    cudaSetDevice(ctx->device);
    cudaStream_t st = ctx->stream;
    DeviceBvh B;
    B.n_prims = n_triangles;
    B.n_meshes = 1;
    float* d_pos = nullptr;
    uint32_t *d_idx = nullptr, *d_prim = nullptr;
    pyre_bvh2_node* d_out = nullptr;
    auto layout = [&](char* base) {
        Arena a{base};
        B.carve(a);
        d_pos = a.take<float>(3 * (size_t)n_vertices);
        d_idx = a.take<uint32_t>(3 * (size_t)n_triangles);
        d_prim = a.take<uint32_t>(n_triangles);
        d_out = a.take<pyre_bvh2_node>(2 * (size_t)n_triangles);
        return a.off;
    };
    const BuildWorkspace arrays(ctx, kKeepBuild);
    int rc = ensure_workspace(ctx, ctx->build_ws, layout(nullptr));
    if (rc) return rc;
    layout((char*)ctx->build_ws.ptr);
    DTRY(cudaMemcpyAsync(d_pos, positions, 3 * (size_t)n_vertices * 4, cudaMemcpyHostToDevice, st));
    DTRY(cudaMemcpyAsync(d_idx, indices, 3 * (size_t)n_triangles * 4, cudaMemcpyHostToDevice, st));
    k_tri_bounds<<<blocks_for(n_triangles), 256, 0, st>>>(d_pos, d_idx, n_triangles, B.blo, B.bhi, B.cen);
    std::vector<uint32_t> base{0};
    rc = build_device_bvh(ctx, B, base);
    if (rc) return rc;
    k_emit_ref<<<blocks_for(2 * (uint64_t)n_triangles), 256, 0, st>>>(B.nodes, B.counters, B.scan(), B.mesh_prim_base, d_out);
    k_emit_prims<<<blocks_for(n_triangles), 256, 0, st>>>(B.idx, n_triangles, B.prim_mesh, B.mesh_prim_base, d_prim);
    uint32_t* leaves = (uint32_t*)ctx->h_stage;
    DTRY(cudaMemcpyAsync(leaves, B.mesh_leaves, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    DTRY(cudaMemcpyAsync(prim_indices_out, d_prim, n_triangles * sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    DTRY(cudaStreamSynchronize(st));
    DTRY(cudaGetLastError());
    const uint32_t n_nodes = 2 * leaves[0] - 1;
    DTRY(cudaMemcpyAsync(nodes_out, d_out, n_nodes * sizeof(pyre_bvh2_node), cudaMemcpyDeviceToHost, st));
    DTRY(cudaStreamSynchronize(st));
    *n_nodes_out = n_nodes;
    return PYRE_OK;
}
