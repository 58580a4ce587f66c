// obb_tree.cu - AABB-BVH -> OBB-tree transform (kr_cuda_bvh_obb_tree,
// src/ads/common/cuda/transforms.cu:966-1059), re-planned for the B200.
//
// The reference needs four synchronising kernels and, for the extents, lets
// every leaf walk to the root doing float CAS atomics on each ancestor
// (refit_obbs_kernel_new, :759-901): O(N * depth) contended atomics.  Here:
//
//   summary_up   bottom-up (arrival counter per node): the leaf OBB and
//                transform of every triangle (:794-834), the 7-direction
//                extremal-vertex summary of every subtree (merge left, then
//                right where strictly better; 112 B per node) and the subtree
//                leaf counts.
//   dfs_rank     each leaf's rank in depth-first order; its triangle is
//                written to that slot, so every subtree's vertices are one
//                contiguous run; each node learns its first rank.
//   candidate    node-parallel DiTO-14 candidate axes from the 14 summary
//                vertices (:676-756) and the initial extents along them.
//   extents      min/max of every subtree vertex on the node's axes, read
//                from the contiguous run: the candidate's own thread for up
//                to 12 leaves, 8 lanes for up to 32, one warp per 512-leaf unit
//                above that (listed by the candidate kernel, dealt to the
//                warps of a persistent grid); blocks of 32 leaves whose boxes
//                lie within the node's extents so far are passed over; only
//                nodes of more than one unit combine partial results, with 6
//                integer atomics per unit.
//                For a Karras tree (the fused build), tiles instead: one CTA
//                per 1,024 (256) consecutive leaves stages their triangles in
//                shared memory once and serves every larger node over them
//                from there.
//   finalize     the listed nodes' boxes (:903-964); others are finalised in
//                place.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <unordered_map>

#include "device_common.cuh"
#include "obb_device.cuh"
#include "obb_tree_host.h"
#include "obvh_transforms.h"
#include "runtime.h"
#include "sort.h"
#include "tree_device.cuh"
#include "unit_plan.h"

namespace obvh {
namespace obbtree {

using namespace tree;

constexpr int kThreads = 256;
constexpr uint32_t kCollapseLeafMax = 8;  // MAX_LEAF_SIZE (transforms.cu:65)
// A node of up to kOwnLeaves leaves is finished by the thread that finds its
// candidate: its axes are at hand, and its 96-byte record is neither written
// nor read again.  (us with the nodes of up to 8 done by the extents kernels /
// with 5, 8, 12 and 16 here: builds of 200,003 triangles 257 / 255, 247, 245,
// 245, of 500,003 438 / 438, 427, 421, -, of 2,000,000 1,446 / 1,483, 1,444,
// 1,437, 1,441; transform of 229,824 - / 266, 264, 260, 262.)
constexpr uint32_t kOwnLeaves = 12;
// Tiled extents: 1,024 leaves per tile, or 256 for up to kSmallTiles leaves, so
// that a small tree spreads over more SMs (us a build, 1,024 / 256: 1,021
// triangles 111 / 99, 10,007 157 / 141, 57,344 211 / 195, 200,003 299 / 274,
// 500,003 466 / 473, 2,000,000 1,534 / 1,614).
constexpr uint32_t kTileShiftLarge = 10, kTileShiftSmall = 8;
constexpr uint32_t kSmallTiles = 300000;
constexpr uint32_t tile_shift(uint32_t n) { return n <= kSmallTiles ? kTileShiftSmall : kTileShiftLarge; }
constexpr uint32_t tiles_of(uint32_t n) {
    return static_cast<uint32_t>((static_cast<uint64_t>(n) + (1u << tile_shift(n)) - 1) >> tile_shift(n));
}
// Ancestors of a leaf in a Karras tree over 30-bit codes with the index
// tie-break: each level lengthens the common prefix of the 62-bit (code,
// index) keys, so there are at most 62.
constexpr uint32_t kChain = 64;
// Extents items per tile kept in shared memory: of 8 lanes, and in all.  With
// the triangles they fit the 48 KB of a static allocation.
constexpr uint32_t tile_groups(uint32_t shift) { return shift == kTileShiftLarge ? 160 : 48; }
constexpr uint32_t tile_items(uint32_t shift) { return shift == kTileShiftLarge ? 320 : 224; }

struct Ctl {
    uint32_t error;
    uint32_t groups;             // PlanArgs
    unsigned long long units;
    uint32_t pad[60];
};

__device__ __forceinline__ uint32_t count_of(const uint32_t* counts, uint32_t node, uint32_t internal) {
    return node >= internal ? 1u : __ldcg(counts + node);
}

__device__ __forceinline__ uint4 leaf_face(const kr_bvh_node* nodes, const kr_uvec4* faces, uint32_t leaf) {
    const uint32_t prim = __ldg(reinterpret_cast<const uint32_t*>(nodes + leaf) + 6);
    return __ldg(reinterpret_cast<const uint4*>(faces) + prim);
}

// ---------------------------------------------------------------------------
// The walks of the two kernels below, a chain of dependent steps each: an
// arrival (a fence and an atomic at GPU scope), the sibling's outputs from L2,
// seven slabs merged one after another.  In three parts:
//   - within the warp: leaves that are close in the tree are mostly close in
//     number, so lanes that stand at one parent meet by a match and hand over
//     by shuffles, without arrivals, until no two do;
//   - across the GPU, a lane per walk, as long as more than kGroups are left
//     (every arrival checks that its parent names the child, the first too:
//     nodes whose children met in a warp have no arrivals to tell by);
//   - then eight lanes per walk, lane k < 7 with slab k and lane 7 with
//     everything else; the warp's fences stay as many as before.
// Bound by the latency of those chains with 32 warps on an SM (64 registers:
// 3 CTAs per SM 320 us where 4 take 314 and 5, spilling, 326).  Boxes and
// transforms of a given 229,824-triangle tree: 332 us with lanes alone, 328
// with groups, 323 with the meeting in the warp, 314 with the leaf boxes staged
// and 4 CTAs per SM; the 917,504-triangle ATRBVH build 2,413 -> 2,363 us.
constexpr uint32_t kGroups = 4;
constexpr uint32_t kWalkCtas = 4;


// The lane whose walk group `lane / 8` takes over (the group's own number
// among the lanes of `going`), and that lane's slab `lane % 8` (7: none).
__device__ __forceinline__ int source_lane(uint32_t going, uint32_t group) {
    for (uint32_t k = 0; k < group; ++k) going &= going - 1;
    return __ffs(static_cast<int>(going)) - 1;
}

__device__ __forceinline__ Slab take_slab(const Summary& s, int src, uint32_t sub) {
    Slab o{0.f, 0.f, 0u, 0u};
#pragma unroll
    for (uint32_t k = 0; k < 7; ++k) {
        const float lo = __shfl_sync(0xffffffffu, s.lo[k], src), hi = __shfl_sync(0xffffffffu, s.hi[k], src);
        const uint32_t ilo = __shfl_sync(0xffffffffu, s.ilo[k], src), ihi = __shfl_sync(0xffffffffu, s.ihi[k], src);
        if (sub == k) o = Slab{lo, hi, ilo, ihi};
    }
    return o;
}

__device__ __forceinline__ void store_slab(uint4* summary, uint32_t p, uint32_t k, const Slab& v) {
    __stcg(summary + 7 * static_cast<size_t>(p) + k,
           make_uint4(__float_as_uint(v.lo), __float_as_uint(v.hi), v.ilo, v.ihi));
}

// Slab k of node x's summary, x a leaf or a node that this kernel completed.
__device__ __forceinline__ Slab load_slab(const kr_bvh_node* nodes, const kr_vec3* verts, const kr_uvec4* faces,
                                          const uint4* summary, uint32_t x, uint32_t internal, uint32_t k) {
    if (x >= internal) return face_slab(verts, leaf_face(nodes, faces, x), static_cast<int>(k));
    const uint4 q = __ldcg(summary + 7 * static_cast<size_t>(x) + k);
    return Slab{__uint_as_float(q.x), __uint_as_float(q.y), q.z, q.w};
}

__device__ __forceinline__ Slab slab_from(const Summary& s, int k, uint32_t lane) {
    return Slab{__shfl_sync(0xffffffffu, s.lo[k], lane), __shfl_sync(0xffffffffu, s.hi[k], lane),
                __shfl_sync(0xffffffffu, s.ilo[k], lane), __shfl_sync(0xffffffffu, s.ihi[k], lane)};
}

// The boxes and transforms of a warp's leaves, consecutive records from obbs
// and xfs on: staged in shared memory (rows of 15 and of 20 words: no two
// lanes of an access in one bank) and written out in full sectors.
struct LeafStage {
    float4 xf[32 * 5];
    float box[32 * 15];
};

__device__ __forceinline__ void leaf_boxes(LeafStage& st, bool live, const kr_vec3* verts, uint4 face, uint32_t lane,
                                           kr_obb3* obbs, kr_mat4* xfs) {
    const uint32_t m = __popc(__ballot_sync(0xffffffffu, live));  // the live lanes come first
    if (live)
        leaf_box(load_vertex(verts, face.x), load_vertex(verts, face.y), load_vertex(verts, face.z),
                 reinterpret_cast<kr_obb3*>(st.box + 15 * lane), reinterpret_cast<kr_mat4*>(st.xf + 5 * lane));
    __syncwarp();
#pragma unroll
    for (uint32_t k = lane; k < 32 * 15; k += 32)
        if (k < 15 * m) reinterpret_cast<float*>(obbs)[k] = st.box[k];
#pragma unroll
    for (uint32_t k = lane; k < 32 * 4; k += 32)
        if (k < 4 * m) reinterpret_cast<float4*>(xfs)[k] = st.xf[5 * (k >> 2) + (k & 3)];
}

__global__ void __launch_bounds__(kThreads, kWalkCtas) summary_up_kernel(const kr_bvh_node* nodes, const uint32_t* parents,
                                                              const kr_vec3* verts, const kr_uvec4* faces,
                                                              uint32_t n, uint32_t internal, uint4* summary,
                                                              uint32_t* counts, uint32_t* visits, kr_obb3* obbs,
                                                              kr_mat4* xfs, uint32_t* err) {
    __shared__ LeafStage stage[kThreads / 32];
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31;
    bool live = j < n;
    const uint32_t leaf = internal + (live ? j : 0u);
    const uint4 face = leaf_face(nodes, faces, leaf);
    const size_t first_leaf = static_cast<size_t>(internal) + (j - lane);
    leaf_boxes(stage[threadIdx.x >> 5], live, verts, face, lane, obbs + first_leaf, xfs + first_leaf);
    Summary own;
    leaf_summary(verts, face, own);
    if (internal == 0) return;
    uint32_t child = leaf, p = live ? parents[leaf] : kNoParent, grand = kNoParent;
    uint32_t L = 0, R = 0, steps = 0, going, count = 1;
    // p's children and its parent are final before this kernel
    const auto at_parent = [&] {
        if (!live) return;
        if (steps > internal || p >= internal) {
            if (p != kNoParent) atomicOr(err, kErrCycle);
            live = false;
            return;
        }
        const uint32_t* w = reinterpret_cast<const uint32_t*>(nodes + p);
        L = __ldg(w + 6);
        R = __ldg(w + 7);
        grand = __ldg(parents + p);
    };
    at_parent();
    for (;;) {
        uint32_t partner;
        const bool pair = paired(live, p, child, L, R, lane, partner);
        if (!__any_sync(0xffffffffu, pair)) break;
        const bool mine = pair && L == child;  // the left child's lane goes on
        const uint32_t theirs = __shfl_sync(0xffffffffu, count, partner);
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            const Slab o = slab_from(own, k, partner);
            if (mine) {
                const Slab m = merge_slab(slab_of(own, k), o);
                set_slab(own, k, m);
                store_slab(summary, p, k, m);
            }
        }
        live = live && (mine || !pair);
        if (mine) {
            count += theirs;
            __stcg(counts + p, count);
            child = p;
            p = grand;
            ++steps;
            at_parent();
        }
        __syncwarp();
    }
    for (;;) {
        going = __ballot_sync(0xffffffffu, live);
        if (__popc(going) <= kGroups) break;
        if (!live) continue;
        const bool second = arrive(visits + p) != 0;
        const uint32_t other = (L == child) ? R : L;
        const bool bad = (L != child && R != child) || other >= internal + n;
        if (bad) atomicOr(err, kErrBadInput);
        live = second && !bad;
        if (!live) continue;
        Summary o;
        if (other >= internal) leaf_summary(verts, leaf_face(nodes, faces, other), o);
        else load_summary(summary + 7 * static_cast<size_t>(other), o);
        if (L == child) {
            merge_right(own, o);
        } else {
            merge_right(o, own);
            own = o;
        }
        store_summary(summary + 7 * static_cast<size_t>(p), own);
        count += count_of(counts, other, internal);
        __stcg(counts + p, count);
        child = p;
        p = grand;
        ++steps;
        at_parent();
    }
    if (going == 0) return;
    const uint32_t sub = lane & 7, group = lane >> 3;
    live = group < __popc(going);
    const int src = live ? source_lane(going, group) : 0;
    Slab mine = take_slab(own, src, sub);
    child = __shfl_sync(0xffffffffu, child, src);
    p = __shfl_sync(0xffffffffu, p, src);
    steps = __shfl_sync(0xffffffffu, steps, src);
    L = __shfl_sync(0xffffffffu, L, src);
    R = __shfl_sync(0xffffffffu, R, src);
    grand = __shfl_sync(0xffffffffu, grand, src);
    count = __shfl_sync(0xffffffffu, count, src);
    __syncwarp();
    while (__any_sync(0xffffffffu, live)) {
        uint32_t before = 0;
        if (live && sub == 0) before = arrive(visits + p);
        before = __shfl_sync(0xffffffffu, before, 0, 8);
        __syncwarp();  // orders the group's loads after lane 0's acquire
        const uint32_t other = (L == child) ? R : L;
        const bool bad = live && ((L != child && R != child) || other >= internal + n);
        if (bad && sub == 0) atomicOr(err, kErrBadInput);
        live = live && before != 0 && !bad;
        if (live) {
            if (sub < 7) {
                const Slab sib = load_slab(nodes, verts, faces, summary, other, internal, sub);
                mine = merge_slab(L == child ? mine : sib, L == child ? sib : mine);
                store_slab(summary, p, sub, mine);
            } else {
                count += count_of(counts, other, internal);
                __stcg(counts + p, count);
            }
            child = p;
            p = grand;
            ++steps;
            at_parent();
        }
        __syncwarp();  // the group's outputs before lane 0's next release
    }
}

// ---------------------------------------------------------------------------
// One leaf-to-root walk doing, on any binary tree, what the LBVH refit
// (lbvh.cu:399-457), summary_up above and the collapse marking
// (transforms.cu:65-136) do in three: internal bounds (kr_aabb_expand of the
// children), counts, SAH costs (the collapse's rule when collapsing, the
// LBVH's otherwise), collapse marks and collapsed records, the 7-direction
// summaries and the leaf boxes.  The arriving thread carries its own child's
// values and reads only the sibling's.
struct WalkArgs {
    kr_bvh_node* nodes;       // children and leaf boxes in; internal bounds out
    kr_bvh_node* collapsed;   // null: no collapse; else every record, with marks
    const uint32_t* parents;
    const kr_vec3* verts;
    const uint4* faces;
    uint32_t n;
    uint32_t* counts;
    float* costs;
    uint8_t* flags;           // null with collapsed
    float ci, ct;
    uint4* summary;           // null: no summaries or leaf boxes
    kr_obb3* obbs;
    kr_mat4* xfs;
    uint32_t* visits;
    uint32_t* err;
};

// nPrimitives = 0xFFFF, the low half of word 8
__device__ __forceinline__ void mark_hidden(kr_bvh_node* collapsed, uint32_t i) {
    unsigned short* h = reinterpret_cast<unsigned short*>(reinterpret_cast<uint32_t*>(collapsed + i) + 8);
    __stcg(h, static_cast<unsigned short>(0xffffu));
}

// A completed node as its parent's walk needs it: bounds, cost and count.
struct Done {
    float lo[3], hi[3], cost;
    uint32_t count;
};

__device__ __forceinline__ Done done_from(const Done& d, uint32_t lane) {
    Done o;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        o.lo[k] = __shfl_sync(0xffffffffu, d.lo[k], lane);
        o.hi[k] = __shfl_sync(0xffffffffu, d.hi[k], lane);
    }
    o.cost = __shfl_sync(0xffffffffu, d.cost, lane);
    o.count = __shfl_sync(0xffffffffu, d.count, lane);
    return o;
}

__device__ __forceinline__ Done load_done(const WalkArgs& a, uint32_t x) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(a.nodes + x);
    Done d;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        d.lo[k] = __uint_as_float(__ldcg(w + k));
        d.hi[k] = __uint_as_float(__ldcg(w + 3 + k));
    }
    d.count = __ldcg(a.counts + x);
    d.cost = __ldcg(a.costs + x);
    return d;
}

// Node p (children L and R, word 8 of its record) from its children: bounds,
// count, cost and collapse marks, all written here.
__device__ __forceinline__ Done complete(const WalkArgs& a, uint32_t p, uint32_t L, uint32_t R, uint32_t w8,
                                         const Done& l, const Done& r) {
    Done o;
#pragma unroll
    for (int k = 0; k < 3; ++k) {  // kr_aabb_expand(left, right)
        o.lo[k] = kmin(kmin(l.lo[k], r.lo[k]), r.hi[k]);
        o.hi[k] = kmax(kmax(l.hi[k], r.lo[k]), r.hi[k]);
    }
    uint32_t* w = reinterpret_cast<uint32_t*>(a.nodes + p);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        __stcg(w + k, __float_as_uint(o.lo[k]));
        __stcg(w + 3 + k, __float_as_uint(o.hi[k]));
    }
    if (a.collapsed) {
        uint32_t* cw = reinterpret_cast<uint32_t*>(a.collapsed + p);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            __stcg(cw + k, __float_as_uint(o.lo[k]));
            __stcg(cw + 3 + k, __float_as_uint(o.hi[k]));
        }
        __stcg(cw + 6, L);
        __stcg(cw + 7, R);
        __stcg(cw + 8, w8);
    }
    o.count = l.count + r.count;
    __stcg(a.counts + p, o.count);
    const float area = box_area(o.lo, o.hi);
    if (a.collapsed) {
        // bvh_mark_collapse_kernel (transforms.cu:111-133)
        const float node_cost = a.ci * area + l.cost + r.cost;
        const float leaf_cost = a.ct * area * static_cast<float>(o.count);
        if (leaf_cost < node_cost && o.count <= kCollapseLeafMax) {
            o.cost = leaf_cost;
            a.flags[p] = 1;
            a.flags[L] = 1;
            a.flags[R] = 1;
            mark_hidden(a.collapsed, L);
            mark_hidden(a.collapsed, R);
        } else {
            o.cost = node_cost;
        }
    } else {
        o.cost = 1.2f * area + r.cost + l.cost;  // calculate_aabbs_kernel (lbvh.cu:452)
    }
    __stcg(a.costs + p, o.cost);
    return o;
}

__global__ void __launch_bounds__(kThreads, kWalkCtas) walk_kernel(WalkArgs a) {
    __shared__ LeafStage stage[kThreads / 32];
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t internal = a.n - 1;
    const bool collapse = a.collapsed != nullptr;
    const bool slabs = a.summary != nullptr;
    bool live = j < a.n;
    const uint32_t leaf = internal + (live ? j : 0u);
    Done own;
    uint32_t prim;
    {
        // the warp's leaf records are consecutive: read, and copied to the
        // collapsed array, as one run of words
        LeafStage& st = stage[threadIdx.x >> 5];
        const uint32_t first = j - lane, words = first < a.n ? 9 * min(32u, a.n - first) : 0u;
        const uint32_t* src = reinterpret_cast<const uint32_t*>(a.nodes + internal + first);
        uint32_t* dst = collapse ? reinterpret_cast<uint32_t*>(a.collapsed + internal + first) : nullptr;
        uint32_t* row = reinterpret_cast<uint32_t*>(st.box);
#pragma unroll
        for (uint32_t k = lane; k < 32 * 9; k += 32) {
            const uint32_t v = k < words ? __ldg(src + k) : 0u;
            row[k] = v;
            if (collapse && k < words) __stcg(dst + k, v);
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            own.lo[k] = __uint_as_float(row[9 * lane + k]);
            own.hi[k] = __uint_as_float(row[9 * lane + 3 + k]);
        }
        prim = row[9 * lane + 6];
        __syncwarp();
    }
    // leaf cost: ct * area in the collapse (transforms.cu:97), 1 * area in the LBVH (lbvh.cu:427)
    own.cost = (collapse ? a.ct : 1.0f) * box_area(own.lo, own.hi);
    own.count = 1;
    if (live) {
        __stcg(a.costs + leaf, own.cost);
        __stcg(a.counts + leaf, 1u);
    }
    Summary sum;
    if (slabs) {
        const uint4 face = __ldg(a.faces + prim);
        const size_t first_leaf = static_cast<size_t>(internal) + (j - lane);
        leaf_boxes(stage[threadIdx.x >> 5], live, a.verts, face, lane, a.obbs + first_leaf, a.xfs + first_leaf);
        leaf_summary(a.verts, face, sum);
    }
    const kr_uvec4* faces = reinterpret_cast<const kr_uvec4*>(a.faces);
    uint32_t child = leaf, p = live ? a.parents[leaf] : kNoParent, grand = kNoParent;
    uint32_t L = 0, R = 0, w8 = 0, steps = 0, going;
    // p's children, its record's word 8 and its parent are final before this kernel
    const auto at_parent = [&] {
        if (!live) return;
        if (steps > internal || p >= internal) {
            if (p != kNoParent) atomicOr(a.err, kErrCycle);
            live = false;
            return;
        }
        const uint32_t* w = reinterpret_cast<const uint32_t*>(a.nodes + p);
        L = __ldg(w + 6);
        R = __ldg(w + 7);
        w8 = __ldg(w + 8);
        grand = __ldg(a.parents + p);
    };
    const auto go_up = [&] {
        child = p;
        p = grand;
        ++steps;
        at_parent();
    };
    at_parent();
    for (;;) {
        uint32_t partner;
        const bool pair = paired(live, p, child, L, R, lane, partner);
        if (!__any_sync(0xffffffffu, pair)) break;
        const bool mine = pair && L == child;  // the left child's lane goes on
        const Done o = done_from(own, partner);
        if (mine) own = complete(a, p, L, R, w8, own, o);
        if (slabs) {
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                const Slab r = slab_from(sum, k, partner);
                if (mine) {
                    const Slab m = merge_slab(slab_of(sum, k), r);
                    set_slab(sum, k, m);
                    store_slab(a.summary, p, k, m);
                }
            }
        }
        live = live && (mine || !pair);
        if (mine) go_up();
        __syncwarp();  // this round's outputs before the next one's marks
    }
    for (;;) {
        going = __ballot_sync(0xffffffffu, live);
        if (__popc(going) <= kGroups) break;
        if (!live) continue;
        const bool second = arrive(a.visits + p) != 0;
        const bool from_left = L == child;
        const uint32_t other = from_left ? R : L;
        const bool bad = (L != child && R != child) || other >= internal + a.n;
        if (bad) atomicOr(a.err, kErrBadInput);
        live = second && !bad;
        if (!live) continue;
        const Done o = load_done(a, other);
        own = complete(a, p, L, R, w8, from_left ? own : o, from_left ? o : own);
        if (slabs) {
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                const Slab sib = load_slab(a.nodes, a.verts, faces, a.summary, other, internal, k);
                const Slab mine = slab_of(sum, k);
                const Slab m = merge_slab(from_left ? mine : sib, from_left ? sib : mine);
                set_slab(sum, k, m);
                store_slab(a.summary, p, k, m);
            }
        }
        go_up();
    }
    if (going == 0) return;
    const uint32_t sub = lane & 7, group = lane >> 3;
    live = group < __popc(going);
    const int src = live ? source_lane(going, group) : 0;
    Slab mine{0.f, 0.f, 0u, 0u};
    if (slabs) mine = take_slab(sum, src, sub);
    own = done_from(own, src);
    child = __shfl_sync(0xffffffffu, child, src);
    p = __shfl_sync(0xffffffffu, p, src);
    steps = __shfl_sync(0xffffffffu, steps, src);
    L = __shfl_sync(0xffffffffu, L, src);
    R = __shfl_sync(0xffffffffu, R, src);
    w8 = __shfl_sync(0xffffffffu, w8, src);
    grand = __shfl_sync(0xffffffffu, grand, src);
    __syncwarp();
    while (__any_sync(0xffffffffu, live)) {
        uint32_t before = 0;
        if (live && sub == 0) before = arrive(a.visits + p);
        before = __shfl_sync(0xffffffffu, before, 0, 8);
        __syncwarp();  // orders the group's loads after lane 0's acquire
        const bool from_left = L == child;
        const uint32_t other = from_left ? R : L;
        const bool bad = live && ((L != child && R != child) || other >= internal + a.n);
        if (bad && sub == 0) atomicOr(a.err, kErrBadInput);
        live = live && before != 0 && !bad;
        if (live) {
            if (sub == 7) {
                const Done o = load_done(a, other);
                own = complete(a, p, L, R, w8, from_left ? own : o, from_left ? o : own);
            } else if (slabs) {
                const Slab sib = load_slab(a.nodes, a.verts, faces, a.summary, other, internal, sub);
                mine = merge_slab(from_left ? mine : sib, from_left ? sib : mine);
                store_slab(a.summary, p, sub, mine);
            }
            go_up();
        }
        __syncwarp();  // the group's outputs before lane 0's next release
    }
}

kr_error enqueue_walk(kr_bvh_node* nodes, const uint32_t* parents, const kr_vec3* verts, const kr_uvec4* faces,
                      uint32_t n, uint32_t* counts, float* costs, kr_obb3* obbs, kr_mat4* xfs, void* obb_workspace,
                      kr_bvh_node* collapsed, uint8_t* flags, float ci, float ct, uint32_t* visits, uint32_t* err,
                      cudaStream_t s) {
    if (n == 0) return kr_success;
    if (!nodes || !parents || !verts || !faces || !counts || !costs || !visits || !err)
        return "enqueue_walk: null pointer argument";
    if (obb_workspace && (!obbs || !xfs)) return "enqueue_walk: summaries need the leaf boxes' outputs";
    if ((collapsed == nullptr) != (flags == nullptr)) return "enqueue_walk: collapsed records and marks go together";
    WalkArgs a{nodes, collapsed, parents, verts, reinterpret_cast<const uint4*>(faces), n, counts, costs, flags, ci, ct,
               obb_workspace ? reinterpret_cast<uint4*>(static_cast<char*>(obb_workspace) + layout(n).summary)
                             : nullptr,
               obbs, xfs, visits, err};
    if (n > 1) OBVH_TRY_CUDA(cudaMemsetAsync(visits, 0, 4ull * (n - 1), s));
    {
        ProfScope prof_scope_("walk_kernel", s);
        walk_kernel<<<(n + kThreads - 1) / kThreads, kThreads, 0, s>>>(a);
    }
    OBVH_TRY_CUDA(cudaGetLastError());
    return kr_success;
}

// DFS rank of every leaf (left subtree first); the leaf's triangle goes to
// that slot of `tris`; the leaf is the first of every ancestor it reaches
// through left children only.
__global__ void __launch_bounds__(kThreads) dfs_rank_kernel(const kr_bvh_node* nodes, const uint32_t* parents,
                                                            const uint32_t* counts, const kr_vec3* verts,
                                                            const kr_uvec4* faces, uint32_t n, uint32_t internal,
                                                            uint32_t* first, float* tris, uint32_t* rank_prims,
                                                            uint32_t* err) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n || *err) return;  // an earlier pass found a malformed tree
    const uint32_t leaf = internal + j;
    uint32_t rank = 0;
    uint32_t child = leaf, p = parents[leaf];
    for (uint32_t steps = 0; p != kNoParent; ++steps) {
        if (steps > internal || p >= internal) {
            atomicOr(err, kErrCycle);
            return;
        }
        const uint32_t* w = reinterpret_cast<const uint32_t*>(nodes + p);
        const uint32_t L = __ldg(w + 6);
        if (L != child) rank += count_of(counts, L, internal);
        child = p;
        p = parents[p];
    }
    if (rank >= n) {
        atomicOr(err, kErrBadInput);
        return;
    }
    rank_prims[rank] = __ldg(reinterpret_cast<const uint32_t*>(nodes + leaf) + 6);
    const uint4 face = leaf_face(nodes, faces, leaf);
    const f3 a = load_vertex(verts, face.x), b = load_vertex(verts, face.y), c = load_vertex(verts, face.z);
    float* t = tris + 9 * static_cast<size_t>(rank);
    t[0] = a.x; t[1] = a.y; t[2] = a.z; t[3] = b.x; t[4] = b.y; t[5] = b.z; t[6] = c.x; t[7] = c.y; t[8] = c.z;
    child = leaf;
    p = parents[leaf];
    while (p != kNoParent && __ldg(reinterpret_cast<const uint32_t*>(nodes + p) + 6) == child) {
        first[p] = rank;
        child = p;
        p = parents[p];
    }
}

// The nodes that a candidate launch takes.  Tiled: a thread per node, extents in tiles; listed: those of chain.list
// (FrameNodes::kAcross), extents in tiles; planned: a thread per node, extents
// by plan_node's lists.
enum class Nodes { kTiled, kListed, kPlanned };

struct ChainArgs {
    const uint32_t* parents;  // null: per-node extents, no chains
    const uint32_t* first;
    uint32_t n;
    uint32_t walker_blocks;   // leading CTAs that walk the tile chains, or box the blocks of leaves
    uint32_t* chains;
    uint32_t* chain_counts;
    uint32_t* err;
    uint32_t* arrivals;       // tiles: per node over several tiles, the tiles done with it
    float nz;                 // -0.0f (tree::mul2)
    uint32_t which;           // FrameNodes: all nodes, or those inside / across aligned leaf blocks
    uint32_t block_shift;     // the blocks hold 2^block_shift leaves
    uint32_t tile_shift;      // the tiles 2^tile_shift
    // Without tiles: the leaves' triangles in depth-first order, the boxes of
    // each 32 of them (block_box), the outputs for the nodes of up to
    // kOwnLeaves leaves (finished by their candidate's thread) and the plan
    // of the others (plan_node).
    const float* tris;
    float* boxes;
    kr_obb3* obbs;
    kr_mat4* xfs;
    uint32_t* plan;
    unsigned long long* plan_start;
    UnitPlan units_of;
    uint32_t* groups;
    unsigned long long* units;
    const uint32_t* list;     // kAcross: the nodes, list_count of them
    const uint32_t* list_count;
};

// The ancestors of tile tau's first leaf (side 0) and last leaf (side 1) whose
// leaf ranges are not inside the tile: the nodes the tile serves partially.
// A node on both chains is listed on side 0 only.
__device__ void walk_chain(const ChainArgs& c, const uint32_t* counts, uint32_t w) {
    const uint32_t tile = 1u << c.tile_shift;
    if (w >= 2 * ((c.n + tile - 1) >> c.tile_shift)) return;
    const uint32_t tau = w >> 1, side = w & 1;
    const uint32_t t0 = tau << c.tile_shift, tend = min(t0 + tile, c.n);
    const uint32_t internal = c.n - 1;
    uint32_t* out = c.chains + static_cast<size_t>(w) * kChain;
    uint32_t count = 0;
    uint32_t p = c.parents[internal + (side ? tend - 1 : t0)];
    for (uint32_t steps = 0; p != kNoParent; ++steps) {
        if (p >= internal || steps >= kChain) {
            atomicOr(c.err, kErrBadInput);
            break;
        }
        const uint32_t f = __ldg(c.first + p), cnt = __ldg(counts + p);
        if (side && f <= t0) break;  // from here on the nodes hold the first leaf too
        if (f < t0 || f + cnt > tend) out[count++] = p;
        p = __ldg(c.parents + p);
    }
    c.chain_counts[w] = count;
}

// The box of leaves 32k to 32k + 31 (of n, in depth-first order), for
// may_extend: six rows of one float per block.
__device__ void block_box(const float* tris, uint32_t n, uint32_t k, uint32_t lane, float* boxes) {
    const uint32_t blocks = (n + 31) / 32;
    if (k >= blocks) return;
    float lo[3] = {kInf, kInf, kInf}, hi[3] = {-kInf, -kInf, -kInf};
    if (32 * k + lane < n) {
        const float* v = tris + 9 * static_cast<size_t>(32 * k + lane);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float a = __ldg(v + d), b = __ldg(v + 3 + d), c = __ldg(v + 6 + d);
            lo[d] = min3f(a, b, c);
            hi[d] = max3f(a, b, c);
        }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float l = warp_min(lo[d]), h = warp_max(hi[d]);
        if (lane == 0) {
            boxes[static_cast<size_t>(d) * blocks + k] = l;
            boxes[static_cast<size_t>(3 + d) * blocks + k] = h;
        }
    }
}

// Lists node a for extents_units_kernel (every lane of a warp calls it): nodes
// of up to kGroupLeaves leaves from the back of chain.plan, groups of them in
// all; larger ones from the front, with the number of the first of their
// units.  *units holds their units in its low bits and the nodes listed in
// front above them (unit_plan), so that both grow by one addition and the
// starts ascend.  A warp adds once.
__device__ __forceinline__ void plan_node(const ChainArgs& c, bool valid, uint32_t a, uint32_t cnt) {
    const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1u, internal = c.n - 1;
    const bool big = valid && cnt > kGroupLeaves, mid = valid && cnt > kOwnLeaves && !big;
    const uint32_t mids = __ballot_sync(0xffffffffu, mid), bigs = __ballot_sync(0xffffffffu, big);
    if (mids) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(c.groups, static_cast<uint32_t>(__popc(mids)));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (mid) c.plan[internal - 1 - (base + __popc(mids & below))] = a;
    }
    if (bigs) {
        const uint32_t own = big ? ((cnt - 1) >> c.units_of.unit_shift) + 1 : 0u;
        uint64_t incl = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t v = __shfl_up_sync(0xffffffffu, incl, d);
            if (static_cast<int>(lane) >= d) incl += v;
        }
        const uint64_t sum = __shfl_sync(0xffffffffu, incl, 31);
        unsigned long long base = 0;
        if (lane == 0)
            base = atomicAdd(c.units, (static_cast<unsigned long long>(__popc(bigs)) << c.units_of.unit_bits) + sum);
        base = __shfl_sync(0xffffffffu, base, 0);
        const uint32_t at = static_cast<uint32_t>(base >> c.units_of.unit_bits) + __popc(bigs & below);
        if (big && at < internal) {
            c.plan[at] = a;
            c.plan_start[at] = (base & ((1ull << c.units_of.unit_bits) - 1)) + incl - own;
        }
    }
}

__device__ __forceinline__ Cand cand_of(const Summary& s, const Candidate& c) {
    Cand out;
    out.ax[0] = c.b0.x; out.ax[1] = c.b0.y; out.ax[2] = c.b0.z;
    out.ax[3] = c.b1.x; out.ax[4] = c.b1.y; out.ax[5] = c.b1.z;
    out.ax[6] = c.b2.x; out.ax[7] = c.b2.y; out.ax[8] = c.b2.z;
    out.olo[0] = c.lo.x; out.olo[1] = c.lo.y; out.olo[2] = c.lo.z;
    out.ohi[0] = c.hi.x; out.ohi[1] = c.hi.y; out.ohi[2] = c.hi.z;
#pragma unroll
    for (int k = 0; k < 3; ++k) { out.alo[k] = s.lo[k]; out.ahi[k] = s.hi[k]; }
    out.pad[0] = out.pad[1] = out.pad[2] = 0.f;
    return out;
}

// The candidate of internal node a, stored for the extents kernels with the
// initial keys of a node that several units or tiles share.  Without tiles a
// node of up to kOwnLeaves leaves is finished here.
template <Nodes kNodes>
__device__ __forceinline__ void candidate_node(uint32_t a, const uint4* summary, const kr_vec3* verts,
                                               const uint32_t* counts, Cand* cand, uint32_t* keys, const ChainArgs& chain) {
    Summary s;
    const Candidate c = summary_candidate<Src::kL2, Src::kReadOnly>(summary, verts, a, chain.nz, s);
    const Cand out = cand_of(s, c);
    const uint32_t cnt = counts[a];  // (not held over the search)
    if (cnt <= kOwnLeaves) {
        float lo[3] = {c.lo.x, c.lo.y, c.lo.z}, hi[3] = {c.hi.x, c.hi.y, c.hi.z};
        const float* t = chain.tris + 9 * static_cast<size_t>(__ldg(chain.first + a));
        const Axes ax = cand_axes(out, chain.nz);
        for (uint32_t i = 0; i < cnt; ++i) project_tri(t + 9 * i, ax, lo, hi);
        finalize_node(out, mk3(lo[0], lo[1], lo[2]), mk3(hi[0], hi[1], hi[2]), chain.obbs + a, chain.xfs + a);
        return;
    }
    float4* dst = reinterpret_cast<float4*>(cand + a);
    const float4* src = reinterpret_cast<const float4*>(&out);
#pragma unroll
    for (int q = 0; q < 6; ++q) dst[q] = src[q];
    bool shared;
    if (kNodes != Nodes::kPlanned) {
        const uint32_t f = __ldg(chain.first + a);
        shared = (f >> chain.tile_shift) != ((f + cnt - 1) >> chain.tile_shift);
        if (shared) chain.arrivals[a] = 0u;  // counted up by extents_tile_kernel
    } else {
        shared = cnt > (1u << chain.units_of.unit_shift);
    }
    if (shared) {
        uint32_t* k = keys + 6 * static_cast<size_t>(a);
        k[0] = f2key(c.lo.x); k[1] = f2key(c.lo.y); k[2] = f2key(c.lo.z);
        k[3] = f2key(c.hi.x); k[4] = f2key(c.hi.y); k[5] = f2key(c.hi.z);
    }
}

// One instantiation for each kind of nodes, so that each holds one inlined copy
// of the search and nothing of the others (fewer spills).
//
// 16 warps on an SM at 128 registers; in CTAs of 128 threads the next four warps
// start as soon as four are done (builds of 57,344 triangles 172.6 -> 169.3 us,
// 2,000,000 1,439 -> 1,424; with CTAs of 64 169.3 and 1,442).
constexpr int kCandThreads = 128;
constexpr int kCandCtas = 4;
template <Nodes kNodes>
__global__ void __launch_bounds__(kCandThreads, kCandCtas) candidate_kernel(const uint4* summary, const kr_vec3* verts,
                                                                            const uint32_t* counts, uint32_t internal,
                                                                            Cand* cand, uint32_t* keys,
                                                                            const uint32_t* err, ChainArgs chain) {
    if constexpr (kNodes == Nodes::kListed) {
        // the listed nodes (written by the walk that completed them), a
        // grid-stride loop so that warps stay full
        const uint32_t total = min(*chain.list_count, internal);
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
            const uint32_t a = chain.list[i];
            if (a >= internal) {
                atomicOr(chain.err, kErrBadInput);
                continue;
            }
            if (*err) continue;
            candidate_node<kNodes>(a, summary, verts, counts, cand, keys, chain);
        }
        return;
    } else {
        if (blockIdx.x < chain.walker_blocks) {
            const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
            if (*err) return;
            if constexpr (kNodes == Nodes::kTiled) walk_chain(chain, counts, w);
            else block_box(chain.tris, chain.n, w >> 5, threadIdx.x & 31, chain.boxes);
            return;
        }
        const uint32_t a = (blockIdx.x - chain.walker_blocks) * blockDim.x + threadIdx.x;
        // malformed tree: no summaries to read; nothing is planned after this
        const bool valid = a < internal && !*err;
        if constexpr (kNodes == Nodes::kPlanned) plan_node(chain, valid, a, valid ? counts[a] : 0u);
        if (!valid) return;
        if (chain.which == static_cast<uint32_t>(FrameNodes::kInside)) {
            const uint32_t f = __ldg(chain.first + a), cnt = __ldg(counts + a);
            if ((f >> chain.block_shift) != ((f + cnt - 1) >> chain.block_shift)) return;
        }
        candidate_node<kNodes>(a, summary, verts, counts, cand, keys, chain);
    }
}

// The planned nodes (plan_node): eight lanes per node of up to kGroupLeaves
// leaves, then the units (unit_plan) of the larger ones, a warp each, dealt
// round-robin so that big and small nodes spread over the warps.  In a unit,
// only the blocks of 32 leaves that could extend the node are projected
// (may_extend).  All extents go to the keys; finalize_multi_kernel builds the
// boxes, a thread per node.
//
// Bound by the latency of a unit: its search, its node's records, its blocks.
// (Before, the units were found by a search among all nodes' starts and a step
// for every node without units in between, after a scan over all nodes; nodes
// of up to 32 leaves were a thread's.  Boxes and transforms of 229,824
// triangles 314 -> 260 us, the 917,504-triangle ATRBVH 2,353 -> 2,270 us.)
__global__ void __launch_bounds__(kThreads) extents_units_kernel(const Cand* cand, const uint32_t* counts,
                                                                 const uint32_t* first, const float* tris,
                                                                 const uint32_t* plan,
                                                                 const unsigned long long* plan_start, UnitPlan units_of,
                                                                 uint32_t internal, const uint32_t* err,
                                                                 const uint32_t* group_count,
                                                                 const unsigned long long* unit_count, uint32_t* keys,
                                                                 const float* boxes, float nz) {
    if (*err) return;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t nblocks = (internal + 1 + 31) / 32;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const uint32_t groups = min(*group_count, internal);
    for (uint32_t g0 = 4 * w; g0 < groups; g0 += 4 * warps) {
        const uint32_t g = g0 + (lane >> 3), sub = lane & 7;
        const bool live = g < groups;
        const uint32_t a = __ldg(plan + (internal - 1 - (live ? g : g0)));
        const Cand c = load_cand(cand, a);
        float lo[3], hi[3];
        group_extents<From::kGlobal>(tris + 9 * static_cast<size_t>(__ldg(first + a)), live ? __ldg(counts + a) : 0u,
                                     cand_axes(c, nz), lo, hi);
        if (live && sub < 6) {
            const float v = sub == 0 ? fminf(c.olo[0], lo[0]) : sub == 1 ? fminf(c.olo[1], lo[1])
                          : sub == 2 ? fminf(c.olo[2], lo[2]) : sub == 3 ? fmaxf(c.ohi[0], hi[0])
                          : sub == 4 ? fmaxf(c.ohi[1], hi[1]) : fmaxf(c.ohi[2], hi[2]);
            keys[6 * static_cast<size_t>(a) + sub] = f2key(v);
        }
    }
    const uint32_t listed = static_cast<uint32_t>(min(*unit_count >> units_of.unit_bits, static_cast<unsigned long long>(internal)));
    const uint64_t total = *unit_count & ((1ull << units_of.unit_bits) - 1);
    for (uint64_t u = w; u < total; u += warps) {
        uint32_t at = 0, end_at = listed;  // the last node whose first unit is <= u owns it
        while (end_at - at > 1) {
            const uint32_t step = (end_at - at + 31) / 32, probe = at + step * lane;
            const uint32_t in = __ballot_sync(0xffffffffu, probe < end_at && __ldg(plan_start + probe) <= u);
            at += step * (31 - __clz(static_cast<int>(in | 1u)));
            end_at = min(end_at, at + step);
        }
        const uint32_t a = __ldg(plan + at);
        const uint32_t cnt = __ldg(counts + a), f = __ldg(first + a);
        const Cand c = load_cand(cand, a);
        const uint32_t begin = static_cast<uint32_t>(u - __ldg(plan_start + at)) << units_of.unit_shift;
        // leaves [b, e); of the blocks of 32 those that could extend the node
        const uint32_t b = f + begin, e = f + min(cnt, begin + (1u << units_of.unit_shift));
        const Axes ax = cand_axes(c, nz);
        float lo[3] = {kInf, kInf, kInf}, hi[3] = {-kInf, -kInf, -kInf};
        for (uint32_t k0 = b / 32; 32 * k0 < e; k0 += 32) {
            const uint32_t k = k0 + lane;
            bool beyond = 32 * k < e;
            if (beyond) {
                float blo[3], bhi[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    blo[d] = __ldg(boxes + static_cast<size_t>(d) * nblocks + k);
                    bhi[d] = __ldg(boxes + static_cast<size_t>(3 + d) * nblocks + k);
                }
                beyond = may_extend(blo, bhi, c);
            }
            for (uint32_t some = __ballot_sync(0xffffffffu, beyond); some; some &= some - 1) {
                const uint32_t i = 32 * (k0 + __ffs(static_cast<int>(some)) - 1) + lane;
                if (i >= b && i < e) project_tri(tris + 9 * static_cast<size_t>(i), ax, lo, hi);
            }
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = warp_min(lo[k]);
            hi[k] = warp_max(hi[k]);
        }
        if (lane < 6) {
            uint32_t* k = keys + 6 * static_cast<size_t>(a) + lane;
            const float v = lane == 0 ? lo[0] : lane == 1 ? lo[1] : lane == 2 ? lo[2] : lane == 3 ? hi[0]
                          : lane == 4 ? hi[1] : hi[2];
            if (cnt <= (1u << units_of.unit_shift)) {  // the whole node in this unit
                const float o = lane == 0 ? c.olo[0] : lane == 1 ? c.olo[1] : lane == 2 ? c.olo[2]
                              : lane == 3 ? c.ohi[0] : lane == 4 ? c.ohi[1] : c.ohi[2];
                *k = f2key(lane < 3 ? fminf(o, v) : fmaxf(o, v));
            } else if (lane < 3) {
                atomicMin(k, f2key(v));
            } else {
                atomicMax(k, f2key(v));
            }
        }
    }
}

// One tile of kTile consecutive leaves: their triangles are staged in shared
// memory once, then every node of more than kOwnLeaves leaves over them is
// served from there as an item: 8 lanes or a warp each compute the extents,
// and the boxes are built afterwards, a thread per item (building them in the
// warp's first lane, 16 of 32 lanes were busy over the kernel).  Nodes crossing the tile's edges (the two chains) are
// warp items over their part in the tile, combined in the keys with integer
// atomics.  Groups and warps take items from shared counters; an item beyond
// the lists' capacity is done by the thread that found it.
//
// A node starts from the extents of its 14 summary points, which are close to
// the final ones, so most of a large node's leaves cannot change them: a warp
// item tests the boxes of its blocks of 32 leaves, a lane each, and projects
// those that could (may_extend; about 3.4 of 8 in a random mesh, fewer the
// larger the node).  What bounds the kernel is issue and the latency of the
// candidates' records.  2,000,000 triangles, with the smallest nodes here too: 298 us with every block projected and each part fenced by its
// warp, 283 with the test, 274 with the parts' atomics and fences a lane each
// at the end (a build 1,482 -> 1,456 us).
// A node over several tiles finishes in the last of them: each tile's part
// folds its extents into the node's keys (atomics), fences them, and counts
// itself in arrivals[a]; the part that completes the count reads the keys and
// writes the box.
__device__ __forceinline__ bool last_part(const uint32_t* counts, const uint32_t* first, uint32_t* arrivals,
                                          uint32_t a, uint32_t shift) {
    const uint32_t f = __ldg(first + a), cnt = __ldg(counts + a);
    const uint32_t parts = ((f + cnt - 1) >> shift) - (f >> shift) + 1;
    if (atomicAdd(arrivals + a, 1u) + 1u != parts) return false;
    __threadfence();
    return true;
}
__device__ __forceinline__ void finalize_keys(const Cand* cand, const uint32_t* keys, uint32_t a, kr_obb3* obbs,
                                              kr_mat4* xfs) {
    const uint32_t* k = keys + 6 * static_cast<size_t>(a);
    finalize_node(load_cand(cand, a), mk3(key2f(__ldcg(k)), key2f(__ldcg(k + 1)), key2f(__ldcg(k + 2))),
                  mk3(key2f(__ldcg(k + 3)), key2f(__ldcg(k + 4)), key2f(__ldcg(k + 5))), obbs + a, xfs + a);
}

constexpr uint32_t kPart = 0x80000000u;   // item over part of its node

template <uint32_t kTileItems>
struct TileItems {
    uint32_t node[kTileItems];
    uint16_t b[kTileItems], e[kTileItems];
    float ext[kTileItems][6];
};

template <uint32_t kTileShift>
__global__ void __launch_bounds__(kThreads) extents_tile_kernel(const Cand* cand, const uint32_t* counts,
                                                                const uint32_t* first, const float* tris, uint32_t n,
                                                                const uint32_t* chains, const uint32_t* chain_counts,
                                                                uint32_t* keys, uint32_t* arrivals, kr_obb3* obbs,
                                                                kr_mat4* xfs, const uint32_t* err, float nz) {
    constexpr uint32_t kTile = 1u << kTileShift, kTileGroups = tile_groups(kTileShift), kTileItems = tile_items(kTileShift);
    __shared__ __align__(16) float tri[kTile * 9];
    // group items from the front, warp items from the back
    __shared__ TileItems<kTileItems> items;
    __shared__ float box[6][kTile / 32];  // of each 32 leaves
    __shared__ uint32_t ngroup, nwarp, next_group, next_warp;
    if (*err) return;
    const uint32_t t = threadIdx.x, lane = t & 31;
    const uint32_t t0 = blockIdx.x << kTileShift;
    const uint32_t tn = min(kTile, n - t0);
    const uint32_t internal = n - 1;
    {
        // 9 * t0 floats = t0 * 36 bytes from a 16-byte aligned base: aligned
        const float4* src = reinterpret_cast<const float4*>(tris + 9 * static_cast<size_t>(t0));
        float4* dst = reinterpret_cast<float4*>(tri);
        const uint32_t n4 = 9 * tn / 4;
        for (uint32_t i = t; i < n4; i += kThreads) dst[i] = __ldg(src + i);
        for (uint32_t i = 4 * n4 + t; i < 9 * tn; i += kThreads) tri[i] = __ldg(tris + 9 * static_cast<size_t>(t0) + i);
    }
    if (t == 0) ngroup = nwarp = next_group = next_warp = 0;
    __syncthreads();
    for (uint32_t k = t >> 5; 32 * k < tn; k += kThreads / 32) {
        float lo[3] = {kInf, kInf, kInf}, hi[3] = {-kInf, -kInf, -kInf};
        if (32 * k + lane < tn) {
            const float* v = tri + 9 * (32 * k + lane);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                lo[d] = min3f(v[d], v[3 + d], v[6 + d]);
                hi[d] = max3f(v[d], v[3 + d], v[6 + d]);
            }
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const float l = warp_min(lo[d]), h = warp_max(hi[d]);
            if (lane == 0) {
                box[d][k] = l;
                box[3 + d][k] = h;
            }
        }
    }
    const auto alone = [&](uint32_t a, uint32_t b, uint32_t e, bool part) {
        const Cand c = load_cand(cand, a);
        const Axes ax = cand_axes(c, nz);
        float lo[3] = {kInf, kInf, kInf}, hi[3] = {-kInf, -kInf, -kInf};
        for (uint32_t i = b; i < e; ++i) project_tri_s(tri + 9 * i, ax, lo, hi);
        if (part) {
            uint32_t* kk = keys + 6 * static_cast<size_t>(a);
            for (int k = 0; k < 3; ++k) {
                atomicMin(kk + k, f2key(lo[k]));
                atomicMax(kk + 3 + k, f2key(hi[k]));
            }
            __threadfence();
            if (last_part(counts, first, arrivals, a, kTileShift)) finalize_keys(cand, keys, a, obbs, xfs);
        } else {
            finalize_node(c, mk3(fminf(c.olo[0], lo[0]), fminf(c.olo[1], lo[1]), fminf(c.olo[2], lo[2])),
                          mk3(fmaxf(c.ohi[0], hi[0]), fmaxf(c.ohi[1], hi[1]), fmaxf(c.ohi[2], hi[2])), obbs + a,
                          xfs + a);
        }
    };
    const auto add_item = [&](uint32_t a, uint32_t b, uint32_t e, bool part) -> bool {
        const bool group = !part && e - b <= kGroupLeaves;
        const uint32_t k = atomicAdd(group ? &ngroup : &nwarp, 1u);
        if (k >= (group ? kTileGroups : kTileItems - kTileGroups)) return false;  // list full
        const uint32_t at = group ? k : kTileItems - 1 - k;
        items.node[at] = a | (part ? kPart : 0u);
        items.b[at] = static_cast<uint16_t>(b);
        items.e[at] = static_cast<uint16_t>(e);
        return true;
    };
    // the nodes inside the tile (their indices lie in the tile too), then the
    // nodes over its edges
    const uint32_t qn = t0 < internal ? min(tn, internal - t0) : 0u;
    const uint32_t w0 = 2 * blockIdx.x;
    const uint32_t c0 = min(chain_counts[w0], kChain), c1 = min(chain_counts[w0 + 1], kChain);
    for (uint32_t i = t; i < qn + c0 + c1; i += kThreads) {
        const bool part = i >= qn;
        const uint32_t a = !part ? t0 + i
                                 : chains[i < qn + c0 ? static_cast<size_t>(w0) * kChain + (i - qn)
                                                      : static_cast<size_t>(w0 + 1) * kChain + (i - qn - c0)];
        const uint32_t f = __ldg(first + a), cnt = __ldg(counts + a);
        if (cnt <= kOwnLeaves || (!part && (f < t0 || f + cnt > t0 + tn))) continue;
        const uint32_t b = max(f, t0) - t0, e = min(f + cnt, t0 + tn) - t0;
        if (!add_item(a, b, e, part)) alone(a, b, e, part);
    }
    __syncthreads();
    const uint32_t groups = min(ngroup, kTileGroups), warps = min(nwarp, kTileItems - kTileGroups);
    for (;;) {  // warp items first: they are longer
        uint32_t it = 0;
        if (lane == 0) it = atomicAdd(&next_warp, 1u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= warps) break;
        const uint32_t at = kTileItems - 1 - it;
        const uint32_t a = items.node[at] & ~kPart;
        const bool part = (items.node[at] & kPart) != 0;
        const uint32_t b = items.b[at], e = items.e[at];
        const Cand c = load_cand(cand, a);
        // the blocks of 32 leaves, a lane each, whose points could extend it
        bool beyond = 32 * lane < e && 32 * lane + 32 > b;  // e <= tn
        if (beyond) {
            const float lo[3] = {box[0][lane], box[1][lane], box[2][lane]}, hi[3] = {box[3][lane], box[4][lane], box[5][lane]};
            beyond = may_extend(lo, hi, c);
        }
        const Axes ax = cand_axes(c, nz);
        float lo[3] = {kInf, kInf, kInf}, hi[3] = {-kInf, -kInf, -kInf};
        for (uint32_t blocks = __ballot_sync(0xffffffffu, beyond); blocks; blocks &= blocks - 1) {
            const uint32_t i = 32 * (__ffs(static_cast<int>(blocks)) - 1) + lane;
            if (i >= b && i < e) project_tri_s(tri + 9 * i, ax, lo, hi);
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = warp_min(lo[k]);
            hi[k] = warp_max(hi[k]);
        }
        const float v = lane == 0 ? lo[0] : lane == 1 ? lo[1] : lane == 2 ? lo[2] : lane == 3 ? hi[0] : lane == 4 ? hi[1] : hi[2];
        if (lane < 6) items.ext[at][lane] = v;
        __syncwarp();
    }
    for (;;) {
        uint32_t it = 0;
        if (lane == 0) it = atomicAdd(&next_group, 4u);
        it = __shfl_sync(0xffffffffu, it, 0);
        if (it >= groups) break;
        it += lane >> 3;
        const bool live = it < groups;
        const uint32_t a = live ? items.node[it] : items.node[0];
        const uint32_t b = live ? items.b[it] : 0, e = live ? items.e[it] : 0;
        const Axes ax = cand_axes(load_cand(cand, a), nz);
        float lo[3], hi[3];
        group_extents<From::kShared>(tri + 9 * b, e - b, ax, lo, hi);
        const uint32_t sub = lane & 7;
        if (live && sub < 6)
            items.ext[it][sub] = sub == 0 ? lo[0] : sub == 1 ? lo[1] : sub == 2 ? lo[2] : sub == 3 ? hi[0] : sub == 4 ? hi[1] : hi[2];
    }
    __syncthreads();
    for (uint32_t i = t; i < groups + warps; i += kThreads) {
        const uint32_t at = i < groups ? i : kTileItems - 1 - (i - groups);
        const uint32_t node = items.node[at];
        const uint32_t a = node & ~kPart;
        const float* x = items.ext[at];
        if (node & kPart) {
            if (x[0] <= x[3] || x[1] <= x[4] || x[2] <= x[5]) {  // else every block was passed over
                uint32_t* kk = keys + 6 * static_cast<size_t>(a);
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    atomicMin(kk + k, f2key(x[k]));
                    atomicMax(kk + 3 + k, f2key(x[3 + k]));
                }
            }
            __threadfence();
            if (last_part(counts, first, arrivals, a, kTileShift)) finalize_keys(cand, keys, a, obbs, xfs);
        } else {
            const Cand c = load_cand(cand, a);
            finalize_node(c, mk3(fminf(c.olo[0], x[0]), fminf(c.olo[1], x[1]), fminf(c.olo[2], x[2])),
                          mk3(fmaxf(c.ohi[0], x[3]), fmaxf(c.ohi[1], x[4]), fmaxf(c.ohi[2], x[5])), obbs + a, xfs + a);
        }
    }
}

// Nodes handled in warp units: the box from the extents in the keys (one unit:
// written by it; several: the atomic min/max over the units).
__global__ void __launch_bounds__(kThreads) finalize_multi_kernel(const Cand* cand, const uint32_t* plan,
                                                                  const uint32_t* group_count,
                                                                  const unsigned long long* unit_count, uint32_t unit_bits,
                                                                  const uint32_t* keys, uint32_t internal,
                                                                  kr_obb3* obbs, kr_mat4* xfs, const uint32_t* err) {
    if (*err) return;
    const uint32_t listed = static_cast<uint32_t>(min(*unit_count >> unit_bits, static_cast<unsigned long long>(internal)));
    const uint32_t all = min(listed + min(*group_count, internal), internal);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < all; i += gridDim.x * blockDim.x)
        finalize_keys(cand, keys, i < listed ? plan[i] : plan[internal - 1 - (i - listed)], obbs, xfs);
}

// ---------------------------------------------------------------------------
// Host side.
size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

Layout layout(uint32_t n) {
    const size_t ni = n > 1 ? n - 1 : 1;
    Layout L;
    size_t o = 0;
    L.ctl = o;      o += align256(sizeof(Ctl));
    L.visits = o;   o += align256(4 * ni);
    L.counts = o;   o += align256(4 * ni);
    L.summary = o;  o += align256(112 * ni);
    L.first = o;    o += align256(4 * ni);
    L.tris = o;     o += align256(36ull * (n > 0 ? n : 1));
    L.rank_prims = o; o += align256(4ull * (n > 0 ? n : 1));
    L.cand = o;     o += align256(sizeof(Cand) * ni);
    L.plan = o;     o += align256(4 * ni);
    L.plan_start = o; o += align256(8 * ni);
    L.keys = o;     o += align256(24 * ni);
    L.total = o;
    return L;
}

kr_error enqueue(const kr_bvh_node* nodes, const uint32_t* parents, const kr_vec3* verts, const kr_uvec4* faces,
                 kr_obb3* obbs, kr_mat4* xfs, uint32_t n, uint32_t internal, void* workspace, cudaStream_t s) {
    if (n == 0) return kr_success;
    if (!nodes || !parents || !verts || !faces || !obbs || !xfs || !workspace)
        return "kr_cuda_bvh_obb_tree: null pointer argument";
    if (internal + 1 != n) return "kr_cuda_bvh_obb_tree: a binary BVH has internal_count == primitive_count - 1";
    if (reinterpret_cast<uintptr_t>(workspace) & 255) return "kr_cuda_bvh_obb_tree: workspace must be 256-aligned";
    char* ws = static_cast<char*>(workspace);
    const Layout L = layout(n);
    Ctl* ctl = reinterpret_cast<Ctl*>(ws + L.ctl);
    uint32_t* counts = reinterpret_cast<uint32_t*>(ws + L.counts);
    uint4* summary = reinterpret_cast<uint4*>(ws + L.summary);
    const unsigned gl = (n + kThreads - 1) / kThreads;

    if (internal > 0) OBVH_TRY_CUDA(cudaMemsetAsync(ws + L.visits, 0, 4ull * internal, s));
    {
        ProfScope prof_scope_("summary_up_kernel", s);
        summary_up_kernel<<<gl, kThreads, 0, s>>>(nodes, parents, verts, faces, n, internal, summary, counts,
                                                  reinterpret_cast<uint32_t*>(ws + L.visits), obbs, xfs, &ctl->error);
    }
    OBVH_TRY_CUDA(cudaGetLastError());
    return enqueue_ranks_frames(nodes, parents, counts, verts, faces, obbs, xfs, n, workspace, s);
}

kr_error enqueue_ranks_frames(const kr_bvh_node* nodes, const uint32_t* parents, const uint32_t* counts,
                              const kr_vec3* verts, const kr_uvec4* faces, kr_obb3* obbs, kr_mat4* xfs, uint32_t n,
                              void* workspace, cudaStream_t s) {
    const uint32_t internal = n - 1;
    if (n < 2) return kr_success;
    char* ws = static_cast<char*>(workspace);
    const Layout L = layout(n);
    Ctl* ctl = reinterpret_cast<Ctl*>(ws + L.ctl);
    uint4* summary = reinterpret_cast<uint4*>(ws + L.summary);
    uint32_t* first = reinterpret_cast<uint32_t*>(ws + L.first);
    float* tris = reinterpret_cast<float*>(ws + L.tris);
    Cand* cand = reinterpret_cast<Cand*>(ws + L.cand);
    uint32_t* keys = reinterpret_cast<uint32_t*>(ws + L.keys);
    const unsigned gl = (n + kThreads - 1) / kThreads;
    {
        ProfScope prof_scope_("dfs_rank_kernel", s);
        dfs_rank_kernel<<<gl, kThreads, 0, s>>>(nodes, parents, counts, verts, faces, n, internal, first, tris,
                                                reinterpret_cast<uint32_t*>(ws + L.rank_prims),
                                                &ctl->error);
    }
    OBVH_TRY_CUDA(cudaGetLastError());
    FrameBuffers fb;
    fb.summary = summary;
    fb.points = verts;
    fb.counts = counts;
    fb.first = first;
    fb.tris = tris;
    fb.cand = cand;
    fb.plan = reinterpret_cast<uint32_t*>(ws + L.plan);
    fb.plan_start = reinterpret_cast<unsigned long long*>(ws + L.plan_start);
    fb.keys = keys;
    fb.err = &ctl->error;
    fb.groups = &ctl->groups;
    fb.units = &ctl->units;
    // the walk's counters are no longer needed (24 bytes per 32 leaves)
    fb.boxes = reinterpret_cast<float*>(ws + L.visits);
    return enqueue_frames(fb, internal, obbs, xfs, s);
}

const uint32_t* dfs_first(const void* workspace, uint32_t n) {
    return reinterpret_cast<const uint32_t*>(static_cast<const char*>(workspace) + layout(n).first);
}
const uint32_t* dfs_prims(const void* workspace, uint32_t n) {
    return reinterpret_cast<const uint32_t*>(static_cast<const char*>(workspace) + layout(n).rank_prims);
}

size_t cand_bytes(uint32_t internal) { return sizeof(Cand) * (internal > 0 ? internal : 1); }
// (the most tiles of any count up to n: a workspace for n serves fewer)
static size_t most_tiles(uint32_t n) {
    const uint32_t few = n < kSmallTiles ? (n > 0 ? n : 1) : kSmallTiles;
    return tiles_of(n) > tiles_of(few) ? tiles_of(n) : tiles_of(few);
}
size_t chain_bytes(uint32_t n) { return 2ull * kChain * 4 * most_tiles(n); }
size_t chain_count_bytes(uint32_t n) { return 2ull * 4 * most_tiles(n); }

namespace {
ChainArgs chain_args(const FrameBuffers& b, uint32_t internal, FrameNodes which, uint32_t block_shift, kr_obb3* obbs,
                     kr_mat4* xfs) {
    const uint32_t n = internal + 1;
    const bool tiled = b.chains != nullptr;
    const uint32_t ntiles = tiles_of(n);
    // the chain walks, or the leaves' boxes, ride along with the first (or only) candidate launch
    const uint32_t walkers = which == FrameNodes::kAcross ? 0u : tiled ? 2 * ntiles : n;
    return ChainArgs{tiled ? b.parents : nullptr, b.first, n,
                     static_cast<uint32_t>((static_cast<uint64_t>(walkers) + kCandThreads - 1) / kCandThreads),
                     b.chains, b.chain_counts, b.err, b.arrivals, -0.0f,
                     static_cast<uint32_t>(which), block_shift, tile_shift(n), b.tris, b.boxes, obbs, xfs, b.plan, b.plan_start,
                     unit_plan(n), b.groups,
                     b.units, b.across_list, b.across_count};
}
}  // namespace

namespace {
kr_error launch_candidates(const FrameBuffers& b, uint32_t internal, FrameNodes which, uint32_t block_shift,
                           kr_obb3* obbs, kr_mat4* xfs, cudaStream_t s) {
    if (internal == 0) return kr_success;
    const bool tiled = b.chains != nullptr;
    if (tiled && !b.parents) return "enqueue_frames: tiled extents need the parents";
    if (which != FrameNodes::kAll && (!tiled || block_shift > 31))
        return "enqueue_candidates: node classes need the tiled path and a block shift below 32";
    if (which == FrameNodes::kAcross && (!b.across_list || !b.across_count))
        return "enqueue_candidates: the nodes across blocks come as a list";
    const ChainArgs chain = chain_args(b, internal, which, block_shift, obbs, xfs);
    // kAcross loops over its list: the CTAs that fit the SMs
    const unsigned gi = which == FrameNodes::kAcross ? static_cast<unsigned>(kCandCtas * device_info().sm_count)
                                                     : (internal + kCandThreads - 1) / kCandThreads;
    // the leading CTAs' work overlaps the candidate search
    ProfScope prof_scope_("candidate_kernel", s);
    const auto kernel = !tiled ? candidate_kernel<Nodes::kPlanned>
                        : which == FrameNodes::kAcross ? candidate_kernel<Nodes::kListed>
                                                       : candidate_kernel<Nodes::kTiled>;
    kernel<<<gi + chain.walker_blocks, kCandThreads, 0, s>>>(b.summary, b.points, b.counts, internal,
                                                             static_cast<Cand*>(b.cand), b.keys, b.err, chain);
    OBVH_TRY_CUDA(cudaGetLastError());
    return kr_success;
}
}  // namespace

kr_error enqueue_candidates(const FrameBuffers& b, uint32_t internal, FrameNodes which, uint32_t block_shift,
                            kr_obb3* obbs, kr_mat4* xfs, cudaStream_t s) {
    if (internal > 0 && !b.chains) return "enqueue_candidates: the tiled path only";
    return launch_candidates(b, internal, which, block_shift, obbs, xfs, s);
}

kr_error enqueue_frames(const FrameBuffers& b, uint32_t internal, kr_obb3* obbs, kr_mat4* xfs, cudaStream_t s) {
    OBVH_TRY(launch_candidates(b, internal, FrameNodes::kAll, 0, obbs, xfs, s));
    return enqueue_extents(b, internal, obbs, xfs, s);
}

kr_error enqueue_extents(const FrameBuffers& b, uint32_t internal, kr_obb3* obbs, kr_mat4* xfs, cudaStream_t s) {
    if (internal == 0) return kr_success;
    const unsigned gi = (internal + kThreads - 1) / kThreads;
    Cand* cand = static_cast<Cand*>(b.cand);
    const uint32_t n = internal + 1;
    const bool tiled = b.chains != nullptr;
    if (tiled) {
        {
            ProfScope prof_scope_("extents_tile_kernel", s);
            const auto kernel = tile_shift(n) == kTileShiftSmall ? extents_tile_kernel<kTileShiftSmall>
                                                                 : extents_tile_kernel<kTileShiftLarge>;
            kernel<<<tiles_of(n), kThreads, 0, s>>>(cand, b.counts, b.first, b.tris, n, b.chains, b.chain_counts,
                                                    b.keys, b.arrivals, obbs, xfs, b.err, -0.0f);
        }
        OBVH_TRY_CUDA(cudaGetLastError());
        return kr_success;
    }
    const int grid = 4 * device_info().sm_count;
    {
        ProfScope prof_scope_("extents_units_kernel", s);
        extents_units_kernel<<<grid, kThreads, 0, s>>>(cand, b.counts, b.first, b.tris, b.plan, b.plan_start,
                                                       unit_plan(n), internal, b.err, b.groups, b.units, b.keys,
                                                       b.boxes, -0.0f);
    }
    OBVH_TRY_CUDA(cudaGetLastError());
    {
        ProfScope prof_scope_("finalize_multi_kernel", s);
        finalize_multi_kernel<<<std::min(gi, 2u * static_cast<unsigned>(grid)), kThreads, 0, s>>>(
            cand, b.plan, b.groups, b.units, unit_plan(n).unit_bits, b.keys, internal, obbs, xfs, b.err);
    }
    OBVH_TRY_CUDA(cudaGetLastError());
    return kr_success;
}

uint32_t* error_word(void* workspace) { return &reinterpret_cast<Ctl*>(workspace)->error; }

struct SyncContext {
    std::mutex mutex;
    DeviceBuffer ws;
    uint32_t prims = 0;
};

SyncContext& sync_context() {
    static std::mutex m;
    static std::unordered_map<int, SyncContext*> ctxs;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(m);
    SyncContext*& c = ctxs[dev];
    if (!c) c = new SyncContext();
    return *c;
}

kr_error run_sync(const kr_bvh_node* nodes, const uint32_t* parents, const kr_vec3* verts, const kr_uvec4* faces,
                  kr_obb3* obbs, kr_mat4* xfs, uint32_t n, uint32_t internal) {
    SyncContext& c = sync_context();
    std::lock_guard<std::mutex> lock(c.mutex);
    const size_t need = layout(n).total;
    OBVH_TRY(c.ws.reserve(need));
    OBVH_TRY_CUDA(cudaMemsetAsync(c.ws.ptr, 0, sizeof(Ctl), nullptr));
    OBVH_TRY(enqueue(nodes, parents, verts, faces, obbs, xfs, n, internal, c.ws.ptr, nullptr));
    uint32_t err = 0;
    OBVH_TRY_CUDA(cudaMemcpyAsync(&err, error_word(c.ws.ptr), sizeof err, cudaMemcpyDeviceToHost, nullptr));
    OBVH_TRY_CUDA(cudaStreamSynchronize(nullptr));
    if (err & kErrCycle) return "kr_cuda_bvh_obb_tree: parent walk longer than the tree (cycle?)";
    if (err) return "kr_cuda_bvh_obb_tree: malformed tree";
    return kr_success;
}

}  // namespace obbtree
}  // namespace obvh

using namespace obvh;

extern "C" kr_error kr_cuda_bvh_obb_tree(kr_bvh_node* nodes, const kr_u32* parents, const kr_u32* primitive_counts,
                                         const kr_scalar* costs, const kr_vec3* vertices, const kr_uvec4* faces,
                                         const kr_u32* primitives, kr_obb3* obbs, kr_mat4* transforms, kr_scalar ci,
                                         kr_scalar ct, kr_scalar obb_cost, kr_u32 primitive_count,
                                         kr_u32 internal_count, kr_u32 primitive_threshold) {
    // primitive_counts, costs, primitives, ci, ct, obb_cost and
    // primitive_threshold are accepted and unused, as in the reference.
    (void)primitive_counts; (void)costs; (void)primitives; (void)ci; (void)ct; (void)obb_cost;
    (void)primitive_threshold;
    kr_error e = obbtree::run_sync(nodes, parents, vertices, faces, obbs, transforms, primitive_count, internal_count);
    if (e) set_last_error(e);
    return e;
}

extern "C" kr_size obvh_obb_tree_workspace_bytes(kr_u32 primitive_count) {
    return obbtree::layout(primitive_count).total;
}

extern "C" kr_error obvh_bvh_obb_tree_async(const kr_bvh_node* d_nodes, const kr_u32* d_parents,
                                            const kr_vec3* d_vertices, const kr_uvec4* d_faces, kr_obb3* d_obbs,
                                            kr_mat4* d_transforms, kr_u32 primitive_count, kr_u32 internal_count,
                                            void* d_workspace, void* stream) {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    kr_error e = kr_success;
    if (d_workspace) {
        cudaError_t ce = cudaMemsetAsync(d_workspace, 0, sizeof(obbtree::Ctl), s);
        if (ce != cudaSuccess) e = cuda_error(ce);
    }
    if (!e)
        e = obbtree::enqueue(d_nodes, d_parents, d_vertices, d_faces, d_obbs, d_transforms, primitive_count,
                             internal_count, d_workspace, s);
    if (e) set_last_error(e);
    return e;
}

extern "C" kr_error obvh_obb_tree_error(const void* d_workspace, void* stream, kr_u32* device_error) {
    if (!d_workspace || !device_error) return "obvh_obb_tree_error: null pointer argument";
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    cudaError_t e = cudaMemcpyAsync(device_error, d_workspace, sizeof(kr_u32), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return e == cudaSuccess ? kr_success : cuda_error(e);
}
