// pipeline.cu - the whole commit of the reference's lbvh_gpu intersector
// (src/ads/lbvh_gpu/lbvh.cu:1646-1723: LBVH, then kr_cuda_bvh_obb_tree on the
// uncollapsed tree, then kr_cuda_bvh_collapse) as one fused chain of kernels.
//
// Results are those of the three separate steps; the fusion only removes
// work the chain would repeat:
//   - a Karras tree keeps its leaves in depth-first order, so each subtree's
//     triangles are one contiguous run of the sorted leaves and every
//     internal node's first leaf is the low end of its key range: the
//     depth-first rank pass of the stand-alone transform is not needed;
//   - the leaf pass writes the leaves, their triangles in that order and the
//     leaves' own boxes (triangle frames) in one go;
//   - one bottom-up pass (two kernels: the nodes inside each CTA's leaves,
//     from shared memory; then the few crossing CTA edges) computes the
//     bounds, the SAH costs and collapse decisions, and the 7-direction
//     subtree summaries that the reference computes in three separate
//     leaf-to-root walks (lbvh.cu:399-457, transforms.cu:287-411,
//     transforms.cu:65-136); primitive counts are the key-range sizes;
//   - a collapse root's primitive list (right child first, transforms.cu:18-63)
//     is its leaf range read backwards, so no tree walk is needed to gather it.
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "device_common.cuh"
#include "lbvh_device.cuh"
#include "lbvh_host.h"
#include "obb_tree_host.h"
#include "obvh_build.h"
#include "pipeline_host.h"
#include "runtime.h"
#include "sort.h"
#include "tree_device.cuh"
#include "up_device.cuh"

namespace obvh {
namespace pipeline {

using namespace tree;

constexpr int kThreads = 256;
constexpr uint32_t kLocalShift = 8;  // fused_up_local covers 2^kLocalShift = kThreads leaves per CTA
static_assert((1 << kLocalShift) == kThreads, "CTA leaf blocks are aligned powers of two");

struct Ctl {
    uint32_t error;
    uint32_t spare0;
    uint32_t total_slots;
    uint32_t spare;
    uint32_t across;    // nodes the cross-CTA pass completed (listed at Layout::across)
    uint32_t pad[59];
};

// Writes `words` staged words to dst with coalesced stores: 4-byte stores up
// to the first 16-byte boundary, 16-byte stores after it.  src (shared) and
// dst (global) have the same address modulo 16.
__device__ __forceinline__ void copy_out(uint32_t* dst, const uint32_t* src, uint32_t words) {
    const uint32_t lead = min(words, static_cast<uint32_t>(((16 - (reinterpret_cast<uintptr_t>(dst) & 15)) & 15) / 4));
    for (uint32_t t = threadIdx.x; t < lead; t += blockDim.x) dst[t] = src[t];
    const uint32_t n4 = (words - lead) / 4;
    float4* d4 = reinterpret_cast<float4*>(dst + lead);
    const float4* s4 = reinterpret_cast<const float4*>(src + lead);
    for (uint32_t t = threadIdx.x; t < n4; t += blockDim.x) d4[t] = s4[t];
    for (uint32_t t = lead + 4 * n4 + threadIdx.x; t < words; t += blockDim.x) dst[t] = src[t];
}

// The staging slot in shared memory for a record of `rw` words of this thread
// whose run of records starts at dst (same address phase modulo 16).
__device__ __forceinline__ uint32_t* stage_at(uint32_t* stage, const void* dst, uint32_t rw) {
    return stage + (reinterpret_cast<uintptr_t>(dst) & 15) / 4 + threadIdx.x * rw;
}

// Sorted leaf j: node internal + j, its triangle at slot j, its own box.  The
// CTA's leaves are consecutive, so every output is one contiguous run per CTA:
// records are staged in shared memory and written out coalesced.
//
// Odd CTAs build the Karras tree over the sorted codes instead (karras_node:
// it needs the codes alone, so the two were one launch after the other; side
// by side the tree's searches run while the leaves wait for memory).  The first
// CTA also clears the chain's control block, which nothing reads before the
// next kernel, and copies the scene and centroid boxes out.
struct TreeArgs {
    const uint32_t* codes;
    uint32_t* parents;
    uint32_t* first;
    uint32_t* counts;
    uint32_t* ctl;         // kCtlWords of them
    const float* boxes;
    float* bounds;         // nullable
};
constexpr uint32_t kCtlWords = sizeof(Ctl) / 4;

__global__ void __launch_bounds__(kThreads) leaves_fused_kernel(TreeArgs tree_args, const uint32_t* order,
                                                                const kr_vec3* verts, const uint4* faces, uint32_t n,
                                                                kr_bvh_node* nodes, kr_bvh_node* collapsed,
                                                                float* tris, kr_obb3* obbs, kr_mat4* xfs,
                                                                uint32_t* visits, uint8_t* cflags) {
    __shared__ __align__(16) uint32_t stage_a[kThreads * 15 + 4];  // node (9), triangle (9) or box (15) records
    __shared__ __align__(16) uint32_t stage_x[kThreads * 16 + 4];  // transforms
    const uint32_t j0 = (blockIdx.x >> 1) * blockDim.x;
    if (blockIdx.x & 1) {
        const uint32_t i = j0 + threadIdx.x;
        if (n >= 2 && i < n - 1)
            lbvh::karras_node(tree_args.codes, n, static_cast<int>(i), nodes, tree_args.parents, tree_args.first,
                              tree_args.counts);
        else if (n == 1 && i == 0)
            tree_args.parents[0] = kNoParent;
        return;
    }
    if (blockIdx.x == 0) {
        for (uint32_t k = threadIdx.x; k < kCtlWords; k += kThreads) tree_args.ctl[k] = 0u;
        if (tree_args.bounds && threadIdx.x < 12) tree_args.bounds[threadIdx.x] = tree_args.boxes[threadIdx.x];
    }
    const uint32_t j = j0 + threadIdx.x;
    const uint32_t count = min(static_cast<uint32_t>(blockDim.x), n - j0);
    const bool live = j < n;
    const uint32_t internal = n - 1;
    // the bottom-up pass's arrival counters (internal entries) and collapse
    // marks (2n - 1 bytes) start at zero; nothing reads them before it
    if (j < internal) visits[j] = 0u;
    if (cflags) {
        if (2 * j < 2 * n - 1) cflags[2 * j] = 0;
        if (2 * j + 1 < 2 * n - 1) cflags[2 * j + 1] = 0;
    }
    uint32_t w[9];
    f3 v0 = mk3(0, 0, 0), v1 = v0, v2 = v0;
    if (live) {
        const uint32_t i = order[j];
        const uint4 f = __ldg(faces + i);
        v0 = load_vertex(verts, f.x);
        v1 = load_vertex(verts, f.y);
        v2 = load_vertex(verts, f.z);
        // the triangle's box, as tri_bounds_kernel computed it (lbvh::tri_box:
        // exact min/max, so recomputing it from the vertices read here gives
        // the same bits as reading it back)
        const f3 lo = vmin3(vmin3(v0, v1), v2), hi = vmax3(vmax3(v0, v1), v2);
        w[0] = __float_as_uint(lo.x); w[1] = __float_as_uint(lo.y); w[2] = __float_as_uint(lo.z);
        w[3] = __float_as_uint(hi.x); w[4] = __float_as_uint(hi.y); w[5] = __float_as_uint(hi.z);
        w[6] = i;  // primitivesOffset
        w[7] = 0;
        w[8] = 1;  // one primitive, axis 0
    }
    for (int out = 0; out < 2; ++out) {
        kr_bvh_node* dst = out == 0 ? nodes : collapsed;
        if (!dst) continue;
        uint32_t* d = reinterpret_cast<uint32_t*>(dst + internal + j0);
        if (live) {
            uint32_t* st = stage_at(stage_a, d, 9);
            for (int k = 0; k < 9; ++k) st[k] = w[k];
        }
        __syncthreads();
        copy_out(d, stage_a + (reinterpret_cast<uintptr_t>(d) & 15) / 4, 9 * count);
        __syncthreads();
    }
    {
        uint32_t* d = reinterpret_cast<uint32_t*>(tris + 9 * static_cast<size_t>(j0));
        if (live) {
            float* st = reinterpret_cast<float*>(stage_at(stage_a, d, 9));
            st[0] = v0.x; st[1] = v0.y; st[2] = v0.z; st[3] = v1.x; st[4] = v1.y; st[5] = v1.z;
            st[6] = v2.x; st[7] = v2.y; st[8] = v2.z;
        }
        __syncthreads();
        copy_out(d, stage_a + (reinterpret_cast<uintptr_t>(d) & 15) / 4, 9 * count);
        __syncthreads();
    }
    if (obbs) {
        uint32_t* db = reinterpret_cast<uint32_t*>(obbs + internal + j0);
        uint32_t* dx = reinterpret_cast<uint32_t*>(xfs + internal + j0);
        if (live)
            leaf_box(v0, v1, v2, reinterpret_cast<kr_obb3*>(stage_at(stage_a, db, 15)),
                     reinterpret_cast<kr_mat4*>(stage_at(stage_x, dx, 16)));
        __syncthreads();
        copy_out(db, stage_a + (reinterpret_cast<uintptr_t>(db) & 15) / 4, 15 * count);
        copy_out(dx, stage_x + (reinterpret_cast<uintptr_t>(dx) & 15) / 4, 16 * count);
    }
}

// Shared memory of the CTA-local part of the bottom-up pass, in rows of
// kRow words (one word per node; the odd row length spreads a node's words
// over the banks).  Internal node rows: bounds (6), cost, the 14 slab values,
// then the 14 slab vertices as 16-bit offsets from 3 * j0, two per word (7).
// Leaf rows: bounds (6), the 14 slab values and which of the leaf's vertices
// they are, two bits each (1); a leaf's cost is recomputed from its bounds.
constexpr uint32_t kRow = kThreads + 1;
constexpr int kSlotRows = 28;
constexpr int kLeafRows = 21;
constexpr uint16_t kLeafKid = 0x8000u;  // child encoding: leaf j0 + q, else internal node j0 + q
constexpr uint16_t kNotLocal = 0xffffu;

struct LocalSmem {
    uint32_t islot[kSlotRows * kRow];
    uint32_t lslot[kLeafRows * kRow];
    uint32_t deg[kThreads];     // children of local node j0 + q not completed yet
    uint16_t kid[2][kThreads];  // its children
    uint16_t cnt[kThreads];     // its primitive count
    uint16_t up[kThreads];      // its parent's local index, or kNotLocal
    uint32_t queue[2][kThreads];  // nodes ready in a round (turn_of)
    uint8_t local[kThreads], iflag[kThreads], lflag[kThreads], hidden[kThreads];
    uint32_t qn[3];
    uint32_t nfront;
};
constexpr size_t kFusedSmemBytes = sizeof(LocalSmem);

__device__ __forceinline__ void put_carry(uint32_t* slots, uint32_t q, const Carry& c) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        slots[k * kRow + q] = __float_as_uint(c.lo[k]);
        slots[(3 + k) * kRow + q] = __float_as_uint(c.hi[k]);
    }
    slots[6 * kRow + q] = __float_as_uint(c.cost);
}

__device__ __forceinline__ void get_bounds(const uint32_t* slots, uint32_t q, Carry& c) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        c.lo[k] = __uint_as_float(slots[k * kRow + q]);
        c.hi[k] = __uint_as_float(slots[(3 + k) * kRow + q]);
    }
}

// Node j0 + q and its children in one word of the queue.
constexpr uint32_t kLeftLeaf = 1u << 24, kRightLeaf = 1u << 25;
__device__ __forceinline__ uint32_t turn_of(const LocalSmem& sm, uint32_t q) {
    const uint32_t l = sm.kid[0][q], r = sm.kid[1][q];
    return q | ((l & 0xffu) << 8) | ((r & 0xffu) << 16) | (l & kLeafKid ? kLeftLeaf : 0u) |
           (r & kLeafKid ? kRightLeaf : 0u);
}

// carry of internal node j0 + q / of leaf j0 + q (its cost: leaf_ct * area)
__device__ __forceinline__ Carry get_carry(const LocalSmem& sm, uint32_t q, bool leaf, float leaf_ct) {
    Carry c;
    get_bounds(leaf ? sm.lslot : sm.islot, q, c);
    c.cost = leaf ? leaf_ct * box_area(c.lo, c.hi) : __uint_as_float(sm.islot[6 * kRow + q]);
    return c;
}

// Slab k of internal node / leaf j0 + q; its vertices as offsets from 3 * j0.
__device__ __forceinline__ void put_slab(uint32_t* islot, uint32_t q, uint32_t k, const Slab& v) {
    islot[(7 + 2 * k) * kRow + q] = __float_as_uint(v.lo);
    islot[(8 + 2 * k) * kRow + q] = __float_as_uint(v.hi);
    islot[(21 + k) * kRow + q] = v.ilo | (v.ihi << 16);
}

__device__ __forceinline__ Slab get_slab(const LocalSmem& sm, uint32_t q, bool leaf, uint32_t k) {
    const uint32_t* at = (leaf ? sm.lslot + 6 * kRow : sm.islot + 7 * kRow) + 2 * k * kRow + q;
    const uint32_t ids = leaf ? sm.lslot[20 * kRow + q] >> (4 * k) : sm.islot[(21 + k) * kRow + q];
    return Slab{__uint_as_float(at[0]), __uint_as_float(at[kRow]), leaf ? 3 * q + (ids & 3u) : ids & 0xffffu,
                leaf ? 3 * q + ((ids >> 2) & 3u) : ids >> 16};
}

// Bottom-up pass, part 1 of 2: bounds, costs, collapse marks and summaries of
// every node whose leaf range lies within one CTA's leaves (the primitive
// counts of internal nodes are the key-range sizes the tree construction
// wrote).
//
// CTA b takes sorted leaves [j0, jend).  A Karras node lies at one end of its
// own leaf range, so an internal node whose range lies within these leaves
// ("local") has its index in [j0, jend) too.  The local nodes are completed
// in rounds separated by CTA barriers: a round's ready nodes sit in a queue;
// a completed node's parent joins the next round's queue once both children
// are done.  Children are read from shared memory, and the outputs are written
// at the end as contiguous runs.  The leaves and local nodes whose parents are
// not local go to a list for part 2.
//
// Bound by the length of a round, a chain of shared memory reads and compares
// that few warps run: a random mesh takes about nine rounds.  So the work on a
// node is dealt out by parts, its carry and each of its seven slabs to a warp
// of its own with up to 32 nodes side by side, and the leaves' slabs are made
// by all threads before the first round.  This kernel in a build of 2,000,000
// triangles: 323 us with a thread for a whole node (eight where few were
// ready), 274 with the parts dealt out, 255 with the children named in the
// queue and the parts turning from warp to warp.
__global__ void __launch_bounds__(kThreads, 4) fused_up_local_kernel(UpArgs a, uint32_t* frontier,
                                                                     uint32_t* frontier_counts) {
    extern __shared__ __align__(16) unsigned char fused_smem[];
    LocalSmem& sm = *reinterpret_cast<LocalSmem*>(fused_smem);
    const uint32_t t = threadIdx.x;
    const uint32_t j0 = blockIdx.x * kThreads;
    const uint32_t jend = min(j0 + kThreads, a.n);
    const uint32_t m = jend - j0;
    const uint32_t internal = a.n - 1;
    const uint32_t mi = j0 < internal ? min(jend, internal) - j0 : 0u;  // internal node indices in [j0, jend)
    const bool with_summary = a.summary != nullptr;
    // leaf cost: ct * area in the collapse (transforms.cu:97), 1 * area in the LBVH (lbvh.cu:427)
    const float leaf_ct = a.flags ? a.ct : 1.0f;
    // The CTA's triangles (or, without summaries, its leaf records) are
    // contiguous runs of 9 words each: read word by word across the CTA
    // (coalesced), every load in flight before the first store: the records'
    // bounds into the leaf rows, the triangles into rows of the internal
    // nodes, which nothing else uses before the rounds.  With the triangles at
    // hand, a leaf's bounds are recomputed from its vertices below (exact
    // min/max: the bits of its record).
    {
        const uint32_t* src = with_summary ? reinterpret_cast<const uint32_t*>(a.tris + 9 * static_cast<size_t>(j0))
                                           : reinterpret_cast<const uint32_t*>(a.nodes + internal + j0);
        uint32_t vw[9];
#pragma unroll
        for (int r = 0; r < 9; ++r) {
            const uint32_t w = t + r * kThreads;
            vw[r] = w < 9 * m ? (with_summary ? __ldg(src + w) : __ldcg(src + w)) : 0u;
        }
#pragma unroll
        for (int r = 0; r < 9; ++r) {
            const uint32_t w = t + r * kThreads;
            if (w >= 9 * m) continue;
            const uint32_t q = w / 9, k = w - 9 * q;
            if (with_summary) sm.islot[k * kRow + q] = vw[r];
            else if (k < 6) sm.lslot[k * kRow + q] = vw[r];
        }
    }
    const uint32_t leaf_parent = t < m ? a.parents[internal + j0 + t] : kNoParent;
    const uint32_t p = j0 + t;
    bool mine = false;
    bool bad = false;
    uint32_t parent = kNoParent;
    if (t < mi) {
        const uint32_t* pw = reinterpret_cast<const uint32_t*>(a.nodes + p);
        const uint32_t L = __ldg(pw + 6), R = __ldg(pw + 7);
        const uint32_t f = __ldg(a.first + p), count = __ldg(a.counts + p);
        parent = __ldg(a.parents + p);
        if (f >= j0 && f + count <= jend) {
            const bool lleaf = L >= internal, rleaf = R >= internal;
            const uint32_t lq = (lleaf ? L - internal : L) - j0, rq = (rleaf ? R - internal : R) - j0;
            if (lq < m && rq < m) {
                mine = true;
                sm.kid[0][t] = static_cast<uint16_t>(lq | (lleaf ? kLeafKid : 0u));
                sm.kid[1][t] = static_cast<uint16_t>(rq | (rleaf ? kLeafKid : 0u));
                sm.cnt[t] = static_cast<uint16_t>(count);
                sm.deg[t] = (lleaf ? 0u : 1u) + (rleaf ? 0u : 1u);
            } else {
                bad = true;  // a child outside its parent's range
            }
        }
    }
    sm.local[t] = mine;
    sm.iflag[t] = 0;
    sm.lflag[t] = 0;
    sm.hidden[t] = 0;
    if (t < 3) sm.qn[t] = 0;
    if (t == 0) sm.nfront = 0;
    __syncthreads();
    if (t < m) {
        if (with_summary) {  // the triangle's box (lbvh::tri_box) and slabs from its vertices
            f3 v[3];
#pragma unroll
            for (int i = 0; i < 3; ++i)
                v[i] = mk3(__uint_as_float(sm.islot[3 * i * kRow + t]), __uint_as_float(sm.islot[(3 * i + 1) * kRow + t]),
                           __uint_as_float(sm.islot[(3 * i + 2) * kRow + t]));
            const f3 lo = vmin3(vmin3(v[0], v[1]), v[2]), hi = vmax3(vmax3(v[0], v[1]), v[2]);
            sm.lslot[0 * kRow + t] = __float_as_uint(lo.x);
            sm.lslot[1 * kRow + t] = __float_as_uint(lo.y);
            sm.lslot[2 * kRow + t] = __float_as_uint(lo.z);
            sm.lslot[3 * kRow + t] = __float_as_uint(hi.x);
            sm.lslot[4 * kRow + t] = __float_as_uint(hi.y);
            sm.lslot[5 * kRow + t] = __float_as_uint(hi.z);
            uint32_t ids = 0;
#pragma unroll
            for (int k = 0; k < 7; ++k) {
                const Slab o = leaf_slab(v, 0, k);
                sm.lslot[(6 + 2 * k) * kRow + t] = __float_as_uint(o.lo);
                sm.lslot[(7 + 2 * k) * kRow + t] = __float_as_uint(o.hi);
                ids |= (o.ilo | (o.ihi << 2)) << (4 * k);
            }
            sm.lslot[20 * kRow + t] = ids;
        }
        Carry c;
        get_bounds(sm.lslot, t, c);
        __stcg(a.costs + internal + j0 + t, leaf_ct * box_area(c.lo, c.hi));
        __stcg(a.counts + internal + j0 + t, 1u);
    }
    const auto is_local = [&](uint32_t x) { return x != kNoParent && x - j0 < m && sm.local[x - j0]; };
    if (mine) {
        sm.up[t] = is_local(parent) ? static_cast<uint16_t>(parent - j0) : kNotLocal;
        if (sm.deg[t] == 0) sm.queue[0][atomicAdd(&sm.qn[0], 1u)] = turn_of(sm, t);
    }
    __syncthreads();
    // Rounds.  The queue's counters rotate over three slots: a round reads one,
    // appends to the next and clears the one read the round before.
    for (uint32_t r = 0;; ++r) {
        const uint32_t cur = r % 3, nxt = (r + 1) % 3, old = (r + 2) % 3;
        const uint32_t K = sm.qn[cur];
        if (K == 0) break;
        if (r > m) {  // unreachable for a well-formed tree
            bad = true;
            break;
        }
        if (t == 0) sm.qn[old] = 0;
        // Part 0 of a node is its carry (and its parent's turn), part 1 + k
        // its slab k; the warps change parts from one 32 nodes to the next,
        // since part 0 is the longest.  Without summaries there is part 0 only.
        const uint32_t step = with_summary ? 32u : static_cast<uint32_t>(kThreads);
        for (uint32_t s = t >> 5, i = t & (step - 1); i < K; ++s, i += step) {
            const uint32_t part = with_summary ? s & 7u : 0u;
            const uint32_t turn = sm.queue[r & 1][i], q = turn & 0xffu;
            const bool lleaf = turn & kLeftLeaf, rleaf = turn & kRightLeaf;
            const uint32_t lq = (turn >> 8) & 0xffu, rq = (turn >> 16) & 0xffu;
            if (part > 0) {
                put_slab(sm.islot, q, part - 1,
                         merge_slab(get_slab(sm, lq, lleaf, part - 1), get_slab(sm, rq, rleaf, part - 1)));
                continue;
            }
            const uint32_t count = sm.cnt[q];
            const Carry l = get_carry(sm, lq, lleaf, leaf_ct);
            const Carry rc = get_carry(sm, rq, rleaf, leaf_ct);
            Carry o;
#pragma unroll
            for (int k = 0; k < 3; ++k) {  // kr_aabb_expand(left, right)
                o.lo[k] = kmin(kmin(l.lo[k], rc.lo[k]), rc.hi[k]);
                o.hi[k] = kmax(kmax(l.hi[k], rc.lo[k]), rc.hi[k]);
            }
            const float area = box_area(o.lo, o.hi);
            if (a.flags) {
                // bvh_mark_collapse_kernel (transforms.cu:111-133)
                const float node_cost = a.ci * area + l.cost + rc.cost;
                const float leaf_cost = a.ct * area * static_cast<float>(count);
                if (leaf_cost < node_cost && count <= kMaxLeafSize) {
                    o.cost = leaf_cost;
                    sm.iflag[q] = 1;
                    // collapsed children: marked, and nPrimitives = 0xFFFF (axis byte and pad are zero)
                    if (lleaf) {
                        sm.lflag[lq] = 1;
                        __stcg(reinterpret_cast<uint32_t*>(a.collapsed + internal + j0 + lq) + 8, kHidden);
                    } else {
                        sm.iflag[lq] = 1;
                        sm.hidden[lq] = 1;
                    }
                    if (rleaf) {
                        sm.lflag[rq] = 1;
                        __stcg(reinterpret_cast<uint32_t*>(a.collapsed + internal + j0 + rq) + 8, kHidden);
                    } else {
                        sm.iflag[rq] = 1;
                        sm.hidden[rq] = 1;
                    }
                } else {
                    o.cost = node_cost;
                }
            } else {
                o.cost = 1.2f * area + rc.cost + l.cost;  // calculate_aabbs_kernel (lbvh.cu:452)
            }
            put_carry(sm.islot, q, o);
            const uint32_t above = sm.up[q];
            if (above != kNotLocal && atomicSub(&sm.deg[above], 1u) == 1u)
                sm.queue[(r + 1) & 1][atomicAdd(&sm.qn[nxt], 1u)] = turn_of(sm, above);
        }
        __syncthreads();
    }
    if (bad) atomicOr(a.err, kErrBadInput);
    // Outputs of the local nodes, as contiguous runs over [j0, j0 + mi).
    {
        uint32_t* nw = reinterpret_cast<uint32_t*>(a.nodes + j0);
        uint32_t* cw = a.collapsed ? reinterpret_cast<uint32_t*>(a.collapsed + j0) : nullptr;
        for (uint32_t w = t; w < 9 * mi; w += kThreads) {
            const uint32_t q = w / 9, k = w - 9 * q;
            if (!sm.local[q]) continue;
            uint32_t v;
            if (k < 6) {
                v = sm.islot[k * kRow + q];
                __stcg(nw + w, v);  // words 6..8 hold the children and 0 already
            } else if (k < 8) {
                const uint32_t kd = sm.kid[k - 6][q];
                v = (kd & kLeafKid) ? internal + j0 + (kd & 0xffu) : j0 + kd;
            } else {
                v = sm.hidden[q] ? kHidden : 0u;
            }
            if (cw) __stcg(cw + w, v);
        }
        for (uint32_t q = t; q < mi; q += kThreads)
            if (sm.local[q]) __stcg(a.costs + j0 + q, __uint_as_float(sm.islot[6 * kRow + q]));
        if (with_summary) {
            uint4* sw = a.summary + 7 * static_cast<size_t>(j0);
            for (uint32_t w = t; w < 7 * mi; w += kThreads) {
                const uint32_t q = w / 7, k = w - 7 * q;
                if (sm.local[q]) {
                    const uint32_t ids = sm.islot[(21 + k) * kRow + q];
                    __stcg(sw + w, make_uint4(sm.islot[(7 + 2 * k) * kRow + q], sm.islot[(8 + 2 * k) * kRow + q],
                                              3 * j0 + (ids & 0xffffu), 3 * j0 + (ids >> 16)));
                }
            }
        }
        if (a.flags) {
            for (uint32_t q = t; q < mi; q += kThreads)
                if (sm.local[q]) a.flags[j0 + q] = sm.iflag[q];
            for (uint32_t q = t; q < m; q += kThreads) a.flags[internal + j0 + q] = sm.lflag[q];
        }
    }
    // Walks for part 2: this thread's leaf and its local node, where their
    // parents are not local.
    const bool leaf_walk = !bad && t < m && leaf_parent != kNoParent && !is_local(leaf_parent);
    const bool node_walk = !bad && mine && parent != kNoParent && sm.up[t] == kNotLocal;
    const uint32_t nf = static_cast<uint32_t>(leaf_walk) + static_cast<uint32_t>(node_walk);
    const uint32_t at = nf ? atomicAdd(&sm.nfront, nf) : 0u;
    if (nf && at + nf <= kThreads) {  // the roots of a forest over the CTA's leaves: at most kThreads
        uint32_t* list = frontier + blockIdx.x * kThreads;
        if (leaf_walk) list[at] = internal + j0 + t;
        if (node_walk) list[at + (leaf_walk ? 1 : 0)] = p;
    } else if (nf) {
        atomicOr(a.err, kErrBadInput);
    }
    __syncthreads();
    if (t == 0) frontier_counts[blockIdx.x] = min(sm.nfront, static_cast<uint32_t>(kThreads));
}

// Bottom-up pass, part 2 of 2: the walks from the listed nodes complete the
// nodes whose leaf ranges cross a CTA's edge.  Part 1 has finished, so a
// listed node's outputs are in memory.
//
// The walk is a chain of levels whose cost is their ordering, so CTA b takes
// the lists of the part-1 CTAs over 2^kSuperShift consecutive leaves: a node
// whose leaves lie inside them has both arrivals from this CTA, and a byte in
// shared memory between CTA-scope fences counts them; only the nodes above pay
// the GPU-scope release, atomic and acquire.  A walk belongs to 8 lanes: 7
// merge a slab of the summary each, the last one completes the node (a thread
// to a walk ran some 600 instructions a level, lanes diverging).  A group
// whose walk ends takes the next one.  More leaves a CTA mean fewer levels
// above but more walks to a CTA; us a build with a thread to a walk and global
// arrivals / 2^10 / 2^11 / 2^12 leaves: 1,021 triangles 129 / 114 / 114 / 114,
// 57,344 236 / 208 / 214 / 213, 200,003 336 / 307 / 316 / 317, 500,003 466 /
// 467 / 467 / 469, 2,000,000 1,551 / 1,558 / 1,551 / 1,535.
constexpr uint32_t kSuperShiftSmall = 10, kSuperShiftLarge = 12;
constexpr uint32_t kSuperLarge = 1u << 20;

template <uint32_t kSuperShift>
struct SuperArrive {
    uint32_t* bytes;  // one per node index of the superblock (a node's index lies in its leaf range)
    __device__ __forceinline__ uint32_t operator()(const UpArgs& a, uint32_t p) const {
        const uint32_t f = __ldg(a.first + p), l = f + __ldg(a.counts + p) - 1;
        if ((f >> kSuperShift) != (l >> kSuperShift)) return arrive(a.visits + p);
        const uint32_t q = p & ((1u << kSuperShift) - 1), shift = 8u * (q & 3u);
        __threadfence_block();  // release: this thread's outputs before its arrival
        const uint32_t old = atomicAdd(bytes + (q >> 2), 1u << shift);  // a byte counts at most 2: no carry
        __threadfence_block();  // acquire: the sibling's outputs after it
        return (old >> shift) & 0xffu;
    }
};

template <uint32_t kSuperShift>
__global__ void __launch_bounds__(kThreads) fused_up_cross_kernel(UpArgs a, const uint32_t* frontier,
                                                                  const uint32_t* frontier_counts, uint32_t blocks) {
    constexpr uint32_t kSuperBlocks = 1u << (kSuperShift - kLocalShift);
    __shared__ uint32_t bytes[(1u << kSuperShift) / 4];
    __shared__ uint32_t start[kSuperBlocks + 1], next;
    const uint32_t t = threadIdx.x, b0 = blockIdx.x * kSuperBlocks;
    const uint32_t internal = a.n - 1;
    for (uint32_t i = t; i < (1u << kSuperShift) / 4; i += kThreads) bytes[i] = 0;
    if (t < 32) {  // where each list starts among this CTA's walks
        uint32_t run = 0;
        for (uint32_t q0 = 0; q0 < kSuperBlocks; q0 += 32) {
            const uint32_t q = q0 + t;
            const uint32_t c = q < kSuperBlocks && b0 + q < blocks ? frontier_counts[b0 + q] : 0u;
            uint32_t incl = c;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
                if (static_cast<int>(t) >= d) incl += v;
            }
            if (q < kSuperBlocks) start[q] = run + incl - c;
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (t == 0) {
            start[kSuperBlocks] = run;
            next = 0;
        }
    }
    __syncthreads();
    const uint32_t lane = t & 7;  // of the walk's group
    const uint32_t total = start[kSuperBlocks];
    const SuperArrive<kSuperShift> arrive_at{bytes};
    const kr_vec3* pts = reinterpret_cast<const kr_vec3*>(a.tris);
    const bool slabs = a.summary != nullptr && lane < 7;
    // slab `lane` of node x's summary; what was read may come from this kernel
    const auto read_slab = [&](uint32_t x) -> Slab {
        if (x >= internal) {
            const f3 v[3] = {load_vertex(pts, 3 * (x - internal)), load_vertex(pts, 3 * (x - internal) + 1),
                             load_vertex(pts, 3 * (x - internal) + 2)};
            return leaf_slab(v, x - internal, static_cast<int>(lane));
        }
        const uint4 q = __ldcg(a.summary + 7 * static_cast<size_t>(x) + lane);
        return Slab{__uint_as_float(q.x), __uint_as_float(q.y), q.z, q.w};
    };
    const auto read_carry = [&](uint32_t x) {
        Carry c;
        const uint32_t* w = reinterpret_cast<const uint32_t*>(a.nodes + x);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            c.lo[k] = __uint_as_float(__ldcg(w + k));
            c.hi[k] = __uint_as_float(__ldcg(w + 3 + k));
        }
        c.cost = __ldcg(a.costs + x);
        return c;
    };
    bool live = false, dry = false;
    uint32_t child = 0, p = kNoParent, steps = 0;
    Slab own{0.f, 0.f, 0u, 0u};
    Carry c{{0.f, 0.f, 0.f}, {0.f, 0.f, 0.f}, 0.f};
    for (;;) {
        // a group whose walk has ended takes the next one
        uint32_t i = total;
        if (!live && !dry && lane == 0) i = atomicAdd(&next, 1u);
        i = __shfl_sync(0xffffffffu, i, 0, 8);
        if (!live && !dry) {
            dry = i >= total;
            if (!dry) {
                uint32_t q = 0;  // the last list that starts at or before walk i
                for (uint32_t step = kSuperBlocks / 2; step > 0; step >>= 1)
                    if (start[q + step] <= i) q += step;
                child = frontier[(b0 + q) * kThreads + (i - start[q])];
                p = a.parents[child];
                steps = 0;
                live = true;
                if (slabs) own = read_slab(child);
                if (lane == 7) c = read_carry(child);
            }
        }
        if (!__any_sync(0xffffffffu, live)) break;
        if (live && (++steps > internal || p >= internal)) {
            if (lane == 0 && p != kNoParent) atomicOr(a.err, kErrCycle);
            live = false;
        }
        uint32_t L = 0, R = 0, grand = kNoParent, count = 0, before = 0;
        if (live) {
            // written before this kernel: read ahead of the arrival
            const uint32_t* pw = reinterpret_cast<const uint32_t*>(a.nodes + p);
            L = __ldg(pw + 6);
            R = __ldg(pw + 7);
            grand = __ldg(a.parents + p);
            count = __ldg(a.counts + p);
            if (lane == 0) before = arrive_at(a, p);
        }
        before = __shfl_sync(0xffffffffu, before, 0, 8);
        __syncwarp();  // orders the group's loads after lane 0's acquire
        live = live && before != 0;
        if (live) {
            const bool from_left = L == child;
            const uint32_t other = from_left ? R : L;
            if (lane == 7) {
                const Carry o = read_carry(other);
                c = complete_node(a, p, L, R, count, from_left ? c : o, from_left ? o : c);
            }
            if (slabs) {
                const Slab sib = read_slab(other);
                own = merge_slab(from_left ? own : sib, from_left ? sib : own);
                store_slab(a.summary, p, static_cast<int>(lane), own);
            }
            if (lane == 0 && a.done_list) a.done_list[atomicAdd(a.done_count, 1u)] = p;
            child = p;
            p = grand;
        }
        __syncwarp();  // the group's outputs before lane 0's next release
    }
}

__global__ void __launch_bounds__(kThreads) roots_kernel(const uint32_t* parents, const uint8_t* flags,
                                                         const uint32_t* counts, uint32_t nn, uint32_t* sizes,
                                                         const uint32_t* err) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nn) return;
    if (*err) {
        sizes[c] = 0;
        return;
    }
    const uint32_t p = parents[c];
    sizes[c] = (c != 0 && p < nn && flags[c] && !flags[p] && counts[c] > 1) ? counts[c] : 0u;
}

// A collapse root's primitives: its sorted leaves backwards (right-first
// depth-first order), repeats skipped.
__global__ void __launch_bounds__(kThreads) gather_kernel(const uint32_t* sizes, const uint32_t* offsets,
                                                          const uint32_t* first, const uint32_t* order, uint32_t nn,
                                                          kr_bvh_node* collapsed, uint32_t* counts,
                                                          uint32_t* primitives, uint32_t* err) {
    const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nn) return;
    const uint32_t cnt = sizes[c];
    if (cnt == 0) return;
    if (cnt > kMaxLeafSize) {
        atomicOr(err, kErrBadInput);
        return;
    }
    const uint32_t f = first[c], off = offsets[c];
    uint32_t out[kMaxLeafSize];
    uint32_t pos = 0;
#pragma unroll
    for (uint32_t t = 0; t < kMaxLeafSize; ++t) {
        if (t < cnt) {
            const uint32_t prim = order[f + cnt - 1 - t];
            bool uniq = true;
#pragma unroll
            for (uint32_t q = 0; q < kMaxLeafSize; ++q) uniq = uniq && !(q < pos && out[q] == prim);
            if (uniq) {
#pragma unroll
                for (uint32_t q = 0; q < kMaxLeafSize; ++q)
                    if (q == pos) out[q] = prim;
                ++pos;
            }
        }
    }
#pragma unroll
    for (uint32_t q = 0; q < kMaxLeafSize; ++q)
        if (q < pos) primitives[off + q] = out[q];
    // pos equals cnt for a permutation order; the count is rewritten only if
    // not, so that the OBB extents (on another stream) read it undisturbed
    if (pos != cnt) counts[c] = pos;
    uint32_t* cw = reinterpret_cast<uint32_t*>(collapsed + c);
    cw[6] = off;
    cw[8] = (cw[8] & 0xffff0000u) | pos;
}

// ---------------------------------------------------------------------------
size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

struct Layout {
    size_t lbvh, ctl, first, tris, summary, flags, cand, arrivals, keys, sizes, offsets, scan, frontier, chains,
        chain_counts, across, total;
};

Layout layout(uint32_t n) {
    const size_t ni = n > 1 ? n - 1 : 1;
    const size_t nn = n > 0 ? 2ull * n - 1 : 1;
    Layout L;
    size_t o = 0;
    L.lbvh = o;     o += align256(lbvh::layout(n).total);
    L.ctl = o;      o += align256(sizeof(Ctl));
    L.first = o;    o += align256(4 * ni);
    L.tris = o;     o += align256(36ull * (n > 0 ? n : 1));
    L.summary = o;  o += align256(112 * ni);
    L.flags = o;    o += align256(nn);
    L.cand = o;     o += align256(obbtree::cand_bytes(static_cast<uint32_t>(ni)));
    L.arrivals = o; o += align256(4 * ni);
    L.keys = o;     o += align256(24 * ni);
    L.sizes = o;    o += align256(4 * nn);
    L.offsets = o;  o += align256(4 * nn);
    L.scan = o;     o += align256(scan_temp_bytes(nn));
    L.frontier = o; o += align256(4 * nn + 4 * kThreads);
    L.chains = o;   o += align256(obbtree::chain_bytes(n));
    L.chain_counts = o; o += align256(obbtree::chain_count_bytes(n));
    L.across = o;   o += align256(4 * ni);
    L.total = o;
    return L;
}

StatusWords status_words(uint32_t n) {
    const Layout L = layout(n);
    StatusWords w;
    w.error = L.ctl + offsetof(Ctl, error);
    w.slots = L.ctl + offsetof(Ctl, total_slots);
    w.lbvh_error = L.lbvh + 4;  // lbvh::Ctl {ticket, error}
    return w;
}

kr_error enqueue(const kr_vec3* verts, const kr_uvec4* faces, uint32_t n, uint32_t flags, float ci, float ct,
                 kr_bvh_node* nodes, uint32_t* parents, uint32_t* counts, float* costs, kr_aabb3* bounds,
                 kr_obb3* obbs, kr_mat4* xfs, kr_bvh_node* collapsed, uint32_t* primitives, void* workspace,
                 cudaStream_t s) {
    const bool want_obbs = (flags & OBVH_BUILD_OBBS) != 0;
    const bool want_collapse = (flags & OBVH_BUILD_COLLAPSE) != 0;
    if (n < 1) return "obvh_build: at least one primitive is needed";
    if (!verts || !faces || !nodes || !parents || !counts || !costs || !workspace)
        return "obvh_build: null pointer argument";
    if (want_obbs && (!obbs || !xfs)) return "obvh_build: OBVH_BUILD_OBBS needs obbs and transforms";
    if (want_obbs && ((reinterpret_cast<uintptr_t>(xfs) & 15) || (reinterpret_cast<uintptr_t>(obbs) & 3)))
        return "obvh_build: transforms must be 16-byte and boxes 4-byte aligned";
    if ((reinterpret_cast<uintptr_t>(nodes) & 3) || (collapsed && (reinterpret_cast<uintptr_t>(collapsed) & 3)))
        return "obvh_build: node arrays must be 4-byte aligned";
    if (want_collapse && (!collapsed || !primitives)) return "obvh_build: OBVH_BUILD_COLLAPSE needs collapsed nodes and primitives";
    if (reinterpret_cast<uintptr_t>(workspace) & 255) return "obvh_build: workspace must be 256-byte aligned";
    char* ws = static_cast<char*>(workspace);
    const Layout L = layout(n);
    const uint32_t internal = n - 1, nn = 2 * n - 1;
    Ctl* ctl = reinterpret_cast<Ctl*>(ws + L.ctl);
    uint32_t* first = reinterpret_cast<uint32_t*>(ws + L.first);
    float* tris = reinterpret_cast<float*>(ws + L.tris);
    uint4* summary = reinterpret_cast<uint4*>(ws + L.summary);
    uint8_t* cflags = reinterpret_cast<uint8_t*>(ws + L.flags);
    const unsigned gn = (n + kThreads - 1) / kThreads;

    lbvh::Codes c;
    OBVH_TRY(lbvh::enqueue_codes(verts, faces, n, ws + L.lbvh, s, &c));
    {
        ProfScope prof_scope_("leaves_fused_kernel", s);
        const TreeArgs ta{c.codes, parents, first, counts, reinterpret_cast<uint32_t*>(ctl),
                          reinterpret_cast<const float*>(c.boxes), reinterpret_cast<float*>(bounds)};
        leaves_fused_kernel<<<2 * gn, kThreads, 0, s>>>(ta, c.order, verts, reinterpret_cast<const uint4*>(faces),
                                                    n, nodes, want_collapse ? collapsed : nullptr, tris,
                                                    want_obbs ? obbs : nullptr, xfs, c.visits,
                                                    want_collapse ? cflags : nullptr);
    }
    OBVH_TRY_CUDA(cudaGetLastError());
    OBVH_TRY(allow_dynamic_smem(reinterpret_cast<const void*>(fused_up_local_kernel), kFusedSmemBytes));
    // Two helper streams.  aux[0] (the highest priority, so that its CTAs
    // are placed first) takes the latency-bound walk up the top of the tree
    // and then the candidate frames of the nodes it completed, while the
    // caller's stream searches the frames of the nodes fused_up_local
    // completed; aux[1] takes the collapse's gather beside the extents.
    const bool frames = want_obbs && internal > 0;
    ForkStreams* fk = nullptr;
    OBVH_TRY(fork_streams(s, &fk));
    obbtree::FrameBuffers fb;
    uint32_t* across = reinterpret_cast<uint32_t*>(ws + L.across);
    if (frames) {
        fb.summary = summary;
        fb.points = reinterpret_cast<const kr_vec3*>(tris);
        fb.counts = counts;
        fb.first = first;
        fb.tris = tris;
        fb.cand = ws + L.cand;
        fb.arrivals = reinterpret_cast<uint32_t*>(ws + L.arrivals);
        fb.keys = reinterpret_cast<uint32_t*>(ws + L.keys);
        fb.err = &ctl->error;
        fb.parents = parents;
        fb.chains = reinterpret_cast<uint32_t*>(ws + L.chains);
        fb.chain_counts = reinterpret_cast<uint32_t*>(ws + L.chain_counts);
        fb.across_list = across;
        fb.across_count = &ctl->across;
    }
    {
        UpArgs a{nodes, want_collapse ? collapsed : nullptr, parents, first, tris, n, counts, costs,
                 want_collapse ? cflags : nullptr, ci, ct, want_obbs ? summary : nullptr, c.visits, &ctl->error};
        // per part-1 CTA: the list of its walks, and its length (the collapse's
        // sizes are written after the walk)
        uint32_t* frontier = reinterpret_cast<uint32_t*>(ws + L.frontier);
        uint32_t* lists = reinterpret_cast<uint32_t*>(ws + L.sizes);
        {
            ProfScope prof_scope_("fused_up_local_kernel", s);
            fused_up_local_kernel<<<gn, kThreads, kFusedSmemBytes, s>>>(a, frontier, lists);
        }
        OBVH_TRY_CUDA(cudaGetLastError());
        OBVH_TRY(fork_to(*fk, 0, s));
        cudaStream_t ws0 = fk->aux[0];
        if (frames) {
            a.done_list = across;
            a.done_count = &ctl->across;
        }
        {
            ProfScope prof_scope_("fused_up_cross_kernel", ws0);
            if (n <= kSuperLarge) {
                constexpr unsigned kBlocks = 1u << (kSuperShiftSmall - kLocalShift);
                fused_up_cross_kernel<kSuperShiftSmall>
                    <<<(gn + kBlocks - 1) / kBlocks, kThreads, 0, ws0>>>(a, frontier, lists, gn);
            } else {
                constexpr unsigned kBlocks = 1u << (kSuperShiftLarge - kLocalShift);
                fused_up_cross_kernel<kSuperShiftLarge>
                    <<<(gn + kBlocks - 1) / kBlocks, kThreads, 0, ws0>>>(a, frontier, lists, gn);
            }
        }
        OBVH_TRY_CUDA(cudaGetLastError());
        if (want_collapse) {
            // reads the collapse marks, counts and first leaves (final after
            // the walk); writes only collapse outputs, which the frames never read
            OBVH_TRY(fork_to(*fk, 1, ws0));
            cudaStream_t cs = fk->aux[1];
            uint32_t* sizes = reinterpret_cast<uint32_t*>(ws + L.sizes);
            uint32_t* offsets = reinterpret_cast<uint32_t*>(ws + L.offsets);
            const unsigned gnn = (nn + kThreads - 1) / kThreads;
            {
                ProfScope prof_scope_("roots_kernel", cs);
                roots_kernel<<<gnn, kThreads, 0, cs>>>(parents, cflags, counts, nn, sizes, &ctl->error);
            }
            OBVH_TRY_CUDA(cudaGetLastError());
            OBVH_TRY(exclusive_scan_u32(sizes, offsets, nn, &ctl->total_slots, ws + L.scan, cs));
            {
                ProfScope prof_scope_("gather_kernel", cs);
                gather_kernel<<<gnn, kThreads, 0, cs>>>(sizes, offsets, first, c.order, nn, collapsed, counts,
                                                        primitives, &ctl->error);
            }
            OBVH_TRY_CUDA(cudaGetLastError());
        }
        if (frames) {
            OBVH_TRY(obbtree::enqueue_candidates(fb, internal, obbtree::FrameNodes::kAcross, kLocalShift, obbs, xfs,
                                                 ws0));
            // a node is completed by fused_up_local iff its leaves lie inside one CTA's kThreads leaves
            OBVH_TRY(obbtree::enqueue_candidates(fb, internal, obbtree::FrameNodes::kInside, kLocalShift, obbs, xfs, s));
        }
        OBVH_TRY(join_from(*fk, 0, s));
    }
    if (frames) OBVH_TRY(obbtree::enqueue_extents(fb, internal, obbs, xfs, s));
    if (want_collapse) OBVH_TRY(join_from(*fk, 1, s));
    return kr_success;
}

}  // namespace pipeline
}  // namespace obvh

using namespace obvh;

extern "C" kr_size obvh_build_workspace_bytes(kr_u32 face_count) { return pipeline::layout(face_count).total; }

extern "C" kr_error obvh_build_workspace_init(void* d_workspace, kr_u32 face_count, void* stream) {
    if (!d_workspace) return "obvh_build_workspace_init: null workspace";
    // the LBVH stage's control block (CTA ticket) must start at zero
    cudaError_t e = cudaMemsetAsync(static_cast<char*>(d_workspace) + pipeline::layout(face_count).lbvh, 0, 256,
                                    static_cast<cudaStream_t>(stream));
    return e == cudaSuccess ? kr_success : cuda_error(e);
}

extern "C" kr_error obvh_build_async(const kr_vec3* d_vertices, const kr_uvec4* d_faces, kr_u32 face_count,
                                     kr_u32 flags, kr_scalar ci, kr_scalar ct, kr_bvh_node* d_nodes,
                                     kr_u32* d_parents, kr_u32* d_primitive_counts, kr_scalar* d_costs,
                                     kr_aabb3* d_bounds, kr_obb3* d_obbs, kr_mat4* d_transforms,
                                     kr_bvh_node* d_collapsed, kr_u32* d_primitives, void* d_workspace,
                                     void* stream) {
    kr_error e = pipeline::enqueue(d_vertices, d_faces, face_count, flags, ci, ct, d_nodes, d_parents,
                                   d_primitive_counts, d_costs, d_bounds, d_obbs, d_transforms, d_collapsed,
                                   d_primitives, d_workspace, static_cast<cudaStream_t>(stream));
    if (e) set_last_error(e);
    return e;
}

extern "C" kr_error obvh_build_graph_create(const kr_vec3* d_vertices, const kr_uvec4* d_faces, kr_u32 face_count,
                                            kr_u32 flags, kr_scalar ci, kr_scalar ct, kr_bvh_node* d_nodes,
                                            kr_u32* d_parents, kr_u32* d_primitive_counts, kr_scalar* d_costs,
                                            kr_aabb3* d_bounds, kr_obb3* d_obbs, kr_mat4* d_transforms,
                                            kr_bvh_node* d_collapsed, kr_u32* d_primitives, void* d_workspace,
                                            obvh_build_graph* out) {
    const kr_error e = create_build_graph(
        [&](cudaStream_t s) {
            return pipeline::enqueue(d_vertices, d_faces, face_count, flags, ci, ct, d_nodes, d_parents,
                                     d_primitive_counts, d_costs, d_bounds, d_obbs, d_transforms, d_collapsed,
                                     d_primitives, d_workspace, s);
        },
        out);
    if (e) set_last_error(e);
    return e;
}

extern "C" kr_error obvh_build_graph_launch(obvh_build_graph g, void* stream) {
    kr_error e = g ? kr_success : "obvh_build_graph_launch: null graph";
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int dev = -1;
    if (!e && cudaStreamGetDevice(s, &dev) != cudaSuccess) e = "obvh_build_graph_launch: unknown stream";
    if (!e && dev != g->device) e = "obvh_build_graph_launch: the stream belongs to another device than the graph";
    if (!e) {
        ProfScope prof_scope_("build_graph", s);
        const cudaError_t ce = cudaGraphLaunch(g->exec, s);
        if (ce != cudaSuccess) e = cuda_error(ce);
    }
    if (e) set_last_error(e);
    return e;
}

extern "C" kr_error obvh_build_graph_destroy(obvh_build_graph g) {
    if (!g) return kr_success;
    kr_error e = kr_success;
    if (g->exec && cudaGraphExecDestroy(g->exec) != cudaSuccess) e = "obvh_build_graph_destroy: graph exec";
    if (g->graph && cudaGraphDestroy(g->graph) != cudaSuccess) e = "obvh_build_graph_destroy: graph";
    delete g;
    if (e) set_last_error(e);
    return e;
}

extern "C" kr_error obvh_build_status(const void* d_workspace, kr_u32 face_count, void* stream, kr_u32* device_error,
                                      kr_u32* primitive_slots) {
    if (!d_workspace) return "obvh_build_status: null workspace";
    pipeline::Ctl ctl;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const char* base = static_cast<const char*>(d_workspace);
    cudaError_t e = cudaMemcpyAsync(&ctl, base + pipeline::layout(face_count).ctl, sizeof ctl, cudaMemcpyDeviceToHost, s);
    uint32_t lerr = 0;
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(&lerr, base + pipeline::layout(face_count).lbvh + 4, sizeof lerr, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_error(e);
    if (device_error) *device_error = ctl.error | lerr;
    if (primitive_slots) *primitive_slots = ctl.total_slots;
    return kr_success;
}
