// atrbvh.cu - the reference's ATRBVH builder on the GPU: an LBVH over 63-bit
// Morton codes, restructured by agglomerative treelet optimisation, handed on
// as kr_bvh_node records (src/ads/atrbvh_gpu/atrbvh.cu:258-380 with
// LBVHBuilder.cpp:33-139 and AgglomerativeTreeletOptimizer.cpp:22-117).
//
//   scene box        union of the triangle boxes (atrbvh.cu:282-298)
//   morton63_kernel  centroid of the triangle box in the scene box, 21 bits
//                    per axis (LBVH.cu:72-93, Commons.cuh:422-430,602-638)
//   radix sort       stable, 64-bit keys with the triangle index as value
//   karras63_kernel  Karras tree with index tie-break and the doubling-divisor
//                    split search (LBVH.cu:156-300)
//   boxes_up_kernel  leaf boxes and bottom-up node boxes and areas
//                    (LBVH.cu:414-447,551-648)
//   treelet_starts_kernel  the nodes where a pass begins
//   treelet_kernel   one bottom-up pass per iteration (gamma = tau, 2 tau,
//                    ...): at every node whose subtree holds at least gamma
//                    triangles, the warp forms a treelet of tau leaves by
//                    largest area, merges them agglomeratively by smallest
//                    union area, and keeps the result if its SAH is lower
//                    (AgglomerativeTreelet.cu:405-570, Treelet.cuh:55-129)
//   emit_kernel      SoA tree -> kr_bvh_node + parents (atrbvh.cu:95-123),
//                    then the LBVH refit for bounds, counts and costs, or,
//                    for a full commit, one walk that also does the
//                    transform's summaries and the collapse's marks
//                    (obbtree::enqueue_walk).
//
// The reference runs its treelet kernel with __syncthreads() inside
// warp-divergent loops; every shared array it touches there is per warp, so
// here each warp synchronises only itself (__syncwarp).  The two warp
// reductions that pick the leaf to expand and the pair to merge are a redux for
// the value and one for the place that the reference's shuffle-down order and
// strict comparisons prefer among equals, so ties resolve as there (a NaN area
// takes the reference's own steps).  Node data written by other warps is read through L2 (__ldcg) after
// the arrival counter's acquire.
#include <cuda_runtime.h>

#include <cfloat>
#include <cstdint>
#include <mutex>
#include <unordered_map>

#include "collapse_host.h"
#include "device_common.cuh"
#include "lbvh_host.h"
#include "obb_tree_host.h"
#include "obvh_atrbvh.h"
#include "obvh_build.h"
#include "runtime.h"
#include "sort.h"
#include "tree_device.cuh"

namespace obvh {
namespace atrbvh {

constexpr int kThreads = 256;
constexpr int kTreeletThreads = 128;
// 72 registers; 6, 8 and 10 blocks an SM were slower (917K-triangle knot:
// 2,448, 2,418, 2,425 and 2,516 us a build with 6, 7, 8 and 10).
constexpr int kTreeletBlocks = 7;
constexpr int kTreeletWarps = kTreeletThreads / 32;
constexpr int kMinTau = 3;
constexpr int kMaxTau = 20;

// One node of the working tree (48 bytes).  A node carries its children's
// areas, so that growing a treelet through it takes one 16-byte load (its
// children) instead of a chain of two (the children, then their areas).
struct __align__(16) TNode {
    float lo[3], hi[3];
    float area;
    int32_t parent;
    int32_t left, right;     // -1 in a leaf
    float area_l, area_r;    // the children's areas; in a leaf area_r holds the triangle's index as bits
};
static_assert(sizeof(TNode) == 48, "TNode is 48 bytes");

struct Ctl {
    uint32_t error;
    uint32_t pad[63];
};

// ---------------------------------------------------------------------------
__device__ __forceinline__ float box_area(const float* lo, const float* hi) {  // Commons.cuh:95-139
    const float sx = hi[0] - lo[0], sy = hi[1] - lo[1], sz = hi[2] - lo[2];
    return 2 * (sx * sy + sx * sz + sy * sz);
}

__device__ __forceinline__ float union_area(const float* alo, const float* ahi, const float* blo, const float* bhi) {
    const float sx = fmaxf(ahi[0], bhi[0]) - fminf(alo[0], blo[0]);  // Commons.cuh:173-190
    const float sy = fmaxf(ahi[1], bhi[1]) - fminf(alo[1], blo[1]);
    const float sz = fmaxf(ahi[2], bhi[2]) - fminf(alo[2], blo[2]);
    return 2 * (sx * sy + sx * sz + sy * sz);
}

__device__ __forceinline__ uint64_t expand_bits64(uint64_t v) {  // 21 bits -> every third of 63
    v &= 0x1fffffu;
    v = (v | v << 32) & 0x1f00000000ffffull;
    v = (v | v << 16) & 0x1f0000ff0000ffull;
    v = (v | v << 8) & 0x100f00f00f00f00full;
    v = (v | v << 4) & 0x10c30c30c30c30c3ull;
    v = (v | v << 2) & 0x1249249249249249ull;
    return v;
}

__global__ void __launch_bounds__(kThreads) morton63_kernel(const kr_vec3* verts, const uint4* faces, uint32_t n,
                                                            const kr_aabb3* scene, uint64_t* keys, uint32_t* vals) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint4 f = __ldg(faces + i);
    const f3 a = tree::load_vertex(verts, f.x), b = tree::load_vertex(verts, f.y), c = tree::load_vertex(verts, f.z);
    const float* sb = reinterpret_cast<const float*>(scene);
    const float va[3] = {a.x, a.y, a.z}, vb[3] = {b.x, b.y, b.z}, vc[3] = {c.x, c.y, c.z};
    uint64_t code = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float lo = fminf(fminf(va[k], vb[k]), vc[k]);
        const float hi = fmaxf(fmaxf(va[k], vb[k]), vc[k]);
        const float centre = (hi + lo) * 0.5f;
        const float u = (centre - sb[k]) / (sb[3 + k] - sb[k]);
        const uint64_t q = static_cast<uint64_t>(fminf(fmaxf(u * 2097152.0f, 0.0f), 2097151.0f));
        code |= expand_bits64(q) << (2 - k);
    }
    keys[i] = code;
    vals[i] = i;
}

__device__ __forceinline__ void set_triangle(TNode* leaf, int32_t tri) {
    *reinterpret_cast<int32_t*>(&leaf->area_r) = tri;
}
__device__ __forceinline__ int32_t triangle_of(const TNode* leaf) {
    return *reinterpret_cast<const int32_t*>(&leaf->area_r);
}

// longestCommonPrefix over 64-bit keys with the index tie-break (LBVH.cu:171-185).
__device__ __forceinline__ int lcp64(const uint64_t* keys, uint32_t n, int i, int j, uint64_t ki) {
    if (j < 0 || j >= static_cast<int>(n)) return -1;
    const uint64_t kj = __ldg(keys + j);
    if (ki == kj) return 64 + __clz(i ^ j);
    return __clzll(ki ^ kj);
}

__global__ void __launch_bounds__(kThreads) karras63_kernel(const uint64_t* keys, const uint32_t* order, uint32_t n,
                                                            TNode* t, int32_t* tris, uint32_t* err) {
    const int i = static_cast<int>(blockIdx.x * blockDim.x + threadIdx.x);
    const int internal = static_cast<int>(n) - 1;
    if (i >= internal) return;
    const uint64_t k1 = __ldg(keys + i);
    const int l1 = lcp64(keys, n, i, i + 1, k1), l2 = lcp64(keys, n, i, i - 1, k1);
    const int d = (l1 - l2 > 0) - (l1 - l2 < 0);
    if (d == 0) {  // cannot happen with the index tie-break; guards the searches below
        atomicOr(err, kErrBadInput);
        return;
    }
    const int minlcp = lcp64(keys, n, i, i - d, k1);
    int lmax = 2;
    while (lcp64(keys, n, i, i + lmax * d, k1) > minlcp) lmax <<= 1;
    int l = 0;
    for (int s = lmax >> 1; s >= 1; s >>= 1)
        if (lcp64(keys, n, i, i + (l + s) * d, k1) > minlcp) l += s;
    const int j = i + l * d;
    const int nodelcp = lcp64(keys, n, i, j, k1);
    int s = 0;
    const int maxdiv = 1 << (32 - __clz(l));
    for (int divisor = 2; divisor <= maxdiv; divisor <<= 1) {
        const int step = (l + divisor - 1) / divisor;
        if (lcp64(keys, n, i, i + (s + step) * d, k1) > nodelcp) s += step;
    }
    const int split = i + s * d + min(d, 0);
    int li = split, ri = split + 1;
    if (min(i, j) == split) {
        li = split + internal;
        set_triangle(t + li, static_cast<int32_t>(__ldg(order + split)));
    }
    if (max(i, j) == split + 1) {
        ri = split + 1 + internal;
        set_triangle(t + ri, static_cast<int32_t>(__ldg(order + split + 1)));
    }
    t[i].left = li;
    t[i].right = ri;
    tris[i] = l + 1;  // a triangle per key of the node's range
    t[li].parent = i;
    t[ri].parent = i;
    if (i == 0) t[0].parent = -1;
}

__device__ __forceinline__ void store_box(TNode* t, int32_t i, const float* lo, const float* hi) {
    __stcg(reinterpret_cast<float4*>(t[i].lo), make_float4(lo[0], lo[1], lo[2], hi[0]));
    __stcg(reinterpret_cast<float2*>(t[i].hi + 1), make_float2(hi[1], hi[2]));
    __stcg(&t[i].area, box_area(lo, hi));
}

__device__ __forceinline__ void load_box(const TNode* t, int32_t i, float* lo, float* hi) {
    const float4 a = __ldcg(reinterpret_cast<const float4*>(t[i].lo));
    const float2 b = __ldcg(reinterpret_cast<const float2*>(t[i].hi + 1));
    lo[0] = a.x; lo[1] = a.y; lo[2] = a.z;
    hi[0] = a.w; hi[1] = b.x; hi[2] = b.y;
}

// A node's children and their areas.
struct Kids {
    int32_t left, right;
    float area_l, area_r;
};
__device__ __forceinline__ Kids load_kids(const TNode* t, int32_t i) {
    const int4 k = __ldcg(reinterpret_cast<const int4*>(&t[i].left));
    return Kids{k.x, k.y, __int_as_float(k.z), __int_as_float(k.w)};
}

// Leaf boxes, then node boxes and SAHs bottom-up (the second thread to arrive
// merges).  The SAH of a node is ci area + left + right, of a leaf ct area
// (AgglomerativeTreelet.cu:405-570); the treelet passes start from them.
__global__ void __launch_bounds__(kThreads) boxes_up_kernel(const kr_vec3* verts, const uint4* faces, uint32_t n,
                                                            TNode* t, int32_t* tris, float* sah_arr, float ci,
                                                            float ct, uint32_t* visits, uint32_t* err) {
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31;
    const int32_t internal = static_cast<int32_t>(n) - 1;
    bool live = j < n;
    int32_t child = internal + static_cast<int32_t>(live ? j : 0u);
    const int32_t tri = triangle_of(t + child);
    if (live && (tri < 0 || tri >= static_cast<int32_t>(n))) {
        atomicOr(err, kErrBadInput);
        live = false;
    }
    float lo[3] = {0.f, 0.f, 0.f}, hi[3] = {0.f, 0.f, 0.f}, area = 0.f, sah = 0.f;
    int32_t p = -1;
    if (live) {
        const uint4 f = __ldg(faces + tri);
        const f3 a = tree::load_vertex(verts, f.x), b = tree::load_vertex(verts, f.y), c = tree::load_vertex(verts, f.z);
        lo[0] = fminf(fminf(a.x, b.x), c.x); lo[1] = fminf(fminf(a.y, b.y), c.y); lo[2] = fminf(fminf(a.z, b.z), c.z);
        hi[0] = fmaxf(fmaxf(a.x, b.x), c.x); hi[1] = fmaxf(fmaxf(a.y, b.y), c.y); hi[2] = fmaxf(fmaxf(a.z, b.z), c.z);
        t[child].left = -1;
        t[child].right = -1;
        tris[child] = 1;
        area = box_area(lo, hi);
        sah = ct * area;
        store_box(t, child, lo, hi);
        __stcg(sah_arr + child, sah);
        p = t[child].parent;
    }
    int32_t L = 0, R = 0, grand = -1;
    uint32_t steps = 0;
    // p's children and parent are final before this kernel
    const auto at_parent = [&] {
        if (!live) return;
        if (p < 0 || steps > n || p >= internal) {
            if (p >= 0) atomicOr(err, kErrCycle);
            live = false;
            return;
        }
        L = __ldg(&t[p].left);
        R = __ldg(&t[p].right);
        grand = __ldg(&t[p].parent);
    };
    // p from its child here and the sibling's box, area and cost
    const auto complete = [&](const float slo[3], const float shi[3], float other, float other_sah) {
        __stcg(reinterpret_cast<float2*>(&t[p].area_l), L == child ? make_float2(area, other) : make_float2(other, area));
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = fminf(lo[k], slo[k]);
            hi[k] = fmaxf(hi[k], shi[k]);
        }
        area = box_area(lo, hi);
        sah = ci * area + (L == child ? sah : other_sah) + (L == child ? other_sah : sah);
        store_box(t, p, lo, hi);
        __stcg(sah_arr + p, sah);
        child = p;
        p = grand;
        ++steps;
        at_parent();
    };
    at_parent();
    // Lanes that stand at one parent meet in the warp, without arrivals, until
    // no two do; only then each walk goes on alone, a fence and an atomic at
    // GPU scope for each level (917,504 triangles 145 -> 138 us, a build of
    // 100,000 857 -> 848 us: the upper levels' chain is what is left).
    for (;;) {
        uint32_t partner;
        const bool pair = tree::paired(live, static_cast<uint32_t>(p), static_cast<uint32_t>(child),
                                       static_cast<uint32_t>(L), static_cast<uint32_t>(R), lane, partner);
        if (!__any_sync(0xffffffffu, pair)) break;
        float slo[3], shi[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            slo[k] = __shfl_sync(0xffffffffu, lo[k], partner);
            shi[k] = __shfl_sync(0xffffffffu, hi[k], partner);
        }
        const float other = __shfl_sync(0xffffffffu, area, partner), other_sah = __shfl_sync(0xffffffffu, sah, partner);
        if (pair) {
            if (L == child) complete(slo, shi, other, other_sah);
            else live = false;
        }
        __syncwarp();
    }
    __syncwarp();  // the warp's outputs before its lanes' releases
    while (live) {
        if (tree::arrive(visits + p) == 0) return;
        const int32_t sib = L == child ? R : L;
        if (sib < 0 || sib >= static_cast<int32_t>(2 * n - 1)) {
            atomicOr(err, kErrCycle);
            return;
        }
        float slo[3], shi[3];
        load_box(t, sib, slo, shi);
        const float other_sah = __ldcg(sah_arr + sib);
        complete(slo, shi, box_area(slo, shi), other_sah);
    }
}

// ---------------------------------------------------------------------------
// Treelet optimisation.

// Per-treelet shared state (one per segment of W lanes; a treelet has at most
// W leaves).
template <int W>
struct SegSmem {
    int32_t internal[W];
    float dist[W * (W - 1) / 2];
};

// A treelet of tau <= W leaves is processed by a segment of W lanes (W = 8,
// 16 or 32), so a warp works on 32 / W treelets at once.  The reference uses a
// whole warp per treelet; its two reductions give the same winners here:
//   - the leaf to expand (Treelet.cuh:21-37): a shuffle-down over the first
//     2 + it <= tau lanes in which a lane keeps its own value on ties.  Lane 0
//     ends with the largest area, of equal ones the first in the order in
//     which the tree's lanes reach it, which depends on the lane count alone
//     (PickOrder);
//   - the pair to merge (AgglomerativeTreelet.cu:59-90): 32 virtual lanes v
//     scan the distance entries v, v + 32, ..., then a shuffle-down by 16, 8,
//     4, 2, 1 with strict '<'.  The smallest distance wins, of equal ones that
//     of the lane whose index has the smallest bit reversal (the last step
//     prefers even lanes, the one before those divisible by 4, ...), and
//     within a lane the first entry.
// So each is one redux for the value and one for the tie.
//
// The kernel's time is the latency of one treelet, level after level up the
// tree (about 23,000 cycles in an earlier form: 7 expansions behind two
// dependent loads each, 8 merges with five-step reductions and 45 shuffles).
template <int W>
__device__ __forceinline__ int seg_lane() { return threadIdx.x & (W - 1); }

template <int W>
__device__ __forceinline__ void reduce_down_max(int count, int& idx, float& val) {
    int amount = count / 2;
    while (count > 1) {
        const int oi = __shfl_down_sync(0xffffffffu, idx, amount, W);
        const float ov = __shfl_down_sync(0xffffffffu, val, amount, W);
        if (ov > val) {
            val = ov;
            idx = oi;
        }
        count = (count + 1) / 2;
        amount = count / 2;
    }
}

// rank[c][lane]: the place of `lane` among c lanes in the reduction's order of
// preference on ties: what lane 0 holds after the steps is its own candidates,
// then those of the lane `amount` above, at every step.
struct PickOrder {
    uint8_t rank[kMaxTau + 1][32];
    constexpr PickOrder() : rank{} {
        for (int c = 1; c <= kMaxTau; ++c) {
            int list[32][32] = {}, len[32] = {};
            for (int l = 0; l < c; ++l) {
                list[l][0] = l;
                len[l] = 1;
            }
            int count = c, amount = c / 2;
            while (count > 1) {
                for (int l = 0; l + amount < c; ++l) {  // ascending: list[l + amount] is still the old one
                    for (int k = 0; k < len[l + amount]; ++k) {
                        bool known = false;
                        for (int q = 0; q < len[l]; ++q) known = known || list[l][q] == list[l + amount][k];
                        if (!known) list[l][len[l]++] = list[l + amount][k];
                    }
                }
                count = (count + 1) / 2;
                amount = count / 2;
            }
            for (int k = 0; k < len[0]; ++k) rank[c][list[0][k]] = static_cast<uint8_t>(k);
        }
    }
};
__constant__ PickOrder c_pick = PickOrder();

// Reductions over the segments of a warp: one full-warp redux per segment, the
// other lanes giving the neutral value.  (A redux with the segment's own mask
// differs within the warp, and the mask of a redux is a uniform operand: the
// treelet passes took 1.67 ms instead of 1.44.)
template <int W>
__device__ __forceinline__ bool in_segment(int q) { return W == 32 || static_cast<int>(threadIdx.x & 31) / W == q; }
template <int W>
__device__ __forceinline__ float seg_min(float v) {
    float mine = v;
#pragma unroll
    for (int q = 0; q < 32 / W; ++q) {
        const float r = warp_min(in_segment<W>(q) ? v : kInf);
        if (in_segment<W>(q)) mine = r;
    }
    return mine;
}
template <int W>
__device__ __forceinline__ uint32_t seg_min(uint32_t v) {
    uint32_t mine = v;
#pragma unroll
    for (int q = 0; q < 32 / W; ++q) {
        const uint32_t r = __reduce_min_sync(0xffffffffu, in_segment<W>(q) ? v : 0xffffffffu);
        if (in_segment<W>(q)) mine = r;
    }
    return mine;
}
template <int W>
__device__ __forceinline__ uint32_t seg_max(uint32_t v) {
    uint32_t mine = v;
#pragma unroll
    for (int q = 0; q < 32 / W; ++q) {
        const uint32_t r = __reduce_max_sync(0xffffffffu, in_segment<W>(q) ? v : 0u);
        if (in_segment<W>(q)) mine = r;
    }
    return mine;
}

__device__ __forceinline__ int trm_index(int row, int col) { return ((row - 1) * row) / 2 + col; }
__device__ __forceinline__ int trm_row(int index) {  // TriangularMatrix.cuh:40-44
    return static_cast<int>((-1 + sqrtf(8.0f * index + 1)) / 2) + 1;
}
__device__ __forceinline__ int trm_col(int index) {
    const int y = trm_row(index);
    return index - (y * (y - 1)) / 2;
}

// Every index of the distance matrices of treelets of up to kMaxTau leaves as
// one word, tabulated once per CTA: its place in the reduction's order of
// preference on ties (bit-reversed virtual lane, then round) above its row and
// column, so that the winning word says which pair it is.
constexpr int kTrmEntries = (kMaxTau - 1) * kMaxTau / 2;
__device__ __forceinline__ uint32_t pair_word(int index) {
    return ((__brev(static_cast<uint32_t>(index & 31)) >> 27) << 24) | (static_cast<uint32_t>(index >> 5) << 16) |
           (static_cast<uint32_t>(trm_row(index)) << 8) | static_cast<uint32_t>(trm_col(index));
}
__device__ __forceinline__ int word_row(uint32_t w) { return (w >> 8) & 0xff; }
__device__ __forceinline__ int word_col(uint32_t w) { return w & 0xff; }

// The pair to merge among the first `size` entries (pair_word).
template <int W>
__device__ __forceinline__ uint32_t nearest_pair(const float* dist, int size, const uint32_t* words) {
    float best = FLT_MAX;
    uint32_t word = 0xffffffffu;
    for (int j = seg_lane<W>(); j < size; j += W) {
        const float d = dist[j];
        const uint32_t e = words[j];
        if (d < best || (d == best && e < word && word != 0xffffffffu)) {
            best = d;
            word = e;
        }
    }
    const float least = seg_min<W>(best);
    const uint32_t win = seg_min<W>(best == least ? word : 0xffffffffu);
    return win == 0xffffffffu ? words[0] : win;  // no finite distance: the reference's index 0
}

// The leaf to expand among the segment's first `count` lanes (area -FLT_MAX:
// not to be expanded).
template <int W>
__device__ __forceinline__ int largest_leaf(int count, float area, const uint8_t* rank) {
    const int sl = seg_lane<W>();
    const bool in = sl < count;
    if (__any_sync(0xffffffffu, in && area != area)) {  // a NaN area: the reference's own steps
        int idx = in ? sl : -1;
        float a = in ? area : -FLT_MAX;
        reduce_down_max<W>(count, idx, a);
        return __shfl_sync(0xffffffffu, idx, 0, W);
    }
    const uint32_t key = in ? f2key(area) : 0u;
    const uint32_t most = seg_max<W>(key);
    const uint32_t place = static_cast<uint32_t>(rank[32 * count + sl]) << 8 | static_cast<uint32_t>(sl);
    return static_cast<int>(seg_min<W>(in && key == most ? place : 0xffffffffu) & 0xffu);
}

template <int W>
__device__ __forceinline__ void shfl_box(const float* lo, const float* hi, int src, float* olo, float* ohi) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        olo[k] = __shfl_sync(0xffffffffu, lo[k], src, W);
        ohi[k] = __shfl_sync(0xffffffffu, hi[k], src, W);
    }
}

// The arrays a treelet pass works on.  `rec` is each node's SAH as a bottom-up
// pass over the tree as it stands would compute it: what the next pass takes
// as the SAH of the subtrees below its gamma.  (A merged node's `sah` is summed
// in another order, children first.)
struct PassArgs {
    TNode* t;
    float* sah;
    float* rec;
    int32_t* tris;
    int32_t n;
    int tau;
    int32_t gamma;
    float ci;
};

// A treelet root on the way up: its record and its sums.
struct Root {
    int32_t node;
    Kids kids;
    float sah, rec;
};

// The treelet rooted at `root`, by a segment of W lanes.  Every lane of the
// warp calls this together (the shuffles span the warp); a segment with
// `active` false computes nothing that is stored.  Leaves the root's SAHs
// after the pass in root.  Returns false (for the segment) on a malformed
// tree.  kLast: no pass follows, rec and the counts are not kept up.
template <int W, bool kLast>
__device__ bool process_treelet(const PassArgs& a, Root& root, bool active, SegSmem<W>& w, const uint32_t* words,
                                const uint8_t* rank) {
    const int sl = seg_lane<W>();
    const int tau = a.tau;
    const int32_t internal_count = a.n - 1;
    const int32_t node_count = 2 * a.n - 1;
    auto valid = [&](int32_t x) { return x >= 0 && x < node_count; };

    // formTreelet: grow by the frontier node of largest area (Treelet.cuh:55-129);
    // lane sl holds frontier node sl
    bool bad = !active || !valid(root.kids.left) || !valid(root.kids.right);
    int32_t node = sl == 0 ? root.kids.left : (sl == 1 ? root.kids.right : -1);
    float area = sl == 0 ? root.kids.area_l : root.kids.area_r;
    if (sl == 0) w.internal[0] = root.node;
    for (int it = 0; it < tau - 2; ++it) {
        const bool grows = !bad && node >= 0 && node < internal_count;
        const int idx = largest_leaf<W>(2 + it, grows ? area : -FLT_MAX, rank);
        const int32_t rep = __shfl_sync(0xffffffffu, node, idx < 0 ? 0 : idx, W);
        bad = bad || idx < 0 || rep < 0 || rep >= internal_count;
        Kids k{-1, -1, 0.f, 0.f};
        if (!bad) k = load_kids(a.t, rep);
        bad = bad || !valid(k.left) || !valid(k.right);
        if (sl == 0) w.internal[it + 1] = rep;
        if (sl == idx) {
            node = k.left;
            area = k.area_l;
        }
        if (sl == it + 2) {
            node = k.right;
            area = k.area_r;
        }
    }

    // Lane sl < tau holds treelet leaf sl: its node, area, SAH, box.
    float sah = 0.f, rec = 0.f, lo[3] = {0.f, 0.f, 0.f}, hi[3] = {0.f, 0.f, 0.f};
    int32_t count = 0;
    if (!bad && sl < tau) {
        sah = __ldcg(a.sah + node);
        if (!kLast) {
            rec = __ldcg(a.rec + node);
            count = __ldcg(a.tris + node);
        }
        load_box(a.t, node, lo, hi);
    }
    const int nd = (tau - 1) * tau / 2;
    for (int k0 = 0; k0 < nd; k0 += W) {  // every pair row > col
        const int k = k0 + sl;
        const uint32_t e = words[min(k, nd - 1)];
        float rlo[3], rhi[3], clo[3], chi[3];
        shfl_box<W>(lo, hi, word_row(e), rlo, rhi);
        shfl_box<W>(lo, hi, word_col(e), clo, chi);
        if (k < nd) w.dist[k] = union_area(rlo, rhi, clo, chi);
    }
    __syncwarp();

    // Merge the nearest pair (jr, jc), jr > jc, until one is left.  The merged
    // node takes place jc, the last one place jr; lane `last` is then free and
    // keeps the merge: its children (node, right), their areas, the box and
    // the sums.
    const int my_row = trm_index(sl, 0);
    int32_t right = -1;
    float area_l = 0.f, area_r = 0.f;
    for (int last = tau - 1; last > 0; --last) {
        const uint32_t e = nearest_pair<W>(w.dist, last * (1 + last) / 2, words);
        const int jr = word_row(e), jc = word_col(e);

        // updateState (AgglomerativeTreelet.cu:92-147).  One shuffle brings
        // place jr's value to all lanes but jr, and the last place's to jr.
        const bool is_jr = sl == jr;
        const int from = is_jr ? last : jr;
        const auto of_jr = [&](auto own, auto& moved) {
            moved = __shfl_sync(0xffffffffu, own, from, W);
            return is_jr ? own : moved;
        };
        int32_t mnode;
        float msah, marea, mlo[3], mhi[3];
        const int32_t li = of_jr(node, mnode), ri = __shfl_sync(0xffffffffu, node, jc, W);
        const float s = of_jr(sah, msah) + __shfl_sync(0xffffffffu, sah, jc, W);
        const float la = of_jr(area, marea), ra = __shfl_sync(0xffffffffu, area, jc, W);
        float ulo[3], uhi[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            ulo[k] = fminf(__shfl_sync(0xffffffffu, lo[k], jc, W), of_jr(lo[k], mlo[k]));
            uhi[k] = fmaxf(__shfl_sync(0xffffffffu, hi[k], jc, W), of_jr(hi[k], mhi[k]));
        }
        const float uarea = box_area(ulo, uhi);
        float mrec = 0.f, urec = 0.f;
        int32_t mcount = 0, ucount = 0;
        if (!kLast) {
            const float lrec = of_jr(rec, mrec);
            urec = a.ci * uarea + lrec + __shfl_sync(0xffffffffu, rec, jc, W);
            ucount = of_jr(count, mcount) + __shfl_sync(0xffffffffu, count, jc, W);
        }
        const bool merged = sl == jc || sl == last;
        if (is_jr || merged) {
            sah = merged ? s + a.ci * uarea : msah;
            area = merged ? uarea : marea;
            node = sl == last ? li : (sl == jc ? w.internal[last - 1] : mnode);
            if (!kLast) {
                rec = merged ? urec : mrec;
                count = merged ? ucount : mcount;
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                lo[k] = merged ? ulo[k] : mlo[k];
                hi[k] = merged ? uhi[k] : mhi[k];
            }
            if (sl == last) {
                right = ri;
                area_l = la;
                area_r = ra;
            }
        }

        // updateDistancesMatrix (AgglomerativeTreelet.cu:149-186): place jr's
        // distances are the last one's, place jc's are new.  The two write
        // different entries: (jr, jc) is left to lane jr's new distance.
        if (sl < last && sl != jc) {
            if (!is_jr) w.dist[sl > jr ? my_row + jr : trm_index(jr, sl)] = w.dist[trm_index(last, sl)];
            w.dist[sl > jc ? my_row + jc : trm_index(jc, sl)] = union_area(lo, hi, ulo, uhi);
        }
        __syncwarp();
    }

    // updateTreelet: keep the new topology if its SAH is lower.  Lane sl >= 1
    // holds the new internal node sl - 1; lane 1 the root.
    const float total = __shfl_sync(0xffffffffu, sah, 1, W);
    const float total_rec = kLast ? 0.f : __shfl_sync(0xffffffffu, rec, 1, W);
    if (!bad && total < root.sah) {
        root.sah = total;
        root.rec = total_rec;
        if (sl >= 1 && sl < tau) {
            const int32_t ni = w.internal[sl - 1];
            __stcg(reinterpret_cast<int4*>(&a.t[ni].left),
                   make_int4(node, right, __float_as_int(area_l), __float_as_int(area_r)));
            __stcg(&a.t[node].parent, ni);
            __stcg(&a.t[right].parent, ni);
            __stcg(a.sah + ni, sah);
            if (!kLast) {
                __stcg(a.rec + ni, rec);
                if (sl > 1) __stcg(a.tris + ni, count);  // the root's does not change
            }
            store_box(a.t, ni, lo, hi);
        }
    }
    __syncwarp();
    return !(active && bad);
}

// The lowest treelet roots: nodes of at least gamma triangles, both of whose
// children have fewer.  count[0] receives their number.
__global__ void __launch_bounds__(kThreads) treelet_starts_kernel(const TNode* t, const int32_t* tris, int32_t n,
                                                                  int32_t gamma, int32_t* starts, uint32_t* count) {
    const int32_t i = static_cast<int32_t>(blockIdx.x * blockDim.x + threadIdx.x);
    bool start = false;
    if (i < n - 1 && tris[i] >= gamma) {
        const Kids k = load_kids(t, i);
        start = tris[k.left] < gamma && tris[k.right] < gamma;
    }
    const uint32_t vote = __ballot_sync(0xffffffffu, start);
    if (!vote) return;
    const int lane = threadIdx.x & 31;
    uint32_t base = 0;
    if (lane == __ffs(vote) - 1) base = atomicAdd(count, __popc(vote));
    base = __shfl_sync(0xffffffffu, base, __ffs(vote) - 1);
    if (start) starts[base + __popc(vote & ((1u << lane) - 1u))] = i;
}

// One pass: each segment of W lanes takes a lowest root from the list, runs
// its treelet and goes up.  At a parent whose other child has fewer than gamma
// triangles nothing is waited for (that subtree has no treelet and does not
// change); else the second child to arrive carries on.  So the subtrees below
// gamma, nine tenths of the nodes, take no part: with a thread walking up from
// every leaf, 515,260 warp rounds of arrivals took 17,600 cycles each against
// 222,622 treelet rounds of 22,500 (917K-triangle knot).
template <int W, bool kLast>
__global__ void __launch_bounds__(kTreeletThreads, kTreeletBlocks)
    treelet_kernel(PassArgs a, uint32_t* counters, const int32_t* starts, uint32_t* queue, uint32_t* err) {
    constexpr int S = 32 / W;  // segments (treelets in flight) per warp
    __shared__ SegSmem<W> smem[kTreeletWarps * S];
    __shared__ uint32_t words[kTrmEntries];
    __shared__ uint8_t rank[(kMaxTau + 1) * 32];
    for (int k = threadIdx.x; k < kTrmEntries; k += kTreeletThreads) words[k] = pair_word(k);
    for (int k = threadIdx.x; k < (kMaxTau + 1) * 32; k += kTreeletThreads) rank[k] = c_pick.rank[k >> 5][k & 31];
    __syncthreads();
    const int lane = threadIdx.x & 31, sl = seg_lane<W>();
    SegSmem<W>& w = smem[(threadIdx.x >> 5) * S + lane / W];
    const int32_t internal = a.n - 1, node_count = 2 * a.n - 1;
    const uint32_t total = queue[0];  // queue: {starts listed, starts taken}
    Root root{-1, {-1, -1, 0.f, 0.f}, 0.f, 0.f};
    float area = 0.f;
    int32_t up = -1;
    uint32_t level = 0;
    bool dry = false;
    for (;;) {
        // a segment without a walk takes the next start
        const bool fresh = root.node < 0 && !dry;
        uint32_t at = total;
        if (fresh && sl == 0) at = atomicAdd(queue + 1, 1u);
        at = __shfl_sync(0xffffffffu, at, 0, W);
        if (fresh) {
            dry = at >= total;
            if (!dry) {
                root.node = __ldg(starts + at);
                root.kids = load_kids(a.t, root.node);
                area = __ldcg(&a.t[root.node].area);
                up = __ldcg(&a.t[root.node].parent);
                root.sah = a.ci * area + __ldcg(a.sah + root.kids.left) + __ldcg(a.sah + root.kids.right);
                if (!kLast)
                    root.rec = a.ci * area + __ldcg(a.rec + root.kids.left) + __ldcg(a.rec + root.kids.right);
                level = 0;
            }
        }
        const bool live = root.node >= 0;
        if (!__any_sync(0xffffffffu, live)) return;
        // the parent's record does not change before its own treelet (its
        // parent link not before an ancestor's): read it ahead
        Kids pk{-1, -1, 0.f, 0.f};
        float parea = 0.f;
        int32_t pup = -1;
        if (live && up >= 0 && up < internal) {
            pk = load_kids(a.t, up);
            parea = __ldcg(&a.t[up].area);
            pup = __ldcg(&a.t[up].parent);
        }
        if (live && sl == 0) {
            __stcg(a.sah + root.node, root.sah);
            if (!kLast) __stcg(a.rec + root.node, root.rec);
        }
        __syncwarp();
        const bool fine = process_treelet<W, kLast>(a, root, live, w, words, rank);
        if (!fine && sl == 0) atomicOr(err, kErrBadInput);
        // one level up: the first of two treelet children to arrive stops
        const bool left = pk.left == root.node;
        const int32_t sib = left ? pk.right : pk.left;
        bool carry = live && fine && up >= 0;
        if (carry && (up >= internal || sib < 0 || sib >= node_count || (!left && pk.right != root.node) ||
                      ++level > static_cast<uint32_t>(a.n))) {
            if (sl == 0) atomicOr(err, kErrCycle);
            carry = false;
        }
        const bool meets = carry && __ldcg(a.tris + sib) >= a.gamma;
        uint32_t before = 1;
        if (meets && sl == 0) before = tree::arrive(counters + up);
        before = __shfl_sync(0xffffffffu, before, 0, W);
        __syncwarp();  // orders the segment's loads after lane 0's acquire
        carry = carry && before != 0;
        if (carry) {
            const float other = __ldcg(a.sah + sib);
            root.sah = a.ci * parea + (left ? root.sah : other) + (left ? other : root.sah);
            if (!kLast) {
                const float orec = __ldcg(a.rec + sib);
                root.rec = a.ci * parea + (left ? root.rec : orec) + (left ? orec : root.rec);
            }
            root.node = up;
            root.kids = pk;
            up = pup;
        } else {
            root.node = -1;
        }
    }
}

// SoA tree -> kr_bvh_node and parents (copyTree_kernel, atrbvh.cu:95-123):
// internal nodes get their children and zero bounds, leaves their box, one
// primitive and the triangle index.
__global__ void __launch_bounds__(kThreads) emit_kernel(const TNode* t, uint32_t n, kr_bvh_node* nodes,
                                                        uint32_t* parents) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 2 * n - 1) return;
    const TNode& s = t[i];
    parents[i] = static_cast<uint32_t>(s.parent);
    uint32_t w[9];
    if (i < n - 1) {
        for (int k = 0; k < 6; ++k) w[k] = 0u;
        w[6] = static_cast<uint32_t>(s.left);
        w[7] = static_cast<uint32_t>(s.right);
        w[8] = 0u;
    } else {
        for (int k = 0; k < 3; ++k) {
            w[k] = __float_as_uint(s.lo[k]);
            w[3 + k] = __float_as_uint(s.hi[k]);
        }
        w[6] = static_cast<uint32_t>(triangle_of(&s));
        w[7] = 0u;
        w[8] = 1u;
    }
    uint32_t* d = reinterpret_cast<uint32_t*>(nodes + i);
    for (int k = 0; k < 9; ++k) d[k] = w[k];
}

// ---------------------------------------------------------------------------
// Host side.

size_t align256(size_t x) { return (x + 255) & ~static_cast<size_t>(255); }

struct Layout {
    size_t ctl, bounds_ws, scene, keys0, keys1, vals0, vals1, sort, tnodes, counters, tris, sah, obb_ws, col_ws,
        total;
};

Layout layout(uint32_t n) {
    const size_t nn = n > 0 ? 2ull * n - 1 : 1;
    Layout L;
    size_t o = 0;
    L.ctl = o;       o += align256(sizeof(Ctl));
    L.bounds_ws = o; o += align256(lbvh::layout(0).total);
    L.scene = o;     o += align256(2 * sizeof(kr_aabb3));
    L.keys0 = o;     o += align256(8ull * n);  // later: recomputed SAHs, 4 (2n - 1)
    L.keys1 = o;     o += align256(8ull * n);
    L.vals0 = o;     o += align256(4ull * n);
    L.vals1 = o;     o += align256(4ull * n);
    L.sort = o;      o += align256(radix_sort_temp_bytes(n));
    L.tnodes = o;    o += align256(sizeof(TNode) * nn);
    L.counters = o;  o += align256(4ull * nn);
    L.tris = o;      o += align256(4ull * nn);
    L.sah = o;       o += align256(4ull * nn);
    L.obb_ws = o;    o += align256(obbtree::layout(n).total);
    L.col_ws = o;    o += align256(collapse::layout(n).total);
    L.total = o;
    return L;
}

kr_error check_args(const kr_vec3* verts, const kr_uvec4* faces, uint32_t n, uint32_t tau, const void* ws) {
    if (n < 2) return "obvh_atrbvh: at least two triangles are needed";
    if (n > (1u << 30)) return "obvh_atrbvh: more than 2^30 triangles";
    if (!verts || !faces || !ws) return "obvh_atrbvh: null pointer argument";
    if (reinterpret_cast<uintptr_t>(ws) & 255) return "obvh_atrbvh: workspace must be 256-byte aligned";
    if (tau < static_cast<uint32_t>(kMinTau) || tau > static_cast<uint32_t>(kMaxTau))
        return "obvh_atrbvh: treelet size must be 3..20";
    return kr_success;
}

// A segment per lowest root (at most n / gamma of them), as far as the blocks
// are resident at once.
template <int W>
void launch_pass(const PassArgs& a, uint32_t* counters, const int32_t* starts, uint32_t* queue, uint32_t* err,
                 bool last, cudaStream_t s) {
    constexpr unsigned kPerBlock = kTreeletThreads / W;
    const unsigned want = static_cast<unsigned>(a.n / a.gamma) / kPerBlock + 1;
    const unsigned cap = kTreeletBlocks * static_cast<unsigned>(device_info().sm_count);
    const unsigned g = want < cap ? want : cap;
    if (last) treelet_kernel<W, true><<<g, kTreeletThreads, 0, s>>>(a, counters, starts, queue, err);
    else treelet_kernel<W, false><<<g, kTreeletThreads, 0, s>>>(a, counters, starts, queue, err);
}

// refit false: the nodes are emitted with zero internal bounds, and counts
// and costs are left to the caller's own bottom-up pass.
kr_error enqueue_tree(const kr_vec3* verts, const kr_uvec4* faces, uint32_t n, uint32_t tau, uint32_t iterations,
                      float ci, float ct, kr_bvh_node* nodes, uint32_t* parents, uint32_t* counts, float* costs,
                      kr_aabb3* scene_out, void* workspace, cudaStream_t s, bool refit = true) {
    OBVH_TRY(check_args(verts, faces, n, tau, workspace));
    if (!nodes || !parents || !counts || !costs) return "obvh_atrbvh: null pointer argument";
    char* ws = static_cast<char*>(workspace);
    const Layout L = layout(n);
    uint32_t* err = &reinterpret_cast<Ctl*>(ws + L.ctl)->error;
    kr_aabb3* scene = reinterpret_cast<kr_aabb3*>(ws + L.scene);
    TNode* t = reinterpret_cast<TNode*>(ws + L.tnodes);
    uint32_t* counters = reinterpret_cast<uint32_t*>(ws + L.counters);
    const unsigned grid_n = (n + kThreads - 1) / kThreads;
    const uint32_t internal = n - 1;
    int32_t* tris = reinterpret_cast<int32_t*>(ws + L.tris);
    float* sah = reinterpret_cast<float*>(ws + L.sah);
    // free once the tree is built: the sort's keys (8n bytes) and values
    float* rec = reinterpret_cast<float*>(ws + L.keys0);
    int32_t* starts = reinterpret_cast<int32_t*>(ws + L.vals0);

    // the transform's and the collapse's control blocks start at zero on every
    // build, so the status reads zero for the steps that do not run
    OBVH_TRY_CUDA(cudaMemsetAsync(ws + L.obb_ws, 0, 256, s));
    OBVH_TRY_CUDA(cudaMemsetAsync(ws + L.col_ws, 0, 256, s));
    OBVH_TRY(lbvh::enqueue_bounds(verts, faces, n, nullptr, ws + L.bounds_ws, scene, nullptr, true, s));
    {
        ProfScope prof_scope_("morton63_kernel", s);
        morton63_kernel<<<grid_n, kThreads, 0, s>>>(verts, reinterpret_cast<const uint4*>(faces), n, scene,
                                                    reinterpret_cast<uint64_t*>(ws + L.keys0),
                                                    reinterpret_cast<uint32_t*>(ws + L.vals0));
    }
    OBVH_TRY_CUDA(cudaGetLastError());
    bool alt = false;
    OBVH_TRY(radix_sort_pairs(ws + L.keys0, ws + L.keys1, reinterpret_cast<uint32_t*>(ws + L.vals0),
                              reinterpret_cast<uint32_t*>(ws + L.vals1), n, 8, 0, 63, ws + L.sort, s, &alt, err));
    const uint64_t* keys = reinterpret_cast<const uint64_t*>(ws + (alt ? L.keys1 : L.keys0));
    const uint32_t* order = reinterpret_cast<const uint32_t*>(ws + (alt ? L.vals1 : L.vals0));
    {
        ProfScope prof_scope_("karras63_kernel", s);
        karras63_kernel<<<(internal + kThreads - 1) / kThreads, kThreads, 0, s>>>(keys, order, n, t, tris, err);
    }
    OBVH_TRY_CUDA(cudaGetLastError());
    OBVH_TRY_CUDA(cudaMemsetAsync(counters, 0, 4ull * internal, s));
    {
        ProfScope prof_scope_("boxes_up_kernel", s);
        boxes_up_kernel<<<grid_n, kThreads, 0, s>>>(verts, reinterpret_cast<const uint4*>(faces), n, t, tris, rec, ci,
                                                    ct, counters, err);
    }
    OBVH_TRY_CUDA(cudaGetLastError());
    int32_t gamma = static_cast<int32_t>(tau);
    for (uint32_t it = 0; it < iterations; ++it) {
        // arrival counters, then the queue's two words behind them
        uint32_t* queue = counters + internal;
        OBVH_TRY_CUDA(cudaMemsetAsync(counters, 0, 4ull * (internal + 2), s));
        OBVH_TRY_CUDA(cudaMemcpyAsync(sah, rec, 4ull * (2ull * n - 1), cudaMemcpyDeviceToDevice, s));
        {
            ProfScope prof_scope_("treelet_starts_kernel", s);
            treelet_starts_kernel<<<(internal + kThreads - 1) / kThreads, kThreads, 0, s>>>(
                t, tris, static_cast<int32_t>(n), gamma, starts, queue);
        }
        OBVH_TRY_CUDA(cudaGetLastError());
        const PassArgs pa{t, sah, rec, tris, static_cast<int32_t>(n), static_cast<int>(tau), gamma, ci};
        const bool last = it + 1 == iterations;
        {
            ProfScope prof_scope_("treelet_kernel", s);
            if (tau <= 8) launch_pass<8>(pa, counters, starts, queue, err, last, s);
            else if (tau <= 16) launch_pass<16>(pa, counters, starts, queue, err, last, s);
            else launch_pass<32>(pa, counters, starts, queue, err, last, s);
        }
        OBVH_TRY_CUDA(cudaGetLastError());
        gamma = gamma > (1 << 29) ? gamma : 2 * gamma;
    }
    {
        ProfScope prof_scope_("emit_kernel", s);
        emit_kernel<<<(2 * n - 1 + kThreads - 1) / kThreads, kThreads, 0, s>>>(t, n, nodes, parents);
    }
    OBVH_TRY_CUDA(cudaGetLastError());
    if (refit) OBVH_TRY(lbvh::enqueue_refit(nodes, parents, counts, costs, counters, n, err, s));
    if (scene_out) OBVH_TRY_CUDA(cudaMemcpyAsync(scene_out, scene, sizeof(kr_aabb3), cudaMemcpyDeviceToDevice, s));
    return kr_success;
}

kr_error enqueue_full(const kr_vec3* verts, const kr_uvec4* faces, uint32_t n, uint32_t flags, uint32_t tau,
                      uint32_t iterations, float ci, float ct, kr_bvh_node* nodes, uint32_t* parents,
                      uint32_t* counts, float* costs, kr_aabb3* scene_out, kr_obb3* obbs, kr_mat4* xfs,
                      kr_bvh_node* collapsed, uint32_t* prims, void* workspace, cudaStream_t s) {
    const bool want_obbs = (flags & OBVH_BUILD_OBBS) != 0, want_collapse = (flags & OBVH_BUILD_COLLAPSE) != 0;
    if (want_obbs && (!obbs || !xfs)) return "obvh_build_atrbvh: OBVH_BUILD_OBBS needs obbs and transforms";
    if (want_collapse && (!collapsed || !prims))
        return "obvh_build_atrbvh: OBVH_BUILD_COLLAPSE needs collapsed and primitives";
    // With a transform or a collapse to follow, the refit, the subtree
    // summaries and the collapse marks are one walk (obbtree::enqueue_walk).
    const bool walk = want_obbs || want_collapse;
    OBVH_TRY(enqueue_tree(verts, faces, n, tau, iterations, ci, ct, nodes, parents, counts, costs, scene_out,
                          workspace, s, !walk));
    if (!walk) return kr_success;
    char* ws = static_cast<char*>(workspace);
    const Layout L = layout(n);
    uint8_t* cflags = want_collapse ? collapse::flags_of(ws + L.col_ws, n) : nullptr;
    if (want_collapse) OBVH_TRY_CUDA(cudaMemsetAsync(cflags, 0, 2ull * n - 1, s));
    OBVH_TRY(obbtree::enqueue_walk(nodes, parents, verts, faces, n, counts, costs, obbs, xfs,
                                   want_obbs ? ws + L.obb_ws : nullptr, want_collapse ? collapsed : nullptr, cflags, ci,
                                   ct, collapse::visits_of(ws + L.col_ws, n), &reinterpret_cast<Ctl*>(ws + L.ctl)->error,
                                   s));
    if (want_obbs) OBVH_TRY(obbtree::enqueue_ranks_frames(nodes, parents, counts, verts, faces, obbs, xfs, n, ws + L.obb_ws, s));
    if (want_collapse) {
        // with the transform's depth-first ranks at hand, the gather reads rank runs
        OBVH_TRY(collapse::enqueue_gather(nodes, parents, collapsed, counts, prims, n, ws + L.col_ws, s,
                                          want_obbs ? obbtree::dfs_first(ws + L.obb_ws, n) : nullptr,
                                          want_obbs ? obbtree::dfs_prims(ws + L.obb_ws, n) : nullptr));
    }
    return kr_success;
}

kr_error status(const void* workspace, uint32_t n, cudaStream_t s, uint32_t* device_error, uint32_t* slots) {
    const char* ws = static_cast<const char*>(workspace);
    const Layout L = layout(n);
    uint32_t e[2] = {0, 0};
    uint32_t col[2] = {0, 0};  // collapse error word, primitive slots
    OBVH_TRY_CUDA(cudaMemcpyAsync(&e[0], ws + L.ctl, 4, cudaMemcpyDeviceToHost, s));
    OBVH_TRY_CUDA(cudaMemcpyAsync(&e[1], ws + L.obb_ws, 4, cudaMemcpyDeviceToHost, s));  // transform error word
    OBVH_TRY_CUDA(cudaMemcpyAsync(col, ws + L.col_ws, 8, cudaMemcpyDeviceToHost, s));
    OBVH_TRY_CUDA(cudaStreamSynchronize(s));
    if (device_error) *device_error = e[0] | e[1] | col[0];
    if (slots) *slots = col[1];
    return kr_success;
}

}  // namespace atrbvh
}  // namespace obvh

namespace {
kr_error fail(kr_error e) {
    obvh::set_last_error(e);
    return e;
}
}  // namespace

extern "C" kr_size obvh_atrbvh_workspace_bytes(kr_u32 face_count) {
    return obvh::atrbvh::layout(face_count).total;
}

extern "C" kr_error obvh_atrbvh_workspace_init(void* d_workspace, kr_u32 face_count, void* stream) {
    if (!d_workspace) return fail("obvh_atrbvh_workspace_init: null workspace");
    cudaError_t e = cudaMemsetAsync(d_workspace, 0, obvh::atrbvh::layout(face_count).total,
                                    static_cast<cudaStream_t>(stream));
    return e != cudaSuccess ? fail(obvh::cuda_error(e)) : kr_success;
}

extern "C" kr_error obvh_atrbvh_build_async(const kr_vec3* d_vertices, const kr_uvec4* d_faces, kr_u32 face_count,
                                            kr_u32 treelet_size, kr_u32 iterations, kr_scalar ci, kr_scalar ct,
                                            kr_bvh_node* d_nodes, kr_u32* d_parents, kr_u32* d_primitive_counts,
                                            kr_scalar* d_costs, kr_aabb3* d_scene, void* d_workspace,
                                            void* stream) {
    kr_error e = obvh::atrbvh::enqueue_tree(d_vertices, d_faces, face_count, treelet_size, iterations, ci, ct, d_nodes,
                                            d_parents, d_primitive_counts, d_costs, d_scene, d_workspace,
                                            static_cast<cudaStream_t>(stream));
    return e ? fail(e) : kr_success;
}

extern "C" kr_error obvh_build_atrbvh_async(const kr_vec3* d_vertices, const kr_uvec4* d_faces, kr_u32 face_count,
                                            kr_u32 flags, kr_u32 treelet_size, kr_u32 iterations, kr_scalar ci,
                                            kr_scalar ct, kr_bvh_node* d_nodes, kr_u32* d_parents,
                                            kr_u32* d_primitive_counts, kr_scalar* d_costs, kr_aabb3* d_scene,
                                            kr_obb3* d_obbs, kr_mat4* d_transforms, kr_bvh_node* d_collapsed,
                                            kr_u32* d_primitives, void* d_workspace, void* stream) {
    kr_error e = obvh::atrbvh::enqueue_full(d_vertices, d_faces, face_count, flags, treelet_size, iterations, ci, ct,
                                            d_nodes, d_parents, d_primitive_counts, d_costs, d_scene, d_obbs,
                                            d_transforms, d_collapsed, d_primitives, d_workspace,
                                            static_cast<cudaStream_t>(stream));
    return e ? fail(e) : kr_success;
}

extern "C" kr_error obvh_build_atrbvh_graph_create(const kr_vec3* d_vertices, const kr_uvec4* d_faces,
                                                   kr_u32 face_count, kr_u32 flags, kr_u32 treelet_size,
                                                   kr_u32 iterations, kr_scalar ci, kr_scalar ct,
                                                   kr_bvh_node* d_nodes, kr_u32* d_parents,
                                                   kr_u32* d_primitive_counts, kr_scalar* d_costs,
                                                   kr_aabb3* d_scene, kr_obb3* d_obbs, kr_mat4* d_transforms,
                                                   kr_bvh_node* d_collapsed, kr_u32* d_primitives,
                                                   void* d_workspace, obvh_build_graph* out) {
    const kr_error e = obvh::create_build_graph(
        [&](cudaStream_t s) {
            return obvh::atrbvh::enqueue_full(d_vertices, d_faces, face_count, flags, treelet_size, iterations, ci,
                                              ct, d_nodes, d_parents, d_primitive_counts, d_costs, d_scene, d_obbs,
                                              d_transforms, d_collapsed, d_primitives, d_workspace, s);
        },
        out);
    return e ? fail(e) : kr_success;
}

extern "C" kr_error obvh_atrbvh_status(const void* d_workspace, kr_u32 face_count, void* stream, kr_u32* device_error,
                                       kr_u32* primitive_slots) {
    if (!d_workspace) return fail("obvh_atrbvh_status: null workspace");
    kr_error e = obvh::atrbvh::status(d_workspace, face_count, static_cast<cudaStream_t>(stream), device_error,
                                      primitive_slots);
    return e ? fail(e) : kr_success;
}
