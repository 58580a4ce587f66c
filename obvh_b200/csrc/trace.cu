// trace.cu - closest-hit ray traversal of the SoA OBVH (the layout pack.cu
// writes): kr_cuda_soa_obvh_intersect (soa_obvh_persistent_intersect,
// src/ads/common/cuda/intersectors.cu:801-974, launched at :1452-1473), and
// of the compressed SoA OBVH: kr_cuda_obvh_compressed_persistent_intersect
// (soa_obvh_compressed_persistent_intersect, :975-1144, launched at
// :1146-1172), the same kernel with another node test.
//
// Each ray follows exactly the reference's per-ray sequence, so results are
// bit-identical: at an internal node both children's 4x3 transforms map the
// ray into the unit cube's frame, the nearer hit child is taken first (ties
// to the left) and the farther pushed; the triangles of a leaf are tested in
// its order when the descent reaches it, and a hit replaces the closest one
// only if strictly nearer; then the next node is popped (the reference pops it
// first, which changes nothing).
// The reference's warp ballots only decide when a warp leaves its loops, so
// the scheduling is free, and what sets the time is how many lanes of a warp
// step together: lane by lane, a warp of incoherent rays ran 7.7 of 32 lanes
// wide.  Here a warp visits nodes only while most of its lanes stand at one
// (25 lanes wide), tests the triangles of all waiting lanes as one dealt-out
// batch, and finished lanes take new rays together.  2,000,003 probe rays into
// the 2M-triangle soup: 6.62 -> 4.75 ms, now waiting for node rows (58 of 100
// sectors miss L1); 1920 x 1080 camera rays into the 917K-triangle knot: 1.15
// -> 0.38 ms; the same with an infinite tmax.  The 64-entry stack lives in local
// memory as in the reference.  Indices are checked: a node, leaf, primitive
// slot or face outside its array, or a stack deeper than 64, stops that ray
// with its miss record and sets the error word.
#include <cuda_runtime.h>

#include <cfloat>
#include <cstdint>
#include <mutex>

#include "device_common.cuh"
#include "obvh_transforms.h"
#include "runtime.h"

namespace obvh {
namespace trace {

// 32 warps an SM at 61 registers, no spills.  More warps do not help: the
// probe rays wait for node rows from L2, and 36 warps (56 registers, spills)
// or 24 (68) ran as fast within 1%.
constexpr int kThreads = 512;
constexpr int kBlocksPerSm = 2;
constexpr int kStack = 64;
constexpr int32_t kSentinel = 0x76543210;
constexpr uint32_t kErrIndex = 1u;
constexpr uint32_t kErrStack = 2u;

struct V3 {
    float x, y, z;
};
__device__ __forceinline__ V3 v3(float x, float y, float z) { return V3{x, y, z}; }
__device__ __forceinline__ float kmin(float a, float b) { return (a < b) ? a : b; }  // kr_min
__device__ __forceinline__ float kmax(float a, float b) { return (a < b) ? b : a; }  // kr_max
__device__ __forceinline__ V3 sub(V3 a, V3 b) { return v3(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 cross(V3 a, V3 b) {
    return v3(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

// A 4x3 matrix as loaded: m[0..11] = (c0.xyz, c1.xyz, c2.xyz, c3.xyz).
struct M43 {
    float m[12];
};
__device__ __forceinline__ M43 load_m43(const kr_mat43* p) {
    const float4* q = reinterpret_cast<const float4*>(p);
    const float4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
    return M43{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w}};
}

// A child's ray: the direction and origin in the frame where its box is the
// unit cube.
struct BoxRay {
    V3 d, o;
};

// (t0, t1) of the ray against the unit cube [-0.5, 0.5]^3; (1, -1) on a miss
// (kr_ray_unit_aabb_intersect).
__device__ __forceinline__ float2 unit_slabs(const BoxRay& r) {
    const V3 rd = r.d, ro = r.o;
    const float nx = (-0.5f - ro.x) / rd.x, ny = (-0.5f - ro.y) / rd.y, nz = (-0.5f - ro.z) / rd.z;
    const float fx = (0.5f - ro.x) / rd.x, fy = (0.5f - ro.y) / rd.y, fz = (0.5f - ro.z) / rd.z;
    const float t0 = kmax(kmax(kmin(nx, fx), kmin(ny, fy)), kmin(nz, fz));
    const float t1 = kmin(kmin(kmax(nx, fx), kmax(ny, fy)), kmax(nz, fz));
    if (!(t0 <= t1 && t1 > 0.0f)) return make_float2(1.0f, -1.0f);
    return make_float2(t0, t1);
}

// The same (t0, t1), each within kSlabError of its size, before the hit test:
// every quotient is the numerator times the hardware's reciprocal (at most
// 2^-23 off, the product 2^-24, the exact quotient's own rounding 2^-24), and
// min and max keep a relative bound.  A NaN reaches t0 and t1.  False where a
// reciprocal is outside [2^-59, 2^59]: the bound needs products that neither
// over- nor underflow (a numerator is zero or at least 2^-25).
constexpr float kSlabError = 0x1p-20f;
__device__ __forceinline__ bool near_slabs(const BoxRay& r, float& t0, float& t1) {
    float yx, yy, yz;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yx) : "f"(r.d.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yy) : "f"(r.d.y));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(yz) : "f"(r.d.z));
    const float nx = (-0.5f - r.o.x) * yx, ny = (-0.5f - r.o.y) * yy, nz = (-0.5f - r.o.z) * yz;
    const float fx = (0.5f - r.o.x) * yx, fy = (0.5f - r.o.y) * yy, fz = (0.5f - r.o.z) * yz;
    asm("{\n\t.reg .f32 x, y, z;\n\tmin.NaN.f32 x, %1, %4;\n\tmin.NaN.f32 y, %2, %5;\n\tmin.NaN.f32 z, %3, %6;\n\t"
        "max.NaN.f32 %0, x, y, z;\n\t}"
        : "=f"(t0) : "f"(nx), "f"(ny), "f"(nz), "f"(fx), "f"(fy), "f"(fz));
    asm("{\n\t.reg .f32 x, y, z;\n\tmax.NaN.f32 x, %1, %4;\n\tmax.NaN.f32 y, %2, %5;\n\tmax.NaN.f32 z, %3, %6;\n\t"
        "min.NaN.f32 %0, x, y, z;\n\t}"
        : "=f"(t1) : "f"(nx), "f"(ny), "f"(nz), "f"(fx), "f"(fy), "f"(fz));
    return min3f(fabsf(yx), fabsf(yy), fabsf(yz)) > 0x1p-59f && max3f(fabsf(yx), fabsf(yy), fabsf(yz)) < 0x1p59f;
}

// Whether a < b (and a <= b) is decided although both may be off by
// kSlabError of their size; false for a NaN or an infinity.
__device__ __forceinline__ bool apart(float a, float b) {
    return fabsf(a - b) > kSlabError * (fabsf(a) + fabsf(b));
}

// The ray in the frame of `l` (kr_n43transform3p / kr_v43transform3p).
__device__ __forceinline__ BoxRay into_box(const M43& l, V3 d, V3 o) {
    const float* m = l.m;
    return BoxRay{v3(m[0] * d.x + m[3] * d.y + m[6] * d.z, m[1] * d.x + m[4] * d.y + m[7] * d.z,
                     m[2] * d.x + m[5] * d.y + m[8] * d.z),
                  v3(m[0] * o.x + m[3] * o.y + m[6] * o.z + m[9], m[1] * o.x + m[4] * o.y + m[7] * o.z + m[10],
                     m[2] * o.x + m[5] * o.y + m[8] * o.z + m[11])};
}

// kr_vrotate_angle_axis3 (vecmath.h:1178-1189): Rodrigues' formula, with the
// reference's cos/sin of a float (cosf, sinf) and its order of operations.
__device__ __forceinline__ V3 rotate_angle_axis(V3 v, V3 axis, float radians) {
    const float c = cosf(radians), s = sinf(radians);
    const float d = dot(axis, v);
    const V3 x = cross(axis, v);
    return v3(c * v.x + s * x.x + (1.0f - c) * d * axis.x, c * v.y + s * x.y + (1.0f - c) * d * axis.y,
              c * v.z + s * x.z + (1.0f - c) * d * axis.z);
}

// A child of the compressed SoA OBVH (intersectors.cu:1047-1071): the axis
// and angle dequantised from the metadata word (byte / 127, the angle times
// the reference's float pi), the ray rotated, offset by `min` and scaled by
// `max`.
__device__ __forceinline__ BoxRay into_quant_box(const kr_aabb3* box, int32_t word, V3 d, V3 o) {
    const float* b = reinterpret_cast<const float*>(box);
    const V3 lo = v3(__ldg(b), __ldg(b + 1), __ldg(b + 2)), sc = v3(__ldg(b + 3), __ldg(b + 4), __ldg(b + 5));
    const uint32_t w = static_cast<uint32_t>(word);
    const V3 axis = v3(static_cast<float>(static_cast<int8_t>(w >> 24)) / 127.0f,
                       static_cast<float>(static_cast<int8_t>(w >> 16)) / 127.0f,
                       static_cast<float>(static_cast<int8_t>(w >> 8)) / 127.0f);
    const float angle = (static_cast<float>(static_cast<int8_t>(w)) / 127.0f) * static_cast<float>(3.14159265359);
    const V3 rd0 = rotate_angle_axis(d, axis, angle);
    const V3 ro0 = rotate_angle_axis(sub(o, lo), axis, angle);
    return BoxRay{v3(rd0.x * sc.x, rd0.y * sc.y, rd0.z * sc.z), v3(ro0.x * sc.x, ro0.y * sc.y, ro0.z * sc.z)};
}

// Node tests of the two layouts: the ray in both children's frames at internal
// node i (m: its metadata).
struct SoaBoxes {
    const kr_mat43* __restrict__ left_t;
    const kr_mat43* __restrict__ right_t;
    __device__ __forceinline__ void rays(int32_t i, const int4& m, V3 d, V3 o, BoxRay& l, BoxRay& r) const {
        const M43 lm = load_m43(left_t + i), rm = load_m43(right_t + i);
        l = into_box(lm, d, o);
        r = into_box(rm, d, o);
    }
};

struct QuantBoxes {
    const kr_aabb3* __restrict__ lbounds;
    const kr_aabb3* __restrict__ rbounds;
    __device__ __forceinline__ void rays(int32_t i, const int4& m, V3 d, V3 o, BoxRay& l, BoxRay& r) const {
        l = into_quant_box(lbounds + i, m.z, d, o);
        r = into_quant_box(rbounds + i, m.w, d, o);
    }
};

__device__ __forceinline__ V3 vertex(const kr_vec3* v, uint32_t i) {
    const float* p = reinterpret_cast<const float*>(v) + 3ull * i;
    return v3(__ldg(p), __ldg(p + 1), __ldg(p + 2));
}

// Per-ray traversal state: everything one ray carries between steps.
struct RayState {
    V3 o, d;
    float hit_t, b1, b2;
    uint32_t hit, fail;
    int32_t cur;  // the node to visit next: >= 0 internal, < 0 a leaf (~index), kSentinel when the ray is done
    int sp;
};

// The reference's record for a finished ray: the miss record, or the hit
// triangle's unit normal, barycentrics and index.
__device__ __forceinline__ void finish(const RayState& st, const kr_vec3* verts, const kr_uvec4* faces,
                                       kr_intersection* out, uint32_t* err) {
    uint32_t hit = st.hit;
    if (st.fail) {
        atomicOr(err, st.fail);
        hit = 0xFFFFFFFFu;
    }
    kr_intersection rec;
    if (hit == 0xFFFFFFFFu) {
        rec.geom_normal = kr_vec3{{st.d.x, st.d.y, st.d.z}};
        rec.barys = kr_vec2{{0.5f, 0.5f}};
    } else {
        const uint4 f = __ldg(reinterpret_cast<const uint4*>(faces + hit));
        const V3 va = vertex(verts, f.x), vb = vertex(verts, f.y), vc = vertex(verts, f.z);
        const V3 n = cross(sub(vb, va), sub(vc, va));
        const float len = sqrtf(dot(n, n));
        rec.geom_normal = kr_vec3{{n.x / len, n.y / len, n.z / len}};
        rec.barys = kr_vec2{{st.b1, st.b2}};
    }
    rec.primitive = hit;
    rec.instance = 0;
    *out = rec;
}

// One visit of an internal node: the nearer hit child next (ties to the
// left), the farther pushed; neither hit: the next node of the stack.  Only
// the outcome of the comparisons matters, so the slabs come from near_slabs
// (3 reciprocals and 6 products a child instead of 6 IEEE divisions) and the
// divisions are made where a comparison lies inside the error bound.
template <class Boxes>
__device__ __forceinline__ void visit_node(const Boxes& boxes, const kr_ivec4* __restrict__ meta,
                                           uint32_t internal_count, RayState& st, int32_t* stack) {
    if (static_cast<uint32_t>(st.cur) >= internal_count) {
        st.fail = kErrIndex;
        st.cur = kSentinel;
        return;
    }
    const int4 m = __ldg(reinterpret_cast<const int4*>(meta + st.cur));
    BoxRay l, r;
    boxes.rays(st.cur, m, st.d, st.o, l, r);
    float l0, l1, r0, r1;
    const bool sl = near_slabs(l, l0, l1), sr = near_slabs(r, r0, r1);
    bool tl = l0 <= l1 && l1 > 0.0f && l0 <= st.hit_t;
    bool tr = r0 <= r1 && r1 > 0.0f && r0 <= st.hit_t;
    // Of an infinite limit (a ray's that has none) apart() decides nothing, so
    // FLT_MAX stands in: it compares with a finite distance alike, and
    // apart(l0, l1) lets no other pass.
    const float limit = fminf(st.hit_t, FLT_MAX);
    const bool sure_l = sl && apart(l0, l1) && apart(l0, limit);
    const bool sure_r = sr && apart(r0, r1) && apart(r0, limit);
    const bool close = (tl || !sure_l) && (tr || !sure_r) && !apart(l0, r0);
    bool exact_l = !sure_l || close, exact_r = !sure_r || close;
    if (exact_l || exact_r) {
        // which child is nearer needs both distances with the bound, or both exact
        if (sl != sr) exact_l = exact_r = true;
        do {
            const float2 e = unit_slabs(exact_l ? l : r);
            const bool hit = e.y >= e.x && e.y >= 0.0f && e.x <= st.hit_t;
            if (exact_l) {
                tl = hit;
                l0 = e.x;
                exact_l = false;
            } else {
                tr = hit;
                r0 = e.x;
                exact_r = false;
            }
        } while (exact_l || exact_r);
    }
    const bool swap = r0 < l0;
    if (tl && tr) {
        if (st.sp + 1 >= kStack) {
            st.fail = kErrStack;
            st.cur = kSentinel;
            return;
        }
        stack[++st.sp] = swap ? m.x : m.y;
        st.cur = swap ? m.y : m.x;
    } else if (tl || tr) {
        st.cur = tl ? m.x : m.y;
    } else {
        st.cur = stack[st.sp--];
    }
}

// t of the ray against one triangle, with its barycentrics; +inf on a miss
// (kr_ray_triangle_intersect; its test against the closest hit so far is the
// caller's strict t < hit_t).
__device__ __forceinline__ float test_triangle(const kr_vec3* __restrict__ verts, uint4 f, V3 o, V3 d, float& c1,
                                               float& c2) {
    const V3 p1 = vertex(verts, f.x), p2 = vertex(verts, f.y), p3 = vertex(verts, f.z);
    const V3 e1 = sub(p2, p1), e2 = sub(p3, p1);
    const V3 s1 = cross(d, e2);
    const float invd = 1.0f / dot(s1, e1);
    const V3 dd = sub(o, p1);
    c1 = dot(dd, s1) * invd;
    const V3 s2 = cross(dd, e1);
    c2 = dot(d, s2) * invd;
    const float t = dot(e2, s2) * invd;
    const bool miss = c1 < 0.0f || c1 > 1.0f || c2 < 0.0f || c1 + c2 > 1.0f || t < 0.0f;
    return miss ? kInf : t;
}

// The leaves of the lanes that stand at one (st.cur < 0), by the whole warp:
// their triangles are dealt out one to a lane, each tested against its
// owner's ray, and the owner takes the first of the smallest t below its
// closest hit -- what testing them in order with strict t < hit_t keeps.  A
// leaf at a time and lane by lane, a warp ran about 3 lanes wide here, each
// triangle behind its own chain of three loads.  Called by all 32 lanes.
__device__ __forceinline__ void visit_leaves(const kr_ivec4* __restrict__ meta, uint32_t node_count,
                                             const kr_vec3* __restrict__ verts, const kr_uvec4* __restrict__ faces,
                                             uint32_t face_count, const kr_u32* __restrict__ prims,
                                             uint32_t prim_slots, RayState& st, const int32_t* stack) {
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31;
    const bool mine = st.cur < 0;
    int32_t beg = 0;
    uint32_t left = 0;  // triangles of this lane's leaf not yet dealt out
    if (mine) {
        const uint32_t li = static_cast<uint32_t>(~st.cur);
        if (li >= node_count) {
            st.fail = kErrIndex;
        } else {
            const int4 m = __ldg(reinterpret_cast<const int4*>(meta + li));
            beg = m.x;
            left = m.x < m.y ? static_cast<uint32_t>(m.y) - static_cast<uint32_t>(m.x) : 0u;
        }
    }
    const bool single = left == 1;
    for (;;) {
        const uint32_t want = min(left, 32u);
        uint32_t incl = want;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const uint32_t v = __shfl_up_sync(kAll, incl, k);
            if (lane >= static_cast<uint32_t>(k)) incl += v;
        }
        const uint32_t base = incl - want;
        const uint32_t total = min(32u, __shfl_sync(kAll, incl, 31));
        if (total == 0) break;
        const uint32_t take = base < 32u ? min(want, 32u - base) : 0u;
        // item `lane` belongs to the last lane whose base is at most `lane`
        uint32_t owner = 0;
#pragma unroll
        for (int k = 16; k > 0; k >>= 1)
            if (__shfl_sync(kAll, base, owner + k) <= lane) owner += k;
        const uint32_t at = static_cast<uint32_t>(__shfl_sync(kAll, beg, owner)) + (lane - __shfl_sync(kAll, base, owner));
        const bool one = __shfl_sync(kAll, static_cast<int>(single), owner) != 0;
        const V3 o = v3(__shfl_sync(kAll, st.o.x, owner), __shfl_sync(kAll, st.o.y, owner), __shfl_sync(kAll, st.o.z, owner));
        const V3 d = v3(__shfl_sync(kAll, st.d.x, owner), __shfl_sync(kAll, st.d.y, owner), __shfl_sync(kAll, st.d.z, owner));
        bool bad = false;
        float t = kInf, c1 = 0.0f, c2 = 0.0f;
        uint32_t pid = at;
        if (lane < total) {
            if (!one) {
                bad = static_cast<int32_t>(at) < 0 || at >= prim_slots;
                if (!bad) pid = __ldg(prims + at);
            }
            bad = bad || pid >= face_count;
            if (!bad) t = test_triangle(verts, __ldg(reinterpret_cast<const uint4*>(faces + pid)), o, d, c1, c2);
        }
        const unsigned wrong = __ballot_sync(kAll, bad);
        const uint32_t most = __reduce_max_sync(kAll, take);
        uint32_t who = lane;
        bool better = false;
        for (uint32_t j = 0; j < most; ++j) {
            const float tj = __shfl_sync(kAll, t, (base + j) & 31u);
            if (j < take && tj < st.hit_t) {
                st.hit_t = tj;
                who = base + j;
                better = true;
            }
        }
        c1 = __shfl_sync(kAll, c1, who);
        c2 = __shfl_sync(kAll, c2, who);
        pid = __shfl_sync(kAll, pid, who);
        if (better) {
            st.b1 = c1;
            st.b2 = c2;
            st.hit = pid;
        }
        beg += static_cast<int32_t>(take);
        left -= take;
        if (take && ((wrong >> base) & (take < 32u ? (1u << take) - 1u : kAll))) {
            st.fail = kErrIndex;
            left = 0;
        }
    }
    if (mine) st.cur = (!st.fail && st.sp >= 0) ? stack[st.sp--] : kSentinel;
}

// A warp visits nodes while at least kNodeLanes of 32 lanes with a ray stand
// at one; the lanes that meanwhile reached a leaf wait and test their leaves
// together.  Finished lanes wait until kRefillLanes of them write their
// records and take new rays together.  Measured (2,000,003 probe rays / 1920 x
// 1080 camera rays, us): 20 of 32 4,785 / 367, 24 4,750 / 379, 28 4,716 / 402;
// 2, 4 and 8 finished lanes 4,690 / 376, 4,750 / 379 and 4,859 / 378.
constexpr int kNodeLanes = 24;
constexpr int kRefillLanes = 4;

// Persistent blocks: the rays lie in chunks of 32 and block b owns chunks b,
// b + gridDim.x, ..., so that costly parts of the ray array (the object in a
// camera's picture) spread over all blocks; a block's warps take its chunks
// one after the other from a shared counter.  A ray's own steps are those of
// the reference, in the same order; only which lanes step together differs.
template <class Boxes>
__global__ void __launch_bounds__(kThreads, kBlocksPerSm)
trace_kernel(Boxes boxes, const kr_ivec4* __restrict__ meta, uint32_t internal_count, uint32_t node_count,
             const kr_vec3* __restrict__ verts, const kr_uvec4* __restrict__ faces, uint32_t face_count,
             const kr_u32* __restrict__ prims, uint32_t prim_slots, const kr_ray* __restrict__ rays,
             kr_intersection* isects, uint32_t ray_count, uint32_t* err) {
    constexpr unsigned kAll = 0xffffffffu;
    __shared__ uint32_t s_taken;  // chunks of this block taken so far
    if (threadIdx.x == 0) s_taken = 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t chunks = (ray_count >> 5) + ((ray_count & 31u) != 0);
    const uint32_t own = blockIdx.x < chunks ? (chunks - 1 - blockIdx.x) / gridDim.x + 1 : 0u;
    uint32_t next = 0, stop = 0;  // the warp's unassigned rays
    bool more = true;             // the block may have chunks left
    int32_t stack[kStack];
    RayState st;
    st.cur = kSentinel;
    st.fail = 0;
    uint32_t r = 0;
    bool busy = false;  // this lane holds a ray (a finished one until its record is written)
    for (;;) {
        const unsigned done = __ballot_sync(kAll, st.cur == kSentinel);
        if (done == kAll || ((more || next < stop) && __popc(done) >= kRefillLanes)) {
            if (busy && st.cur == kSentinel) {
                finish(st, verts, faces, isects + r, err);
                busy = false;
            }
            for (;;) {
                if (next == stop && more) {
                    uint32_t c = 0;
                    if (lane == 0) c = atomicAdd(&s_taken, 1u);
                    c = __shfl_sync(kAll, c, 0);
                    more = c < own;
                    if (more) {
                        const uint64_t first = (static_cast<uint64_t>(c) * gridDim.x + blockIdx.x) * 32u;
                        next = static_cast<uint32_t>(first);
                        stop = ray_count - next > 32u ? next + 32u : ray_count;
                    }
                }
                const unsigned idle = __ballot_sync(kAll, !busy);
                if (idle == 0 || next == stop) break;
                const uint32_t k = __popc(idle & ((1u << lane) - 1u));
                if (!busy && k < stop - next) {
                    r = next + k;
                    busy = true;
                    const float4* rp = reinterpret_cast<const float4*>(rays + r);
                    const float4 ra = __ldg(rp), rb = __ldg(rp + 1);
                    st.o = v3(ra.x, ra.y, ra.z);
                    st.d = v3(rb.x, rb.y, rb.z);
                    st.hit_t = rb.w;
                    st.hit = 0xFFFFFFFFu;
                    st.b1 = st.b2 = 0.0f;
                    st.fail = 0;
                    st.cur = 0;
                    st.sp = 0;
                    stack[0] = kSentinel;
                }
                next += min(static_cast<uint32_t>(__popc(idle)), stop - next);
            }
            if (!__any_sync(kAll, busy)) break;
        }
        // nodes, while enough of the lanes with a ray stand at one
        const int alive = __popc(__ballot_sync(kAll, st.cur != kSentinel));
        const int enough = max(1, (alive * kNodeLanes) >> 5);
        for (;;) {
            const bool at_node = st.cur >= 0 && st.cur != kSentinel;
            if (__popc(__ballot_sync(kAll, at_node)) < enough) break;
            if (at_node) visit_node(boxes, meta, internal_count, st, stack);
            __syncwarp();
        }
        if (__any_sync(kAll, st.cur < 0))
            visit_leaves(meta, node_count, verts, faces, face_count, prims, prim_slots, st, stack);
    }
}

// Persistent grid: every block resident at once (the occupancy of
// trace_kernel, looked up once per device), and no more blocks than rays
// need.
template <class Boxes>
inline unsigned grid_for(uint32_t n) {
    static int per_sm[64] = {0};
    const DeviceInfo& dev = device_info();
    int& k = per_sm[dev.device & 63];
    if (k == 0 &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, trace_kernel<Boxes>, kThreads, 0) != cudaSuccess) {
        (void)cudaGetLastError();
        k = 8;
    }
    if (k < 1) k = 1;
    const unsigned want = n / 32 + (n % 32 != 0);  // a chunk a block at least
    const unsigned cap = static_cast<unsigned>(dev.sm_count) * static_cast<unsigned>(k);
    return want < cap ? (want ? want : 1u) : cap;
}


bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <class Boxes>
kr_error launch(const Boxes& boxes, const kr_ivec4* meta, uint32_t internal_count, uint32_t node_count,
                const kr_vec3* verts, const kr_uvec4* faces, uint32_t face_count, const kr_u32* prims,
                uint32_t prim_slots, const kr_ray* rays, kr_intersection* isects, uint32_t ray_count, uint32_t* err,
                cudaStream_t s, const char* name) {
    const unsigned g = grid_for<Boxes>(ray_count);
    ProfScope prof_scope_(name, s);
    trace_kernel<Boxes><<<g, kThreads, 0, s>>>(boxes, meta, internal_count, node_count, verts, faces, face_count,
                                               prims, prim_slots, rays, isects, ray_count, err);
    OBVH_TRY_CUDA(cudaGetLastError());
    return kr_success;
}

kr_error check_common(const kr_ivec4* meta, uint32_t internal_count, const kr_vec3* verts, const kr_uvec4* faces,
                      const kr_ray* rays, kr_intersection* isects, uint32_t* err) {
    if (!meta || !verts || !faces || !rays || !isects || !err) return "obvh trace: null pointer argument";
    if (internal_count == 0) return "obvh trace: the tree has no internal node (one primitive) to traverse";
    if (!aligned16(meta) || !aligned16(faces) || !aligned16(rays))
        return "obvh trace: metadata, faces and rays must be 16-byte aligned";
    return kr_success;
}

kr_error enqueue(const kr_mat43* left_t, const kr_mat43* right_t, const kr_ivec4* meta, uint32_t internal_count,
                 uint32_t node_count, const kr_vec3* verts, const kr_uvec4* faces, uint32_t face_count,
                 const kr_u32* prims, uint32_t prim_slots, const kr_ray* rays, kr_intersection* isects,
                 uint32_t ray_count, uint32_t* err, cudaStream_t s) {
    if (ray_count == 0) return kr_success;
    OBVH_TRY(check_common(meta, internal_count, verts, faces, rays, isects, err));
    if (!left_t || !right_t) return "obvh trace: null pointer argument";
    if (!aligned16(left_t) || !aligned16(right_t)) return "obvh trace: SoA arrays must be 16-byte aligned";
    return launch(SoaBoxes{left_t, right_t}, meta, internal_count, node_count, verts, faces, face_count, prims,
                  prim_slots, rays, isects, ray_count, err, s, "trace_kernel");
}

kr_error enqueue_compressed(const kr_aabb3* lbounds, const kr_aabb3* rbounds, const kr_ivec4* meta,
                            uint32_t internal_count, uint32_t node_count, const kr_vec3* verts, const kr_uvec4* faces,
                            uint32_t face_count, const kr_u32* prims, uint32_t prim_slots, const kr_ray* rays,
                            kr_intersection* isects, uint32_t ray_count, uint32_t* err, cudaStream_t s) {
    if (ray_count == 0) return kr_success;
    OBVH_TRY(check_common(meta, internal_count, verts, faces, rays, isects, err));
    if (!lbounds || !rbounds) return "obvh trace: null pointer argument";
    if ((reinterpret_cast<uintptr_t>(lbounds) & 3) || (reinterpret_cast<uintptr_t>(rbounds) & 3))
        return "obvh trace: boxes must be 4-byte aligned";
    return launch(QuantBoxes{lbounds, rbounds}, meta, internal_count, node_count, verts, faces, face_count, prims,
                  prim_slots, rays, isects, ray_count, err, s, "trace_compressed_kernel");
}

// The synchronous entry point's error word: one device word owned by the
// library (allocated on first use, kept until exit), one call at a time.
struct ErrWord {
    std::mutex mu;
    DeviceBuffer buf;
};
ErrWord& err_word() {
    static ErrWord w;
    return w;
}

}  // namespace trace
}  // namespace obvh

using namespace obvh;

extern "C" kr_error kr_cuda_soa_obvh_intersect(const kr_SoA_OBVH* bvh, const kr_vec3* vertices, const kr_uvec4* faces,
                                               const kr_u32* primitives, const kr_ray* rays, kr_intersection* isects,
                                               kr_u32 ray_count, kr_u32 block_size, kr_u32 grid_size,
                                               kr_u32* warp_counter) {
    (void)block_size;
    (void)grid_size;
    (void)warp_counter;
    kr_error e = kr_success;
    if (!bvh) e = "kr_cuda_soa_obvh_intersect: null pointer argument";
    kr_SoA_OBVH h{};
    if (!e) {
        cudaError_t ce = cudaMemcpy(&h, bvh, sizeof h, cudaMemcpyDeviceToHost);
        if (ce != cudaSuccess) e = cuda_error(ce);
    }
    if (!e) {
        // The reference's signature carries no sizes: indices are trusted as
        // the reference trusts them, and the checks only catch negative ones
        // and a stack deeper than 64 (obvh_soa_obvh_intersect_async checks
        // every index against the sizes it is given).
        trace::ErrWord& w = trace::err_word();
        std::lock_guard<std::mutex> lock(w.mu);
        e = w.buf.reserve(256);
        uint32_t* d_err = static_cast<uint32_t*>(w.buf.ptr);
        if (!e) {
            cudaError_t ce = cudaMemsetAsync(d_err, 0, 4, nullptr);
            if (ce != cudaSuccess) e = cuda_error(ce);
        }
        if (!e)
            e = trace::enqueue(h.left_T, h.right_T, h.metadata, 0x7FFFFFFFu, 0x7FFFFFFFu, vertices, faces, 0x7FFFFFFFu,
                               primitives, 0x7FFFFFFFu, rays, isects, ray_count, d_err, nullptr);
        uint32_t flag = 0;
        if (!e) {
            cudaError_t ce = cudaMemcpyAsync(&flag, d_err, 4, cudaMemcpyDeviceToHost, nullptr);
            if (ce == cudaSuccess) ce = cudaStreamSynchronize(nullptr);
            if (ce != cudaSuccess) e = cuda_error(ce);
        }
        if (!e && flag) e = "kr_cuda_soa_obvh_intersect: a traversal index was negative or a stack passed 64 entries";
    }
    if (e) set_last_error(e);
    return e;
}

extern "C" kr_error obvh_soa_obvh_intersect_async(const kr_mat43* d_left_t, const kr_mat43* d_right_t,
                                                  const kr_ivec4* d_metadata, kr_u32 internal_count,
                                                  kr_u32 node_count, const kr_vec3* d_vertices,
                                                  const kr_uvec4* d_faces, kr_u32 face_count,
                                                  const kr_u32* d_primitives, kr_u32 primitive_slots,
                                                  const kr_ray* d_rays, kr_intersection* d_isects, kr_u32 ray_count,
                                                  kr_u32* d_error, void* stream) {
    kr_error e = trace::enqueue(d_left_t, d_right_t, d_metadata, internal_count, node_count, d_vertices, d_faces,
                                face_count, d_primitives, primitive_slots, d_rays, d_isects, ray_count, d_error,
                                static_cast<cudaStream_t>(stream));
    if (e) set_last_error(e);
    return e;
}

extern "C" kr_error kr_cuda_obvh_compressed_persistent_intersect(const kr_SoA_OBVH_Compressed* bvh,
                                                                 const kr_vec3* vertices, const kr_uvec4* faces,
                                                                 const kr_u32* primitives, const kr_ray* rays,
                                                                 kr_intersection* isects, kr_u32 ray_count,
                                                                 kr_u32 block_size, kr_u32 grid_size,
                                                                 kr_u32* warp_counter) {
    (void)block_size;
    (void)grid_size;
    (void)warp_counter;
    kr_error e = kr_success;
    if (!bvh) e = "kr_cuda_obvh_compressed_persistent_intersect: null pointer argument";
    kr_SoA_OBVH_Compressed h{};
    if (!e) {
        cudaError_t ce = cudaMemcpy(&h, bvh, sizeof h, cudaMemcpyDeviceToHost);
        if (ce != cudaSuccess) e = cuda_error(ce);
    }
    if (!e) {
        // no sizes in the reference's signature: indices are trusted (as in
        // kr_cuda_soa_obvh_intersect)
        trace::ErrWord& w = trace::err_word();
        std::lock_guard<std::mutex> lock(w.mu);
        e = w.buf.reserve(256);
        uint32_t* d_err = static_cast<uint32_t*>(w.buf.ptr);
        if (!e) {
            cudaError_t ce = cudaMemsetAsync(d_err, 0, 4, nullptr);
            if (ce != cudaSuccess) e = cuda_error(ce);
        }
        if (!e)
            e = trace::enqueue_compressed(h.lbounds, h.rbounds, h.metadata, 0x7FFFFFFFu, 0x7FFFFFFFu, vertices, faces,
                                          0x7FFFFFFFu, primitives, 0x7FFFFFFFu, rays, isects, ray_count, d_err,
                                          nullptr);
        uint32_t flag = 0;
        if (!e) {
            cudaError_t ce = cudaMemcpyAsync(&flag, d_err, 4, cudaMemcpyDeviceToHost, nullptr);
            if (ce == cudaSuccess) ce = cudaStreamSynchronize(nullptr);
            if (ce != cudaSuccess) e = cuda_error(ce);
        }
        if (!e && flag)
            e = "kr_cuda_obvh_compressed_persistent_intersect: a traversal index was negative or a stack passed 64 "
                "entries";
    }
    if (e) set_last_error(e);
    return e;
}

extern "C" kr_error obvh_soa_compressed_obvh_intersect_async(const kr_aabb3* d_lbounds, const kr_aabb3* d_rbounds,
                                                             const kr_ivec4* d_metadata, kr_u32 internal_count,
                                                             kr_u32 node_count, const kr_vec3* d_vertices,
                                                             const kr_uvec4* d_faces, kr_u32 face_count,
                                                             const kr_u32* d_primitives, kr_u32 primitive_slots,
                                                             const kr_ray* d_rays, kr_intersection* d_isects,
                                                             kr_u32 ray_count, kr_u32* d_error, void* stream) {
    kr_error e = trace::enqueue_compressed(d_lbounds, d_rbounds, d_metadata, internal_count, node_count, d_vertices,
                                           d_faces, face_count, d_primitives, primitive_slots, d_rays, d_isects,
                                           ray_count, d_error, static_cast<cudaStream_t>(stream));
    if (e) set_last_error(e);
    return e;
}
