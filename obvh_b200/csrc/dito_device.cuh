// dito_device.cuh - the per-set pieces of a DiTO-14 fit that run once per
// point set rather than once per point: the candidate-axis search over the
// 14 extremal points and the final box assembly.  Shared by the single-fit
// kernels (dito.cu) and the batched kernels (dito_batch.cu).
#pragma once

#include <cfloat>
#include <cstdint>

#include "device_common.cuh"
#include "obvh_dito.h"

namespace obvh {
namespace dito {

// Control block at the start of a fit's workspace (256 bytes).
struct Ctl {
    uint32_t ticket[2];  // CTAs finished in pass 1 / pass 2; reset by the last one
    uint32_t error;      // kErr* flags
    uint32_t path;       // 0 empty, 1 degenerate pair, 2 degenerate line, 3 OBB, 4 AABB kept
    uint32_t plan;       // 0 box final after pass 1; 1 pass 2 + final test; 2 pass 2, no test
    uint32_t flags;
    uint32_t pad[2];
    float axes[9];
    float al_mid[3];
    float al_len[3];
    float al_val;
    uint32_t pad2[40];
};
static_assert(sizeof(Ctl) == 256, "control block is 256 bytes");

// Workspace layout (device): the control block, an output slot used by the
// host-pointer entry points, then the per-CTA records of both passes.
constexpr int kMaxGrid = 1024;
constexpr size_t kOffObb = 256;                                   // host-API output slot
constexpr size_t kOffRec1Val = 512;                               // [kMaxGrid][14] float
constexpr size_t kOffRec1Idx = kOffRec1Val + kMaxGrid * 14 * 4;   // [kMaxGrid][14] u64
constexpr size_t kOffRec2 = kOffRec1Idx + kMaxGrid * 14 * 8;      // [kMaxGrid][6] float
constexpr size_t kWorkspaceBytes = kOffRec2 + kMaxGrid * 6 * 4;

// Slab projection k of the 7 fixed DiTO directions, in the reference's
// evaluation order (dito.cpp:115-172); k is a compile-time constant after unrolling.
__device__ __forceinline__ float slab(int k, float x, float y, float z) {
    switch (k) {
        case 0: return x;
        case 1: return y;
        case 2: return z;
        case 3: return x + y + z;
        case 4: return x + y - z;
        case 5: return x - y + z;
        default: return x - y - z;
    }
}

// Per-thread running extremes.  For each direction the thread keeps the
// extreme value and the CTA-local index of the first point of the first
// 4-point group reaching it (groups are visited in increasing index order and
// replaced only on strict improvement).  The hot loop is branch-free; the
// exact point inside a winning group is resolved once per CTA.
struct Extremes {
    float mn[7], mx[7];
    uint32_t gmn[7], gmx[7];
    __device__ void init() {
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            mn[k] = kInf;
            mx[k] = -kInf;
            gmn[k] = 0xffffffffu;
            gmx[k] = 0xffffffffu;
        }
    }
    // the 4 points x/y/z[0..4) with indices g, g+1, g+2, g+3
    __device__ __forceinline__ void group(const float* x, const float* y, const float* z, uint32_t g) {
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            float v0 = slab(k, x[0], y[0], z[0]), v1 = slab(k, x[1], y[1], z[1]);
            float v2 = slab(k, x[2], y[2], z[2]), v3 = slab(k, x[3], y[3], z[3]);
            float lo = min3f(v0, v1, fminf(v2, v3));
            float hi = max3f(v0, v1, fmaxf(v2, v3));
            bool a = lo < mn[k];
            mn[k] = a ? lo : mn[k];
            gmn[k] = a ? g : gmn[k];
            bool b = hi > mx[k];
            mx[k] = b ? hi : mx[k];
            gmx[k] = b ? g : gmx[k];
        }
    }
};

// Extents along three axes (values only).
struct Extents {
    f3 b0, b1, b2;
    float lo[3], hi[3];
    __device__ void init(const float* axes) {
        b0 = mk3(axes[0], axes[1], axes[2]);
        b1 = mk3(axes[3], axes[4], axes[5]);
        b2 = mk3(axes[6], axes[7], axes[8]);
#pragma unroll
        for (int k = 0; k < 3; ++k) { lo[k] = kInf; hi[k] = -kInf; }
    }
    __device__ __forceinline__ void point(float x, float y, float z) {
        f3 p = mk3(x, y, z);
        float q0 = dot3(p, b0), q1 = dot3(p, b1), q2 = dot3(p, b2);
        lo[0] = fminf(lo[0], q0); hi[0] = fmaxf(hi[0], q0);
        lo[1] = fminf(lo[1], q1); hi[1] = fmaxf(hi[1], q1);
        lo[2] = fminf(lo[2], q2); hi[2] = fmaxf(hi[2], q2);
    }
};

// Unpacks 4-point groups (3 float4 each) into coordinate arrays.
__device__ __forceinline__ void unpack4(const float4& a, const float4& b, const float4& c, float* x, float* y,
                                        float* z) {
    x[0] = a.x; y[0] = a.y; z[0] = a.z;
    x[1] = a.w; y[1] = b.x; z[1] = b.y;
    x[2] = b.z; y[2] = b.w; z[2] = c.x;
    x[3] = c.y; y[3] = c.z; z[3] = c.w;
}

// ---------------------------------------------------------------------------
// A set of fewer than 2^32 points read straight from global memory (the batched
// and the one-launch fits).
constexpr uint32_t kNoIndex = 0xffffffffu;

// One set: its points, and the split into an unaligned head (< 4 points), a
// body of 16-byte-aligned 4-point groups and a tail.
struct SetView {
    const float* base;
    uint32_t n, head, groups;
    __device__ uint32_t tail0() const { return head + 4 * groups; }
};

__device__ __forceinline__ SetView view_of(const float* base, uint32_t n) {
    SetView v;
    v.base = base;
    v.n = n;
    // A point is 12 bytes: base misaligned by 4*m bytes becomes aligned after m points.
    const uint32_t m = static_cast<uint32_t>((reinterpret_cast<uintptr_t>(v.base) & 15u) >> 2);
    v.head = m < v.n ? m : v.n;
    v.groups = (v.n - v.head) / 4;
    return v;
}

__device__ __forceinline__ void load_group(const SetView& v, uint32_t g, float* x, float* y, float* z) {
    const float4* q = reinterpret_cast<const float4*>(v.base + 3 * (v.head + 4ull * g));
    unpack4(q[0], q[1], q[2], x, y, z);
}

// Groups g0 + t, g0 + t + stride, ... below g1, in increasing order, U at a
// time (U groups' loads issued before any is used).
template <int U>
__device__ __forceinline__ void scan_extremes(const SetView& v, uint32_t g0, uint32_t g1, uint32_t t,
                                              uint32_t stride, Extremes& ex) {
    uint32_t g = g0 + t;
    for (; g + (U - 1) * stride < g1; g += U * stride) {
        float x[4 * U], y[4 * U], z[4 * U];
#pragma unroll
        for (int u = 0; u < U; ++u) load_group(v, g + u * stride, x + 4 * u, y + 4 * u, z + 4 * u);
#pragma unroll
        for (int u = 0; u < U; ++u) ex.group(x + 4 * u, y + 4 * u, z + 4 * u, 4 * (g + u * stride));
    }
    for (; g < g1; g += stride) {
        float x[4], y[4], z[4];
        load_group(v, g, x, y, z);
        ex.group(x, y, z, 4 * g);
    }
}

template <int U>
__device__ __forceinline__ void scan_extents(const SetView& v, uint32_t g0, uint32_t g1, uint32_t t, uint32_t stride,
                                             Extents& ex) {
    uint32_t g = g0 + t;
    for (; g + (U - 1) * stride < g1; g += U * stride) {
        float x[4 * U], y[4 * U], z[4 * U];
#pragma unroll
        for (int u = 0; u < U; ++u) load_group(v, g + u * stride, x + 4 * u, y + 4 * u, z + 4 * u);
#pragma unroll
        for (int j = 0; j < 4 * U; ++j) ex.point(x[j], y[j], z[j]);
    }
    for (; g < g1; g += stride) {
        float x[4], y[4], z[4];
        load_group(v, g, x, y, z);
#pragma unroll
        for (int j = 0; j < 4; ++j) ex.point(x[j], y[j], z[j]);
    }
}

// Extreme e (0..6 min of slab e, 7..13 max of slab e-7): from the first
// 4-point group reaching `val` (body offset r of its first point) to the first
// point reaching it, then merged with the head points (which precede the
// body) and the tail points (which follow it) when asked.
inline __device__ uint32_t resolve(const SetView& v, int e, float& val, uint32_t r, bool with_head, bool with_tail) {
    const int k = e < 7 ? e : e - 7;
    const bool is_min = e < 7;
    uint64_t best = ~0ull;
    if (r != kNoIndex) {
        for (int j = 3; j >= 0; --j) {
            const float* q = v.base + 3 * (static_cast<uint64_t>(v.head) + r + j);
            if (slab(k, q[0], q[1], q[2]) == val) best = v.head + r + j;
        }
    }
    auto merge = [&](uint32_t i) {
        const float* q = v.base + 3 * static_cast<uint64_t>(i);
        const float s = slab(k, q[0], q[1], q[2]);
        const bool b = is_min ? better_min(s, i, val, best) : better_max(s, i, val, best);
        if (b) {
            val = s;
            best = i;
        }
    };
    if (with_head)
        for (uint32_t i = 0; i < v.head; ++i) merge(i);
    if (with_tail)
        for (uint32_t i = v.tail0(); i < v.n; ++i) merge(i);
    return best == ~0ull ? kNoIndex : static_cast<uint32_t>(best);
}

struct Mode {
    bool gpu;  // OBVH_DITO_REFERENCE_GPU semantics
    // dito.cpp:98-103 multiplies by the reciprocal length; kr_vnormalize3
    // (vecmath.h:548-549) divides by the length.
    __device__ __forceinline__ f3 unit(f3 a) const {
        float l = sqrtf(len2_3(a));
        if (gpu) return mk3(a.x / l, a.y / l, a.z / l);
        float inv = 1.0f / l;
        return mk3(a.x * inv, a.y * inv, a.z * inv);
    }
    // dito.cpp:83-87 forms y as -(ax*bz - az*bx); kr_vcross3 (vecmath.h:812-814)
    // as az*bx - ax*bz.  Same value, different sign of a zero.
    __device__ __forceinline__ f3 cross(f3 a, f3 b) const {
        float y = gpu ? (a.z * b.x - a.x * b.z) : -(a.x * b.z - a.z * b.x);
        return mk3(a.y * b.z - a.z * b.y, y, a.x * b.y - a.y * b.x);
    }
};

__device__ __forceinline__ void store_obb(kr_obb3* out, f3 mid, f3 b0, f3 b1, f3 b2, f3 ext, bool clamp) {
    if (clamp) {
        // kr_points_obb: ext = kr_vmax3(ext, 0.001) with kr_max(a,b) = (a < b) ? b : a
        ext.x = (ext.x < 0.001f) ? 0.001f : ext.x;
        ext.y = (ext.y < 0.001f) ? 0.001f : ext.y;
        ext.z = (ext.z < 0.001f) ? 0.001f : ext.z;
    }
    float* o = reinterpret_cast<float*>(out);
    o[0] = mid.x; o[1] = mid.y; o[2] = mid.z;
    o[3] = b0.x; o[4] = b0.y; o[5] = b0.z;
    o[6] = b1.x; o[7] = b1.y; o[8] = b1.z;
    o[9] = b2.x; o[10] = b2.y; o[11] = b2.z;
    o[12] = ext.x; o[13] = ext.y; o[14] = ext.z;
}

// dito.cpp:442-449
__device__ __forceinline__ void store_aabb(kr_obb3* out, f3 mid, f3 len, bool clamp) {
    store_obb(out, mid, mk3(1, 0, 0), mk3(0, 1, 0), mk3(0, 0, 1), scale3(0.5f, len), clamp);
}

// dito.cpp:428-440
__device__ __forceinline__ void store_from_bounds(kr_obb3* out, f3 b0, f3 b1, f3 b2, f3 lo, f3 hi, bool clamp) {
    f3 len = sub3(hi, lo);
    f3 q = scale3(0.5f, add3(lo, hi));
    f3 mid = scale3(q.x, b0);
    mid = add3(mid, scale3(q.y, b1));
    mid = add3(mid, scale3(q.z, b2));
    store_obb(out, mid, b0, b1, b2, scale3(0.5f, len), clamp);
}

// Lane `src`'s point.
__device__ __forceinline__ f3 shfl3(f3 p, int src) {
    return mk3(__shfl_sync(0xffffffffu, p.x, src), __shfl_sync(0xffffffffu, p.y, src),
               __shfl_sync(0xffffffffu, p.z, src));
}

// The lane a sequential scan with strict improvement ends at: lane 0 first,
// a later lane only where its value is larger.  A NaN in lane 0 keeps lane 0,
// a NaN elsewhere is never taken, equal values (zeros of either sign too) keep
// the first.
__device__ __forceinline__ int scan_argmax(float v) {
    const uint32_t key = v == v ? f2key(v + 0.0f) : 0u;
    const uint32_t best = __reduce_max_sync(0xffffffffu, key);
    const int at = __ffs(__ballot_sync(0xffffffffu, key == best)) - 1;
    return __shfl_sync(0xffffffffu, v, 0) == __shfl_sync(0xffffffffu, v, 0) ? at : 0;
}
__device__ __forceinline__ int scan_argmin(float v) {
    const uint32_t key = v == v ? f2key(v + 0.0f) : 0xffffffffu;
    const uint32_t best = __reduce_min_sync(0xffffffffu, key);
    const int at = __ffs(__ballot_sync(0xffffffffu, key == best)) - 1;
    return __shfl_sync(0xffffffffu, v, 0) == __shfl_sync(0xffffffffu, v, 0) ? at : 0;
}

// The candidate-axis search of DiTO-14 (dito.cpp:478-528, including
// findBestObbAxesFromBaseTriangle :347-380 and the di-tetrahedron :382-418).
// Called by all 32 lanes of one warp: lane e < 14 holds extreme e (min of slab
// 0..6, then max of slab 0..6), its value and the first point reaching it.
// The search is a chain of dependent steps that runs once per set, so what
// counts is its latency: each scan over the points is one value per lane and
// a redux, the up to 21 candidate frames are scored by 21 lanes at once, lane
// f taking frame f in the reference's evaluation order, and the reference's
// "strictly better than the best so far" scan is an argmin with the lowest
// frame index winning ties.  No array is indexed at run time.  (With the
// points in every lane's local memory and the scans run in turn by all lanes,
// pass 1 of a 4,093-point fit took 21.7 us.)
// Writes the plan for the extent pass into ctl, or the final box into out.
inline __device__ void candidate_warp(uint64_t n, float val, f3 sel, const float* xyz, uint32_t flags, Ctl* ctl,
                                      kr_obb3* out) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const Mode md{(flags & OBVH_DITO_REFERENCE_GPU) != 0};
    const bool clamp = !md.gpu;
    const float eps = 0.000001f;
    auto publish = [&](uint32_t path, uint32_t plan, f3 b0, f3 b1, f3 b2, f3 al_mid, f3 al_len, float al_val) {
        if (lane == 0) {
            ctl->path = path;
            ctl->plan = plan;
            ctl->flags = flags;
            float ax[9] = {b0.x, b0.y, b0.z, b1.x, b1.y, b1.z, b2.x, b2.y, b2.z};
            for (int k = 0; k < 9; ++k) ctl->axes[k] = ax[k];
            ctl->al_mid[0] = al_mid.x; ctl->al_mid[1] = al_mid.y; ctl->al_mid[2] = al_mid.z;
            ctl->al_len[0] = al_len.x; ctl->al_len[1] = al_len.y; ctl->al_len[2] = al_len.z;
            ctl->al_val = al_val;
        }
    };
    const f3 I0 = mk3(1, 0, 0), I1 = mk3(0, 1, 0), I2 = mk3(0, 0, 1);

    if (n == 0) {
        if (lane == 0) store_aabb(out, mk3(0, 0, 0), mk3(0, 0, 0), clamp);
        publish(0, 0, I0, I1, I2, mk3(0, 0, 0), mk3(0, 0, 0), 0.f);
        return;
    }

    // The axis extremes as their own points have them: of zeros of both signs a
    // reduction may have returned either, depending on how the points were
    // split over warps and CTAs (the scan from the first point keeps its own).
    {
        const int k = lane < 7 ? lane : lane - 7;
        const float own = k == 0 ? sel.x : (k == 1 ? sel.y : sel.z);
        if (lane < 14 && k < 3 && own == val) val = own;
    }

    // AABB from slabs 0..2 (dito.cpp:507-510)
    const f3 lo3 = mk3(__shfl_sync(kAll, val, 0), __shfl_sync(kAll, val, 1), __shfl_sync(kAll, val, 2));
    const f3 hi3 = mk3(__shfl_sync(kAll, val, 7), __shfl_sync(kAll, val, 8), __shfl_sync(kAll, val, 9));
    const f3 al_mid = mk3((lo3.x + hi3.x) * 0.5f, (lo3.y + hi3.y) * 0.5f, (lo3.z + hi3.z) * 0.5f);
    const f3 al_len = sub3(hi3, lo3);
    const float al_val = half_area3(al_len);

    // Selection set, a point per lane: the 14 extremal points, or every point
    // when there are few; the lanes past it repeat its first point, which
    // changes no extent and never wins a tie.
    const int np = n > 14 ? 14 : static_cast<int>(n);
    f3 P = sel;
    if (n <= 14 && lane < np) P = mk3(xyz[3 * lane], xyz[3 * lane + 1], xyz[3 * lane + 2]);
    {
        const f3 p = shfl3(P, 0);
        if (lane >= np) P = p;
    }

    // Furthest (min, max) pair (dito.cpp:280-292); lanes 7.. repeat pair 0
    const f3 other = shfl3(sel, lane < 7 ? lane + 7 : 7);
    const f3 first = shfl3(sel, lane < 7 ? lane : 0);
    const int far = scan_argmax(len2_3(sub3(first, other)));
    const f3 p0 = shfl3(sel, far), p1 = shfl3(sel, 7 + far);
    if (len2_3(sub3(p1, p0)) < eps) {
        if (lane == 0) store_aabb(out, al_mid, al_len, clamp);
        publish(1, 0, I0, I1, I2, al_mid, al_len, al_val);
        return;
    }
    const f3 e0 = md.unit(sub3(p0, p1));

    // Point furthest from the line through p0 along e0 (dito.cpp:230-258)
    const f3 u = sub3(P, p0);
    const float along = dot3(e0, u);
    const float from_line = len2_3(u) - along * along / len2_3(e0);
    const int far2 = scan_argmax(from_line);
    const f3 p2 = shfl3(P, far2);
    if (__shfl_sync(kAll, from_line, far2) < eps) {
        if (md.gpu) {
            if (lane == 0) store_aabb(out, al_mid, al_len, clamp);
            publish(2, 0, I0, I1, I2, al_mid, al_len, al_val);
            return;
        }
        // Line-aligned frame (dito.cpp:451-476); its extents come from pass 2.
        f3 r = e0;
        if (fabsf(e0.x) > fabsf(e0.y) && fabsf(e0.x) > fabsf(e0.z)) r.x = 0;
        else if (fabsf(e0.y) > fabsf(e0.z)) r.y = 0;
        else r.z = 0;
        if (len2_3(r) < eps) r = mk3(1, 1, 1);
        const f3 v = md.unit(md.cross(e0, r));
        const f3 w = md.unit(md.cross(e0, v));
        publish(2, 2, e0, v, w, al_mid, al_len, al_val);
        return;
    }

    const f3 e1 = md.unit(sub3(p1, p2));
    const f3 e2 = md.unit(sub3(p2, p0));
    const f3 nb = md.unit(md.cross(e1, e0));

    // Di-tetrahedron apexes (dito.cpp:294-307)
    const float height = dot3(P, nb);
    const int top = scan_argmax(height), bottom = scan_argmin(height);
    const f3 q0 = shfl3(P, top), q1 = shfl3(P, bottom);
    const float qhi = __shfl_sync(kAll, height, top), qlo = __shfl_sync(kAll, height, bottom);
    const float tri = dot3(p0, nb);
    const bool up = (qhi - eps > tri);
    const bool down = (qlo + eps < tri);

    // Frames in the reference's evaluation order: triangle t = lane/3, edge
    // k = lane%3.  Triangle 0 is the base (edges e0 e1 e2); triangle 1 + r has
    // the upper apex, 4 + r the lower one, the base edge e_r, the apex edges
    // a_{r+1} and a_r (a_i = unit(apex - p_i)) and the normal
    // unit(a_{r+1} x e_r).  All lanes run the same instructions.
    const int t = lane / 3, k = lane - 3 * t;
    const bool lower = t >= 4;
    const int r = t == 0 ? k : (lower ? t - 4 : t - 1);
    const f3 er = r == 0 ? e0 : (r == 1 ? e1 : e2);
    const f3 from0 = r == 0 ? p0 : (r == 1 ? p1 : p2);
    const f3 from1 = r == 0 ? p1 : (r == 1 ? p2 : p0);
    const f3 apex = lower ? q1 : q0;
    const f3 a0 = md.unit(sub3(apex, from0)), a1 = md.unit(sub3(apex, from1));
    const f3 na = md.unit(md.cross(a1, er));
    const f3 tn = t == 0 ? nb : na;
    const f3 te = t == 0 || k == 0 ? er : (k == 1 ? a1 : a0);
    const f3 tm = md.cross(te, tn);
    const bool valid = lane < 21 && (t == 0 || (lower ? down : up));

    // Extents of the selection set along the three axes.  The reference's scan
    // keeps a NaN of the first point, and such a frame never wins.
    float nlo = kInf, nhi = -kInf, elo = kInf, ehi = -kInf, mlo = kInf, mhi = -kInf;
    bool clean = true;
#pragma unroll
    for (int i = 0; i < 14; ++i) {
        const f3 p = shfl3(P, i);
        const float qn = dot3(p, tn), qe = dot3(p, te), qm = dot3(p, tm);
        if (i == 0) clean = qn == qn && qe == qe && qm == qm;
        nlo = fminf(nlo, qn); nhi = fmaxf(nhi, qn);
        elo = fminf(elo, qe); ehi = fmaxf(ehi, qe);
        mlo = fminf(mlo, qm); mhi = fmaxf(mhi, qm);
    }
    const float q = half_area3(mk3(ehi - elo, nhi - nlo, mhi - mlo));
    float key = valid && clean && q == q ? q : kInf;  // +inf: not a candidate (NaN never wins a strict '<')
    uint32_t who = static_cast<uint32_t>(lane);
    warp_argmin(key, who);
    const int src = static_cast<int>(who);
    const f3 b0 = shfl3(te, src), b1 = shfl3(tn, src), b2 = shfl3(tm, src);

    if (!(key < al_val)) {
        // No frame beats the AABB: its projections give the AABB back exactly,
        // so the box is final without a second pass.
        if (lane == 0) store_aabb(out, al_mid, al_len, clamp);
        publish(md.gpu ? 3 : 4, 0, I0, I1, I2, al_mid, al_len, al_val);
        return;
    }
    publish(3, md.gpu ? 2 : 1, b0, b1, b2, al_mid, al_len, al_val);
}

// Turns the extents along ctl->axes into the final box (dito.cpp:530-537).
__device__ __forceinline__ void finalize_extents(Ctl* ctl, const float lohi[6], uint32_t flags, kr_obb3* out) {
    const bool clamp = (flags & OBVH_DITO_REFERENCE_GPU) == 0;
    const f3 lo = mk3(lohi[0], lohi[1], lohi[2]);
    const f3 hi = mk3(lohi[3], lohi[4], lohi[5]);
    const f3 b0 = mk3(ctl->axes[0], ctl->axes[1], ctl->axes[2]);
    const f3 b1 = mk3(ctl->axes[3], ctl->axes[4], ctl->axes[5]);
    const f3 b2 = mk3(ctl->axes[6], ctl->axes[7], ctl->axes[8]);
    if (ctl->plan == 1) {
        float val = half_area3(sub3(hi, lo));
        if (!(val < ctl->al_val)) {
            store_aabb(out, mk3(ctl->al_mid[0], ctl->al_mid[1], ctl->al_mid[2]),
                       mk3(ctl->al_len[0], ctl->al_len[1], ctl->al_len[2]), clamp);
            ctl->path = 4;
            return;
        }
        ctl->path = 3;
    }
    store_from_bounds(out, b0, b1, b2, lo, hi, clamp);
}

}  // namespace dito
}  // namespace obvh
