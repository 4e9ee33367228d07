// Ray/shape intersection and BVH traversal with the reference's semantics.
//
// Triangle hits are solved exactly as Triangle::Intersect/IntersectTest do
// (src/Shapes/Triangle.cpp:32-93): res = inverse(mat3(v1-v0, v2-v0, -d)) * (o - v0) with glm's
// cofactor inverse (glm/detail/func_matrix.inl compute_inverse<3,3>) and every operation
// rounded separately, and the object box test is RayBoxTest (src/Core/Geometry.h:136-157) with
// the same rounding.  Bit-identical arithmetic matters here because the BVH shadow query hands
// the object-box-clipped interval [t1, t2] to the triangle test (BVH.cpp:132-134): for an
// axis-aligned triangle t1 == t2 and the test passes only when both computations agree to the
// last bit, which makes such triangles partly transparent to shadow rays in the reference.
#pragma once
#include <climits>

#include "dev_common.cuh"

namespace c2g {

struct RayQ {
    float3 o, d, inv;
    int neg[3];
};

__device__ __forceinline__ RayQ make_rayq(float3 o, float3 d) {
    RayQ r;
    r.o = o;
    r.d = d;
    r.inv = f3(__frcp_rn(d.x), __frcp_rn(d.y), __frcp_rn(d.z));
    r.neg[0] = r.inv.x < 0.f;
    r.neg[1] = r.inv.y < 0.f;
    r.neg[2] = r.inv.z < 0.f;
    return r;
}

// Ray of the four-wide traversal with quantised planes: iv is the reciprocal direction clamped to
// +-S.inv_max, m the amount by which its slab distances are widened (see slab_axis).  NEAR: m holds the
// ray's own part, and every node adds what its numbers need; else m covers the whole scene.
template <bool NEAR>
struct QuantRay {
    float3 o, d, iv, m;
};
using Ray4 = QuantRay<false>;
using Ray4n = QuantRay<true>;
constexpr float kUlp = 0x1p-24f;

__device__ __forceinline__ float inv_clamped(const DevScene& S, float d) { return fminf(fmaxf(__frcp_rn(d), -S.inv_max), S.inv_max); }
__device__ __forceinline__ float max_abs(float3 v) { return fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fabsf(v.z)); }

// R: Ray4 or Ray4n (quantised planes), or RayQ (exact planes)
template <class R>
struct RayMaker;
template <>
struct RayMaker<RayQ> {
    static __device__ __forceinline__ RayQ make(const DevScene&, float3 o, float3 d) { return make_rayq(o, d); }
};
template <bool NEAR>
struct RayMaker<QuantRay<NEAR>> {
    static __device__ __forceinline__ QuantRay<NEAR> make(const DevScene& S, float3 o, float3 d) {
        QuantRay<NEAR> r;
        r.o = o;
        r.d = d;
        r.iv = f3(inv_clamped(S, d.x), inv_clamped(S, d.y), inv_clamped(S, d.z));
        // clamped components: no distance at which the ray can meet the scene may lie outside their slabs
        const float ix = fabsf(r.iv.x), iy = fabsf(r.iv.y), iz = fabsf(r.iv.z);
        const float whole = max_abs(d) > 0.f ? 8.f * fmaxf(max_abs(o), S.reach) * fminf(fminf(ix, iy), iz) : 0.f;
        r.m = f3(margin(S.extent[0], o.x) * ix + (ix == S.inv_max ? whole : 0.f), margin(S.extent[1], o.y) * iy + (iy == S.inv_max ? whole : 0.f),
                 margin(S.extent[2], o.z) * iz + (iz == S.inv_max ? whole : 0.f));
        return r;
    }
    static __device__ __forceinline__ float margin(float extent, float o) {
        return NEAR ? 2.f * kUlp * fabsf(o) : __fmaf_rn(fabsf(o), 7.f * kUlp, extent * (16.f * kUlp));
    }
};
template <class R>
__device__ __forceinline__ R make_ray(const DevScene& S, float3 o, float3 d) { return RayMaker<R>::make(S, o, d); }

// Thresholds of trace_queue.
template <class R> struct QueueTuning { static constexpr int kWalkers = 10, kLeaves = 8; };
template <> struct QueueTuning<RayQ> { static constexpr int kWalkers = 0, kLeaves = 1; };

// Whether the boxes above a leaf may be larger than exact.
__device__ __forceinline__ constexpr bool loose_boxes(const RayQ&) { return false; }
template <bool NEAR>
__device__ __forceinline__ constexpr bool loose_boxes(const QuantRay<NEAR>&) { return true; }
// The exact ray of the primitive tests.
__device__ __forceinline__ const RayQ& exact_ray(const DevScene&, const RayQ& r) { return r; }
template <bool NEAR>
__device__ __forceinline__ RayQ exact_ray(const DevScene& S, const QuantRay<NEAR>& r) {
    RayQ q;
    q.o = r.o;
    q.d = r.d;
    q.inv = r.iv;
    if (fabsf(r.iv.x) == S.inv_max) q.inv.x = __frcp_rn(r.d.x);
    if (fabsf(r.iv.y) == S.inv_max) q.inv.y = __frcp_rn(r.d.y);
    if (fabsf(r.iv.z) == S.inv_max) q.inv.z = __frcp_rn(r.d.z);
    q.neg[0] = q.inv.x < 0.f;
    q.neg[1] = q.inv.y < 0.f;
    q.neg[2] = q.inv.z < 0.f;
    return q;
}

// RayBoxTest(ray, inv, invD, box, tMin, tMax): updates t0/t1 like the reference.
__device__ __forceinline__ bool box_test(const RayQ& r, const float* mn, const float* mx, float& t0, float& t1) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
        float o = k == 0 ? r.o.x : (k == 1 ? r.o.y : r.o.z);
        float iv = k == 0 ? r.inv.x : (k == 1 ? r.inv.y : r.inv.z);
        float a = __fmul_rn(__fsub_rn(mn[k], o), iv);
        float b = __fmul_rn(__fsub_rn(mx[k], o), iv);
        if (r.neg[k]) { float t = a; a = b; b = t; }
        t0 = smax(t0, a);
        t1 = smin(t1, b);
        if (t1 < t0) return false;
    }
    return true;
}

// Solve for res (see file comment).  Returns false as soon as a component is rejected.
// mode 0: Intersect acceptance (u+v <= 1 + EPS); mode 1: IntersectTest acceptance (u+v <= 1).
template <int MODE>
__device__ __forceinline__ bool tri_solve(float3 v0, float3 v1, float3 v2, float3 o, float3 d, float& rx, float& ry, float& rz) {
    const float m00 = __fsub_rn(v1.x, v0.x), m01 = __fsub_rn(v1.y, v0.y), m02 = __fsub_rn(v1.z, v0.z);
    const float m10 = __fsub_rn(v2.x, v0.x), m11 = __fsub_rn(v2.y, v0.y), m12 = __fsub_rn(v2.z, v0.z);
    const float m20 = -d.x, m21 = -d.y, m22 = -d.z;
    const float px = __fsub_rn(o.x, v0.x), py = __fsub_rn(o.y, v0.y), pz = __fsub_rn(o.z, v0.z);
    const float c00 = __fsub_rn(__fmul_rn(m11, m22), __fmul_rn(m21, m12));
    const float c01 = __fsub_rn(__fmul_rn(m01, m22), __fmul_rn(m21, m02));
    const float c02 = __fsub_rn(__fmul_rn(m01, m12), __fmul_rn(m11, m02));
    const float det = __fadd_rn(__fsub_rn(__fmul_rn(m00, c00), __fmul_rn(m10, c01)), __fmul_rn(m20, c02));
    const float ood = __frcp_rn(det);
    // row 0 of the inverse -> res.x
    const float i00 = __fmul_rn(c00, ood);
    const float i10 = __fmul_rn(-__fsub_rn(__fmul_rn(m10, m22), __fmul_rn(m20, m12)), ood);
    const float i20 = __fmul_rn(__fsub_rn(__fmul_rn(m10, m21), __fmul_rn(m20, m11)), ood);
    rx = __fadd_rn(__fadd_rn(__fmul_rn(i00, px), __fmul_rn(i10, py)), __fmul_rn(i20, pz));
    if (!(rx >= 0.f && rx <= 1.f)) return false;  // also rejects NaN
    const float i01 = __fmul_rn(-c01, ood);
    const float i11 = __fmul_rn(__fsub_rn(__fmul_rn(m00, m22), __fmul_rn(m20, m02)), ood);
    const float i21 = __fmul_rn(-__fsub_rn(__fmul_rn(m00, m21), __fmul_rn(m20, m01)), ood);
    ry = __fadd_rn(__fadd_rn(__fmul_rn(i01, px), __fmul_rn(i11, py)), __fmul_rn(i21, pz));
    if (!(ry >= 0.f && ry <= 1.f)) return false;
    const float i02 = __fmul_rn(c02, ood);
    const float i12 = __fmul_rn(-__fsub_rn(__fmul_rn(m00, m12), __fmul_rn(m10, m02)), ood);
    const float i22 = __fmul_rn(__fsub_rn(__fmul_rn(m00, m11), __fmul_rn(m10, m01)), ood);
    rz = __fadd_rn(__fadd_rn(__fmul_rn(i02, px), __fmul_rn(i12, py)), __fmul_rn(i22, pz));
    if (rz != rz) return false;
    const float uv = __fadd_rn(rx, ry);
    if (MODE == 0) {
        if (uv > 1.0f + kEpsTri) return false;
    } else {
        if (uv > 1.0f) return false;
    }
    return !(rz < 0.f);
}

// Sphere quadratic (Sphere.cpp:39-91).  Returns the hit distance of Intersect semantics,
// or -1 on a miss.  For IntersectTest semantics use sphere_test.
__device__ __forceinline__ void quadric_local(const Quadric& q, float3 o, float3 dir, float3& P, float3& d) {
    float3 c = f3(q.c[0], q.c[1], q.c[2]);
    float3 rel = o - c;
    // _world2Local * v: column-major mat3 times vector
    P = f3(q.w2l[0] * rel.x + q.w2l[4] * rel.y + q.w2l[8] * rel.z,
           q.w2l[1] * rel.x + q.w2l[5] * rel.y + q.w2l[9] * rel.z,
           q.w2l[2] * rel.x + q.w2l[6] * rel.y + q.w2l[10] * rel.z);
    d = f3(q.w2l[0] * dir.x + q.w2l[4] * dir.y + q.w2l[8] * dir.z,
           q.w2l[1] * dir.x + q.w2l[5] * dir.y + q.w2l[9] * dir.z,
           q.w2l[2] * dir.x + q.w2l[6] * dir.y + q.w2l[10] * dir.z);
}

__device__ __forceinline__ bool sphere_roots(const Quadric& q, float3 o, float3 dir, float& t1, float& t2) {
    float3 P, d;
    quadric_local(q, o, dir, P, d);
    float rad = q.c[3];
    float a = dot(d, d);
    float b = 2 * dot(d, P);
    float c = dot(P, P) - rad * rad;
    float disc = b * b - 4 * a * c;
    if (disc < 0) return false;
    disc = sqrtf(disc);
    t1 = (-b + disc) / (2 * a);
    t2 = (-b - disc) / (2 * a);
    return true;
}

__device__ __forceinline__ float sphere_hit(const Quadric& q, float3 o, float3 dir) {
    float t1, t2;
    if (!sphere_roots(q, o, dir, t1, t2)) return -1.f;
    if (t1 > t2) { float t = t1; t1 = t2; t2 = t; }
    float t = t1;
    if (isnan(t1) || t1 < 0) t = t2;
    if (isnan(t) || t < 0) return -1.f;
    return t;
}

__device__ __forceinline__ bool sphere_test(const Quadric& q, float3 o, float3 dir, float tmin, float tmax) {
    if (tmin > tmax) return false;
    float t1, t2;
    if (!sphere_roots(q, o, dir, t1, t2)) return false;
    return (t1 >= tmin && t1 <= tmax) || (t2 >= tmin && t2 <= tmax);
}

// Disk (Disk.cpp:45-78)
__device__ __forceinline__ float disk_hit(const Quadric& q, float3 o, float3 dir, float tmin, float tmax, bool test) {
    float3 P, d;
    quadric_local(q, o, dir, P, d);
    if (d.y == 0.f) return -1.f;
    float t = -P.y / d.y;
    if (test) {
        if (t < tmin || t > tmax) return -1.f;
    } else if (t < 0) {
        return -1.f;
    }
    float3 h = P + d * t;
    if (dot(h, h) > q.c[3] * q.c[3]) return -1.f;
    return t;
}

// Object box of a prim (IIntersectable::GetBoundingBox): triangle vertex min/max or stored box.
__device__ __forceinline__ void prim_box(const float4& a, const float4& b, const float4& c, int type, float* mn, float* mx) {
    if (type == SHAPE_TRI) {
        mn[0] = fminf(fminf(a.x, b.x), c.x); mn[1] = fminf(fminf(a.y, b.y), c.y); mn[2] = fminf(fminf(a.z, b.z), c.z);
        mx[0] = fmaxf(fmaxf(a.x, b.x), c.x); mx[1] = fmaxf(fmaxf(a.y, b.y), c.y); mx[2] = fmaxf(fmaxf(a.z, b.z), c.z);
    } else {
        mn[0] = b.x; mn[1] = b.y; mn[2] = b.z;
        mx[0] = c.x; mx[1] = c.y; mx[2] = c.z;
    }
}

struct Hit {
    float t, u, v;
    int obj;
};

struct TraceCounters {
    unsigned nodes, prims;
};

// Without object box tests (Brute semantics) a leaf's primitives are tested when the ray meets the
// leaf's exact box (the union of its object boxes).  The quantised boxes of the four-wide nodes
// contain the exact ones, so they alone would let through primitives grazed by rounding only.
template <class R>
__device__ __forceinline__ bool leaf_box_hit(const DevScene& S, int first, int count, const R& r, float t0, float t1) {
    float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int i = 0; i < count; i++) {
        const float4* P = reinterpret_cast<const float4*>(S.prims + first + i);
        const float4 a = __ldg(P), b = __ldg(P + 1), c = __ldg(P + 2);
        float lo[3], hi[3];
        prim_box(a, b, c, prim_type(__float_as_int(a.w)), lo, hi);
#pragma unroll
        for (int k = 0; k < 3; k++) { mn[k] = fminf(mn[k], lo[k]); mx[k] = fmaxf(mx[k], hi[k]); }
    }
    return box_test(exact_ray(S, r), mn, mx, t0, t1);
}

// Closest-hit test of one prim (the leaf body of BVH::Intersect, BVH.cpp:73-90).
template <class R>
__device__ __forceinline__ void closest_prim(const DevScene& S, int pi, const R& r, float tmax, Hit& h, int first = 0, int count = 0) {
    const float4* P = reinterpret_cast<const float4*>(S.prims + pi);
    float4 a = __ldg(P), b = __ldg(P + 1), c = __ldg(P + 2);
    int ot = __float_as_int(a.w);
    int type = prim_type(ot);
    if (S.closest_box) {
        float mn[3], mx[3];
        prim_box(a, b, c, type, mn, mx);
        float t0 = 0.f, t1 = smin(tmax, h.t);
        if (!box_test(exact_ray(S, r), mn, mx, t0, t1)) return;
    }
    float dis;
    float u = 0.f, v = 0.f;
    if (type == SHAPE_TRI) {
        float rz;
        if (!tri_solve<0>(f3(a), f3(b), f3(c), r.o, r.d, u, v, rz)) return;
        dis = rz;
    } else {
        const Quadric& q = S.quads[__float_as_int(b.w)];
        dis = type == SHAPE_SPHERE ? sphere_hit(q, r.o, r.d) : disk_hit(q, r.o, r.d, 0.f, 0.f, false);
        if (dis < 0.f) return;
    }
    if (dis < h.t) {
        if (count > 0 && !S.closest_box && !leaf_box_hit(S, first, count, r, 0.f, smin(tmax, h.t))) return;
        h.t = dis;
        h.u = u;
        h.v = v;
        h.obj = prim_obj(ot);
    }
}

// Any-hit test of one prim (leaf body of BVH::IntersectTest, BVH.cpp:127-136).
template <class R>
__device__ __forceinline__ bool anyhit_prim(const DevScene& S, int pi, const R& r, float tmin, float tmax, int ignore, int first = 0,
                                            int count = 0) {
    const float4* P = reinterpret_cast<const float4*>(S.prims + pi);
    float4 a = __ldg(P), b = __ldg(P + 1), c = __ldg(P + 2);
    int ot = __float_as_int(a.w);
    if (prim_obj(ot) == ignore) return false;
    int type = prim_type(ot);
    float t0 = tmin, t1 = tmax;
    if (S.anyhit_clip) {
        float mn[3], mx[3];
        prim_box(a, b, c, type, mn, mx);
        if (!box_test(exact_ray(S, r), mn, mx, t0, t1)) return false;
    }
    if (type == SHAPE_TRI) {
        if (t0 > t1) return false;
        float rx, ry, rz;
        if (!tri_solve<1>(f3(a), f3(b), f3(c), r.o, r.d, rx, ry, rz)) return false;
        if (!(rz >= t0 && rz <= t1)) return false;
    } else {
        const Quadric& q = S.quads[__float_as_int(b.w)];
        if (type == SHAPE_SPHERE ? !sphere_test(q, r.o, r.d, t0, t1) : !(disk_hit(q, r.o, r.d, t0, t1, true) >= 0.f)) return false;
    }
    return !(count > 0 && !S.anyhit_clip) || leaf_box_hit(S, first, count, r, tmin, tmax);
}

constexpr int kStack = 64;

// BVH::Intersect over the reference tree (BVH.cpp:56-108): near child by the sign of the ray
// on the split axis, node box clipped by the current closest distance.
template <bool COUNT>
__device__ __forceinline__ Hit trace_closest_ref(const DevScene& S, const RayQ& r, float tmax, TraceCounters* cnt) {
    Hit h{INFINITY, 0.f, 0.f, -1};
    int stack[kStack];
    int top = 0;
    int cur = 1;
    while (true) {
        const float4* N = reinterpret_cast<const float4*>(S.ref_nodes + cur);
        float4 A = __ldg(N), B = __ldg(N + 1);
        if (COUNT) cnt->nodes++;
        float mn[3] = {A.x, A.y, A.z}, mx[3] = {B.x, B.y, B.z};
        float t0 = 0.f, t1 = smin(tmax, h.t);
        bool ok = box_test(r, mn, mx, t0, t1);
        int a = __float_as_int(A.w), b = __float_as_int(B.w);
        int axis = (b >> 28) & 3;
        if (ok && axis == 3) {
            int cnt_ = b & 0x0fffffff;
            for (int i = 0; i < cnt_; i++) {
                if (COUNT) cnt->prims++;
                closest_prim(S, a + i, r, tmax, h);
            }
        } else if (ok) {
            int c1 = b & 0x0fffffff;
            int neg = axis == 0 ? r.neg[0] : (axis == 1 ? r.neg[1] : r.neg[2]);
            if (top >= kStack) { dev_flag_error(S.err, DEVERR_STACK); break; }
            stack[top++] = neg ? a : c1;
            cur = neg ? c1 : a;
            continue;
        }
        if (!top) break;
        cur = stack[--top];
    }
    return h;
}

template <bool COUNT>
__device__ __forceinline__ bool trace_any_ref(const DevScene& S, const RayQ& r, float tmin, float tmax, int ignore, TraceCounters* cnt) {
    int stack[kStack];
    int top = 0;
    int cur = 1;
    while (true) {
        const float4* N = reinterpret_cast<const float4*>(S.ref_nodes + cur);
        float4 A = __ldg(N), B = __ldg(N + 1);
        if (COUNT) cnt->nodes++;
        float mn[3] = {A.x, A.y, A.z}, mx[3] = {B.x, B.y, B.z};
        float t0 = tmin, t1 = tmax;
        bool ok = box_test(r, mn, mx, t0, t1);
        int a = __float_as_int(A.w), b = __float_as_int(B.w);
        int axis = (b >> 28) & 3;
        if (ok && axis == 3) {
            int cnt_ = b & 0x0fffffff;
            for (int i = 0; i < cnt_; i++) {
                if (COUNT) cnt->prims++;
                if (anyhit_prim(S, a + i, r, tmin, tmax, ignore)) return true;
            }
        } else if (ok) {
            int c1 = b & 0x0fffffff;
            int neg = axis == 0 ? r.neg[0] : (axis == 1 ? r.neg[1] : r.neg[2]);
            if (top >= kStack) { dev_flag_error(S.err, DEVERR_STACK); return false; }
            stack[top++] = neg ? a : c1;
            cur = neg ? c1 : a;
            continue;
        }
        if (!top) break;
        cur = stack[--top];
    }
    return false;
}

// Compact SAH tree traversal ("while-while" with leaf postponing).  Both child boxes live in the
// parent node; a child is an inner-node index or a leaf (first prim, count) packed into a negative
// reference.  Each lane walks inner nodes until it has found a leaf, then keeps walking while other
// lanes of the warp still search; the leaves are intersected together once every active lane has
// one, so the expensive exact triangle tests run with most lanes active.  Closest-hit pushes carry
// the entry distance so that subtrees beyond the current hit are dropped on pop.
constexpr int kNoRef = INT_MIN;
__device__ __forceinline__ int leaf_ref(int first, int count) { return -1 - ((first << 3) | count); }
__device__ __forceinline__ bool is_leaf(int ref) { return ref < 0 && ref != kNoRef; }
__device__ __forceinline__ void leaf_range(int ref, int& first, int& count) {
    int v = -1 - ref;
    first = v >> 3;
    count = v & 7;
}

template <bool COUNT>
__device__ __forceinline__ Hit trace_closest_sah(const DevScene& S, const RayQ& r, float tmax, TraceCounters* cnt) {
    Hit h{INFINITY, 0.f, 0.f, -1};
    int stack[kStack];
    float stack_t[kStack];
    int top = 0;
    int ref = 0, leaf = kNoRef;
    auto pop = [&]() -> int {
        while (top > 0) {
            --top;
            if (stack_t[top] <= h.t) return stack[top];
        }
        return kNoRef;
    };
    while (ref != kNoRef || leaf != kNoRef) {
        while (ref >= 0) {
            const float4* N = reinterpret_cast<const float4*>(S.wide_nodes + ref);
            float4 L0 = __ldg(N), H0 = __ldg(N + 1), L1 = __ldg(N + 2), H1 = __ldg(N + 3);
            if (COUNT) cnt->nodes++;
            float lim = smin(tmax, h.t);
            float mn0[3] = {L0.x, L0.y, L0.z}, mx0[3] = {H0.x, H0.y, H0.z};
            float mn1[3] = {L1.x, L1.y, L1.z}, mx1[3] = {H1.x, H1.y, H1.z};
            float a0 = 0.f, b0 = lim, a1 = 0.f, b1 = lim;
            bool hit0 = box_test(r, mn0, mx0, a0, b0);
            bool hit1 = box_test(r, mn1, mx1, a1, b1);
            int n0 = __float_as_int(H0.w), n1 = __float_as_int(H1.w);
            int r0 = n0 > 0 ? leaf_ref(__float_as_int(L0.w), n0) : __float_as_int(L0.w);
            int r1 = n1 > 0 ? leaf_ref(__float_as_int(L1.w), n1) : __float_as_int(L1.w);
            if (hit0 && hit1) {
                bool swap = a1 < a0;
                int nr = swap ? r1 : r0, fr = swap ? r0 : r1;
                float ft = swap ? a0 : a1;
                if (top >= kStack) { dev_flag_error(S.err, DEVERR_STACK); return h; }
                stack[top] = fr;
                stack_t[top] = ft;
                top++;
                ref = nr;
            } else if (hit0) {
                ref = r0;
            } else if (hit1) {
                ref = r1;
            } else {
                ref = pop();
            }
            if (is_leaf(ref) && leaf == kNoRef) {
                leaf = ref;
                ref = pop();
            }
            if (!__any_sync(__activemask(), leaf == kNoRef)) break;
        }
        while (leaf != kNoRef) {
            int first, count;
            leaf_range(leaf, first, count);
            for (int i = 0; i < count; i++) {
                if (COUNT) cnt->prims++;
                closest_prim(S, first + i, r, tmax, h);
            }
            leaf = kNoRef;
            if (is_leaf(ref)) {
                leaf = ref;
                ref = pop();
            }
        }
    }
    return h;
}

template <bool COUNT>
__device__ __forceinline__ bool trace_any_sah(const DevScene& S, const RayQ& r, float tmin, float tmax, int ignore, TraceCounters* cnt) {
    int stack[kStack];
    int top = 0;
    int ref = 0, leaf = kNoRef;
    while (ref != kNoRef || leaf != kNoRef) {
        while (ref >= 0) {
            const float4* N = reinterpret_cast<const float4*>(S.wide_nodes + ref);
            float4 L0 = __ldg(N), H0 = __ldg(N + 1), L1 = __ldg(N + 2), H1 = __ldg(N + 3);
            if (COUNT) cnt->nodes++;
            float mn0[3] = {L0.x, L0.y, L0.z}, mx0[3] = {H0.x, H0.y, H0.z};
            float mn1[3] = {L1.x, L1.y, L1.z}, mx1[3] = {H1.x, H1.y, H1.z};
            float a0 = tmin, b0 = tmax, a1 = tmin, b1 = tmax;
            bool hit0 = box_test(r, mn0, mx0, a0, b0);
            bool hit1 = box_test(r, mn1, mx1, a1, b1);
            int n0 = __float_as_int(H0.w), n1 = __float_as_int(H1.w);
            int r0 = n0 > 0 ? leaf_ref(__float_as_int(L0.w), n0) : __float_as_int(L0.w);
            int r1 = n1 > 0 ? leaf_ref(__float_as_int(L1.w), n1) : __float_as_int(L1.w);
            if (hit0 && hit1) {
                if (top >= kStack) { dev_flag_error(S.err, DEVERR_STACK); return false; }
                stack[top++] = r1;
                ref = r0;
            } else if (hit0) {
                ref = r0;
            } else if (hit1) {
                ref = r1;
            } else {
                ref = top ? stack[--top] : kNoRef;
            }
            if (is_leaf(ref) && leaf == kNoRef) {
                leaf = ref;
                ref = top ? stack[--top] : kNoRef;
            }
            if (!__any_sync(__activemask(), leaf == kNoRef)) break;
        }
        while (leaf != kNoRef) {
            int first, count;
            leaf_range(leaf, first, count);
            for (int i = 0; i < count; i++) {
                if (COUNT) cnt->prims++;
                if (anyhit_prim(S, first + i, r, tmin, tmax, ignore)) return true;
            }
            leaf = kNoRef;
            if (is_leaf(ref)) {
                leaf = ref;
                ref = top ? stack[--top] : kNoRef;
            }
        }
    }
    return false;
}

// ---- four-wide SAH traversal --------------------------------------------------------------------
// Node boxes are tested conservatively: every child whose exact box the reference's RayBoxTest would
// accept is entered, so the primitives tested include all the reference's, and the exact tests of the
// primitives (their own boxes under BVH semantics, their leaf's box under Brute semantics) decide.
//
// What bounds the traversal is the latency of dependent node loads with few lanes per warp active,
// then issue.  A node is 64 bytes read as two 256-bit loads (it was 128 bytes in seven 128-bit loads
// with FP32 planes): half the footprint in L1 and L2, 16 instead of 28 registers in flight, and the
// planes decode with one byte permutation each into packed FMAs.  1080p many-material step, shadow
// rays 21.4 -> 17.4 ms, extension 12.6 -> 11.2 ms; 2M closest-hit rays of a 65k-triangle soup
// 1.38 -> 0.93 ms, any hit 0.82 -> 0.54 ms.  15-bit planes (96 bytes) measured 18.8 / 12.3 ms.
//
// Slab distances: t = v(q) * a + p with a = scale * iv and p = (org - o) * iv, widened by m.  With
// u = 2^-24 and v < 2 the roundings of t (a, org - o, the offset and the final FMA) come to at most
// u (4 |a| + 3 |p|), those of the exact test of a plane, at most 2 scale from org, to u (4 |a| + 2 |p|),
// and a plane may lie inside its box by u (1.5 scale + |org|) (quantise_axis), where
// |org| <= |org - o| + |o|: together u (9.5 |a| + 6 |p| + |o iv|).
//   Ray4n: m = u (12 |a| + 8 |p| + 2 |o iv|), from the node's own numbers.
//   Ray4: with E the scene's largest coordinate on the axis, planes and o at most E + |o| apart,
//   scale <= 1.35 E and |org| <= 1.7 E, the same sum is below u (13 E + 5 |o|) |iv|; m = u (16 E + 7 |o|) |iv|
//   is the ray's for all nodes, and saves two FMAs per axis.
// One object far from all others makes E large against most boxes: 1e5 units from a soup of triangles of
// 0.05 in the unit cube a ray tested 280 of them instead of 11, and every one at 1e6.  So scenes with more
// than 64 leaves narrower than 2^-14 of their reach, 64 times m, take Ray4n: 11 there, as without the far
// object.  For every scene it would cost the 1080p many-material frame 0.4%, and 2M closest-hit rays of a
// 65k-triangle soup 5%.
//
// A direction component that is zero, or so small that the ray crosses the whole scene without moving along
// the axis, gives iv = S.inv_max, and m then adds the largest distance at which the ray can meet the scene:
// the slab accepts when the origin lies within it, up to 2^-116 reach^2 for unit directions, whatever the
// length of the direction.  (Without this term directions of 1e-28 and shorter, whose hits lie beyond 2^100
// times their slab, lost them.)  S.inv_max is 2^120 over the scene's reach, so that scale * iv and the
// offset of an origin among the scene's coordinates stay finite (with 2^100 for every scene the product
// overflowed from 4e8 units on, and a near plane at infinity hid the whole node).
constexpr int kStack4 = 128;

__device__ __forceinline__ unsigned long long pack2(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
// (a0, a1) * s + b on both halves of a register pair
__device__ __forceinline__ void fma2(float a0, float a1, float s, float b, float& r0, float& r1) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(pack2(a0, a1)), "l"(pack2(s, s)), "l"(pack2(b, b)));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r0), "=f"(r1) : "l"(r));
}
// byte K of a plane word as its plane value (Node4)
template <int K>
__device__ __forceinline__ float plane_byte(uint32_t w) {
    return __uint_as_float(__byte_perm(w, 0x3f000000u, 0x7044u | (K << 8)));
}
template <bool NEAR>
__device__ __forceinline__ void slab_axis(uint32_t qlo, uint32_t qhi, float org, float scale, float o, float iv, float m,
                                          float tn[4], float tf[4]) {
    const float dx = org - o, a = scale * iv;
    if (NEAR) m = __fmaf_rn(__fmaf_rn(scale, 1.5f, fabsf(dx)), 8.f * kUlp * fabsf(iv), m);
    const float bn = __fmaf_rn(dx, iv, -m), bf = __fmaf_rn(dx, iv, m);
    const uint32_t wn = iv < 0.f ? qhi : qlo, wf = iv < 0.f ? qlo : qhi;
    fma2(plane_byte<0>(wn), plane_byte<1>(wn), a, bn, tn[0], tn[1]);
    fma2(plane_byte<2>(wn), plane_byte<3>(wn), a, bn, tn[2], tn[3]);
    fma2(plane_byte<0>(wf), plane_byte<1>(wf), a, bf, tf[0], tf[1]);
    fma2(plane_byte<2>(wf), plane_byte<3>(wf), a, bf, tf[2], tf[3]);
}
// 32 bytes (32-byte aligned) of read-only data in one load
__device__ __forceinline__ void ld256(const void* p, uint32_t v[8]) {
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "l"(p));
}
// Entry and exit distances of a node's four child boxes, and its children.
template <bool NEAR>
__device__ __forceinline__ int4 node4_slabs(const DevScene& S, int ref, const QuantRay<NEAR>& r, float t0, float t1, float tn[4], float tf[4]) {
    const Node4* nodes = S.nodes4;
    uint32_t u[8], v[8];
    ld256(nodes + ref, u);
    ld256(reinterpret_cast<const char*>(nodes + ref) + 32, v);
    float xn[4], xf[4], yn[4], yf[4], zn[4], zf[4];
    slab_axis<NEAR>(u[6], u[7], __uint_as_float(u[0]), __uint_as_float(u[3]), r.o.x, r.iv.x, r.m.x, xn, xf);
    slab_axis<NEAR>(v[0], v[1], __uint_as_float(u[1]), __uint_as_float(u[4]), r.o.y, r.iv.y, r.m.y, yn, yf);
    slab_axis<NEAR>(v[2], v[3], __uint_as_float(u[2]), __uint_as_float(u[5]), r.o.z, r.iv.z, r.m.z, zn, zf);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        tn[k] = fmaxf(fmaxf(xn[k], yn[k]), fmaxf(zn[k], t0));
        tf[k] = fminf(fminf(xf[k], yf[k]), fminf(zf[k], t1));
    }
    return make_int4((int)v[4], (int)v[5], (int)v[6], (int)v[7]);
}

// The same with exact planes: RayBoxTest's own operations (subtract, multiply, each rounded; two planes
// per packed instruction), combined with fmaxf / fminf, which ignore NaN as the reference's std::max /
// std::min argument order does.  The ray's direction signs pick the near and far planes.
__device__ __forceinline__ void slab_exact(const float4& p, float o, float iv, float t[4]) {
    unsigned long long a = pack2(p.x, p.y), b = pack2(p.z, p.w);
    const unsigned long long no = pack2(-o, -o), i2 = pack2(iv, iv);
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(a) : "l"(no));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(b) : "l"(no));
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(a) : "l"(i2));
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(b) : "l"(i2));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(t[0]), "=f"(t[1]) : "l"(a));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(t[2]), "=f"(t[3]) : "l"(b));
}
__device__ __forceinline__ int4 node4_slabs(const DevScene& S, int ref, const RayQ& r, float t0, float t1, float tn[4], float tf[4]) {
    const float4* N = reinterpret_cast<const float4*>(S.nodes4x + ref);
    float xn[4], xf[4], yn[4], yf[4], zn[4], zf[4];
    slab_exact(__ldg(N + r.neg[0]), r.o.x, r.inv.x, xn);
    slab_exact(__ldg(N + (r.neg[0] ^ 1)), r.o.x, r.inv.x, xf);
    slab_exact(__ldg(N + 2 + r.neg[1]), r.o.y, r.inv.y, yn);
    slab_exact(__ldg(N + 2 + (r.neg[1] ^ 1)), r.o.y, r.inv.y, yf);
    slab_exact(__ldg(N + 4 + r.neg[2]), r.o.z, r.inv.z, zn);
    slab_exact(__ldg(N + 4 + (r.neg[2] ^ 1)), r.o.z, r.inv.z, zf);
    const int4 ch = __ldg(reinterpret_cast<const int4*>(N + 6));
#pragma unroll
    for (int k = 0; k < 4; k++) {
        tn[k] = fmaxf(fmaxf(xn[k], yn[k]), fmaxf(zn[k], t0));
        tf[k] = fminf(fminf(xf[k], yf[k]), fminf(zf[k], t1));
    }
    return ch;
}

__device__ __forceinline__ void cswap(float& ta, int& ca, float& tb, int& cb) {
    if (tb < ta) {
        float t = ta; ta = tb; tb = t;
        int c = ca; ca = cb; cb = c;
    }
}

// Traversal state of one ray: the next subtree (inner node, leaf or kNoRef), a postponed leaf, and
// the stacked subtrees.  A lane keeps walking inner nodes past its first leaf while the other lanes
// of its warp walk too; the exact primitive tests then run with many lanes active.  The stack is an
// array of its own (any hit: subtrees; closest hit: (subtree, entry distance) pairs), so that the
// rest of the state stays in registers.
struct Bvh4State {
    int top, ref, leaf;
};
__device__ __forceinline__ int bvh4_pop(const int* stack, Bvh4State& st) { return st.top > 0 ? stack[--st.top] : kNoRef; }
// subtrees beyond the current hit are dropped
__device__ __forceinline__ int bvh4_pop(const float2* stack, Bvh4State& st, float t) {
    while (st.top > 0) {
        const float2 e = stack[--st.top];
        if (e.y <= t) return __float_as_int(e.x);
    }
    return kNoRef;
}

__device__ __forceinline__ void bvh4_begin(Bvh4State& st) {
    st.top = 0;
    st.ref = 0;
    st.leaf = kNoRef;
}
__device__ __forceinline__ bool bvh4_done(const Bvh4State& st) { return st.ref == kNoRef && st.leaf == kNoRef; }

// One inner node (st.ref >= 0) of an any-hit ray on (tmin, tmax).
template <bool COUNT, class R>
__device__ __forceinline__ void bvh4_any_node(const DevScene& S, const R& r, float tmin, float tmax, int* stack, Bvh4State& st,
                                              TraceCounters* cnt) {
    if (COUNT) cnt->nodes++;
    float tn[4], tf[4];
    const int4 ch = node4_slabs(S, st.ref, r, tmin, tmax, tn, tf);
    if (st.top + 3 > kStack4) { dev_flag_error(S.err, DEVERR_STACK); st.top = 0; st.ref = kNoRef; st.leaf = kNoRef; return; }
    int next = kNoRef;
    if (tn[3] <= tf[3]) next = ch.w;
    if (tn[2] <= tf[2]) { if (next != kNoRef) stack[st.top++] = next; next = ch.z; }
    if (tn[1] <= tf[1]) { if (next != kNoRef) stack[st.top++] = next; next = ch.y; }
    if (tn[0] <= tf[0]) { if (next != kNoRef) stack[st.top++] = next; next = ch.x; }
    st.ref = next != kNoRef ? next : bvh4_pop(stack, st);
    if (is_leaf(st.ref) && st.leaf == kNoRef) {
        st.leaf = st.ref;
        st.ref = bvh4_pop(stack, st);
    }
}

// The postponed leaf of an any-hit ray; true when the ray is occluded.
template <bool COUNT, class R>
__device__ __forceinline__ bool bvh4_any_leaf(const DevScene& S, const R& r, float tmin, float tmax, int ignore,
                                              int* stack, Bvh4State& st, TraceCounters* cnt) {
    int first, count;
    leaf_range(st.leaf, first, count);
    st.leaf = kNoRef;
    for (int k = 0; k < count; k++) {
        if (COUNT) cnt->prims++;
        if (anyhit_prim(S, first + k, r, tmin, tmax, ignore, first, loose_boxes(r) ? count : 0)) return true;
    }
    if (is_leaf(st.ref)) {
        st.leaf = st.ref;
        st.ref = bvh4_pop(stack, st);
    }
    return false;
}

// One inner node of a closest-hit ray (h carries the running result): children nearest first.
template <bool COUNT, class R>
__device__ __forceinline__ void bvh4_closest_node(const DevScene& S, const R& r, float tmax, const Hit& h, float2* stack, Bvh4State& st,
                                                  TraceCounters* cnt) {
    if (COUNT) cnt->nodes++;
    float t[4], tf[4];
    const int4 ch = node4_slabs(S, st.ref, r, 0.f, smin(tmax, h.t), t, tf);
    int c[4] = {ch.x, ch.y, ch.z, ch.w};
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (!(t[k] <= tf[k])) { t[k] = INFINITY; c[k] = kNoRef; }
    cswap(t[0], c[0], t[1], c[1]);
    cswap(t[2], c[2], t[3], c[3]);
    cswap(t[0], c[0], t[2], c[2]);
    cswap(t[1], c[1], t[3], c[3]);
    cswap(t[1], c[1], t[2], c[2]);
    if (st.top + 3 > kStack4) { dev_flag_error(S.err, DEVERR_STACK); st.top = 0; st.ref = kNoRef; st.leaf = kNoRef; return; }
#pragma unroll
    for (int k = 3; k >= 1; k--)
        if (c[k] != kNoRef) stack[st.top++] = make_float2(__int_as_float(c[k]), t[k]);
    st.ref = c[0] != kNoRef ? c[0] : bvh4_pop(stack, st, h.t);
    if (is_leaf(st.ref) && st.leaf == kNoRef) {
        st.leaf = st.ref;
        st.ref = bvh4_pop(stack, st, h.t);
    }
}

template <bool COUNT, class R>
__device__ __forceinline__ void bvh4_closest_leaf(const DevScene& S, const R& r, float tmax, Hit& h, float2* stack, Bvh4State& st,
                                                  TraceCounters* cnt) {
    int first, count;
    leaf_range(st.leaf, first, count);
    st.leaf = kNoRef;
    for (int k = 0; k < count; k++) {
        if (COUNT) cnt->prims++;
        closest_prim(S, first + k, r, tmax, h, first, loose_boxes(r) ? count : 0);
    }
    if (is_leaf(st.ref)) {
        st.leaf = st.ref;
        st.ref = bvh4_pop(stack, st, h.t);
    }
}

// ---- persistent warps with ray replacement -----------------------------------------------------
// Warp-wide refill: lanes that need a ray take consecutive indices from *fetch.  Returns the index
// for this lane (-1: none left) and must be called by all 32 lanes.
__device__ __forceinline__ int warp_fetch(int* fetch, bool need, int n) {
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(0xffffffffu, need);
    if (!m) return -1;
    const int leader = __ffs(m) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(fetch, __popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (!need) return -1;
    const int idx = base + __popc(m & ((1u << lane) - 1u));
    return idx < n ? idx : -1;
}

// Traces the n queued rays with every lane of the grid: rounds of inner nodes, then postponed leaves; a
// lane whose ray is finished takes the next ray of the queue after the round (persistent threads with
// ray replacement).  All 32 lanes take part in the votes, so the warp reconverges at every step.
//
// The node loop ends when at most Lane::kWalkers lanes still walk (they wait for the leaves and the
// refill instead of the others for them), the leaf loop when fewer than Lane::kLeaves lanes hold a
// leaf.  Quantised planes (scenes of some size) take 10 and 8: 1080p many-material step, extension +
// shadow rays, 27.6 ms; 10 and 32 28.5; 10 and 1 29.4; 14 and 1 30.9; 6 and 1 30.1; 0 and 1 33.3; a
// refill as soon as 8 lanes are idle, without rounds, 31.7 (coherent rays lose their common path).
// Exact planes (a handful of nodes, all in L1: bound by issue) take 0 and 1: Cornell box at 64 spp,
// extension + shadow rays, 1.64 ms against 1.90 with 10 and 32, 1.83 with 10 and 8.  An empty queue
// ends the waiting for a refill.
//
// The first rays are dealt out by thread index, the others by the counter *fetch.  Fewer rays than
// threads are spread over the warps (one ray in every 2nd, 4th, ... lane): a late bounce level's time
// is its slowest warp's, and a warp of few rays diverges less.
// `L` is one lane's tracer:
//   begin(idx)                 loads ray idx and resets the traversal
//   node(stack), leaf(stack)   one step on L.st
//   end(idx, done)             called by all lanes of the warp: the lanes with `done` store their result
template <class Lane>
__device__ __forceinline__ void trace_queue(Lane& L, int* fetch, int n) {
    typename Lane::Stack stack[kStack4];
    const int threads = gridDim.x * blockDim.x, tid = blockIdx.x * blockDim.x + threadIdx.x;
    int spread = 0;  // log2
    while (spread < 5 && (long long)n << (spread + 1) <= threads) spread++;
    int ray = (tid & ((1 << spread) - 1)) == 0 && tid >> spread < n ? tid >> spread : -1;
    L.st.top = 0;
    L.st.ref = L.st.leaf = kNoRef;  // an idle lane has nothing to walk
    if (ray >= 0) L.begin(ray);
    bool more = n > threads;        // rays may be left in the queue (warp-uniform)
    while (true) {
        if (__ballot_sync(0xffffffffu, ray >= 0) == 0) break;
        const int enough = more ? Lane::kWalkers : 0;
        unsigned walk = __ballot_sync(0xffffffffu, L.st.ref >= 0);
        while (walk) {
            if (L.st.ref >= 0) L.node(stack);
            walk = __ballot_sync(0xffffffffu, L.st.ref >= 0);
            if (__popc(walk) <= enough) break;
        }
        unsigned leaves = __ballot_sync(0xffffffffu, L.st.leaf != kNoRef);
        while (leaves) {
            if (L.st.leaf != kNoRef) L.leaf(stack);
            leaves = __ballot_sync(0xffffffffu, L.st.leaf != kNoRef);
            if (__popc(leaves) < Lane::kLeaves) break;
        }
        const bool done = ray >= 0 && bvh4_done(L.st);
        if (__any_sync(0xffffffffu, done)) {
            L.end(ray, done);
            if (done) ray = -1;
        }
        if (more) {
            const int idx = warp_fetch(fetch, ray < 0, n - threads);
            if (idx >= 0) {
                ray = threads + idx;
                L.begin(ray);
            }
            more = !__any_sync(0xffffffffu, ray < 0);
        }
    }
}

// One ray per thread: the reference tree and the binary SAH tree (four-wide nodes: trace_queue).
template <bool COUNT>
__device__ __forceinline__ Hit trace_closest(const DevScene& S, float3 o, float3 d, TraceCounters* cnt) {
    RayQ r = make_rayq(o, d);
    if (S.tree == 1) return trace_closest_sah<COUNT>(S, r, INFINITY, cnt);
    return trace_closest_ref<COUNT>(S, r, INFINITY, cnt);
}

template <bool COUNT>
__device__ __forceinline__ bool trace_any(const DevScene& S, float3 o, float3 d, float tmin, float tmax, int ignore, TraceCounters* cnt) {
    RayQ r = make_rayq(o, d);
    if (S.tree == 1) return trace_any_sah<COUNT>(S, r, tmin, tmax, ignore, cnt);
    return trace_any_ref<COUNT>(S, r, tmin, tmax, ignore, cnt);
}

}  // namespace c2g
