// Ray-primitive tests and BVH traversal (closest hit and any hit).
//
// Primitive tests repeat the reference's arithmetic in its order
// (TriangleDetail.h:21-57, SphereDetail.h:33-74, QuadDetail.h:21-57,
// PlaneDetail.h:19-46) so that the hit distance of every candidate equals the
// reference's.  Which candidate wins also follows the reference: a hit on an
// object with a finite box only counts if the reference's own slab test
// (AABBDetail.h:18-50, with its +EPSILON direction perturbation) accepts
// that box, and exact ties go to the smaller primitive key, where keys run
// in the leaf order of the reference's object BVH (first object in its
// depth-first order, then triangle index, MeshDetail.h:28-35).
//
// The SAH BVH itself is traversed with conservative FMA slab tests against
// boxes that the builder inflated, a per-thread short stack of (t_near, node)
// entries and near-child-first ordering.
#pragma once

#include "bvh_build.hpp"
#include "dev_common.cuh"
#include "slab.hpp"

namespace cupbr_b200 {

#ifndef CUPBR_STACK_SIZE
#define CUPBR_STACK_SIZE 64
#endif

// TriangleDetail.h:21-57
__device__ __forceinline__ bool isect_tri(float4 a, float4 b, float4 c, f3 o, f3 d, float& t) {
    f3 v0v1 = xyz(b), v0v2 = xyz(c);
    f3 pvec = cross(d, v0v2);
    float det = dot(v0v1, pvec);
    if (feq0(det)) return false;
    float invDet = 1.0f / det;
    f3 tvec = o - xyz(a);
    float u = dot(tvec, pvec) * invDet;
    if (u < 0.0f || u > 1.0f) return false;
    f3 qvec = cross(tvec, v0v1);
    float v = dot(d, qvec) * invDet;
    if (v < 0.0f || u + v > 1.0f) return false;
    t = dot(v0v2, qvec) * invDet;
    return !(t < 0.0f);
}

// SphereDetail.h:33-74
__device__ __forceinline__ bool isect_sphere(float4 s0, float4 s1, f3 o, f3 d, float& t) {
    f3 OS = o - xyz(s0);
    float b = 2.0f * dot(d, OS);
    float c = dot(OS, OS) - s1.y;
    float disc = b * b - 4.0f * c;
    if (!(disc > 0.0f)) return false;
    float ds = sqrtf(disc);
    float q = b < 0.0f ? (-b - ds) / 2.0f : (-b + ds) / 2.0f;
    float t0 = q, t1 = c / q;
    float mn = fminf(t0, t1), mx = fmaxf(t0, t1);
    t = mn < 0.0f ? mx : mn;
    return t >= 0.0f;
}

// QuadDetail.h:21-57 (check_extent) and PlaneDetail.h:19-46
__device__ __forceinline__ bool isect_quad(float4 q0, float4 q1, float4 q2, float4 q3, f3 o, f3 d, float& t) {
    f3 n = xyz(q1);
    float OdotN = dot(o, n);
    float DdotN = dot(d, n);
    if (feq0(DdotN)) return false;
    t = (q1.w - OdotN) / DdotN;
    if (t < 0.0f) return false;
    f3 I = o + t * d;
    f3 r = I - xyz(q0);
    float x = dot(r, xyz(q2));
    float y = dot(r, xyz(q3));
    float s1 = q2.w, s2 = q3.w;
    return !(x < -s1 || x > s1 || y < -s2 || y > s2);
}
__device__ __forceinline__ bool isect_plane(float4 p0, float4 p1, f3 o, f3 d, float& t) {
    f3 n = xyz(p1);
    float PdotN = dot(xyz(p0), n);
    float OdotN = dot(o, n);
    float DdotN = dot(d, n);
    if (feq0(DdotN)) return false;
    t = (PdotN - OdotN) / DdotN;
    return !(t < 0.0f);
}

// AABBDetail.h:18-50 on the object's own box
__device__ __forceinline__ bool ref_box_hit(float4 lo, float4 hi, f3 o, f3 d) {
    bool hit = true;
    float tmin = 0.0f, tmax = __int_as_float(0x7f800000);
    const float los[3] = {lo.x, lo.y, lo.z}, his[3] = {hi.x, hi.y, hi.z};
    const float os[3] = {o.x, o.y, o.z}, ds[3] = {d.x, d.y, d.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float invD = 1.0f / (ds[a] + CUPBR_EPS);
        float t0 = (los[a] - os[a]) * invD;
        float t1 = (his[a] - os[a]) * invD;
        if (invD < 0.0f) { float tt = t0; t0 = t1; t1 = tt; }
        tmin = t0 > tmin ? t0 : tmin;
        tmax = t1 < tmax ? t1 : tmax;
        if (tmax <= tmin) hit = false;
    }
    return hit;
}

// Per-ray cache of the reference box predicate for the last object asked.
struct RefBoxCache {
    int32_t obj = -1;
    bool ok = true;
    __device__ __forceinline__ bool test(const DeviceScene& S, int32_t o_id, f3 o, f3 d) {
        if (o_id == obj) return ok;
        obj = o_id;
        float4 lo = __ldg(&S.objects[o_id].lo);
        if (lo.w == 0.0f) { ok = true; return true; }
        float4 hi = __ldg(&S.objects[o_id].hi);
        ok = ref_box_hit(lo, hi, o, d);
        return ok;
    }
};

struct TraceCounters {
    uint32_t nodes = 0, tris = 0;
};

// Normal and object of a closest-hit primitive at the hit point P
// (TriangleDetail.h:52, SphereDetail.h:64, QuadDetail.h:50, PlaneDetail.h:40).
__device__ __forceinline__ void hit_normal(const DeviceScene& S, int32_t prim, f3 P, f3& N, int32_t& obj) {
    const uint32_t slot = prim_slot(prim);
    switch (prim_type(prim)) {
        case 0:
            N = xyz(__ldg(&S.tri_n[slot]));
            obj = __float_as_int(__ldg(&S.tris[3 * (size_t)slot + 1]).w);
            break;
        case 1: {
            float4 s0 = __ldg(&S.spheres[2 * (size_t)slot]);
            N = normalize(P - xyz(s0));
            obj = __float_as_int(__ldg(&S.spheres[2 * (size_t)slot + 1]).z);
            break;
        }
        case 2:
            N = xyz(__ldg(&S.quads[4 * (size_t)slot + 1]));
            obj = __ldg(&S.quad_obj[slot]);
            break;
        default: {
            float4 p1 = __ldg(&S.planes[2 * (size_t)slot + 1]);
            N = xyz(p1);
            obj = __float_as_int(p1.w);
            break;
        }
    }
}

// Tracing::traceRay(scene, ray, index) (TracingDetail.h:68-116): the one
// object's own intersection, no box test; a mesh keeps its first strictly
// nearer triangle (MeshDetail.h:28-35).  t = INF when nothing is hit.
__device__ __forceinline__ bool trace_object(const DeviceScene& S, int32_t obj, f3 o, f3 d, float& t, f3& N) {
    const int4 info = __ldg(&S.obj_info[obj]);
    const float INF = __int_as_float(0x7f800000);
    t = INF;
    switch (info.x) {
        case 3:
        case 4: {  // TRIANGLE, MESH
            bool any = false;
            for (int k = 0; k < info.z; ++k) {
                const uint32_t s = __ldg(&S.key_slot[info.y + k]);
                const float4* p = S.tris + 3 * (size_t)s;
                float tt;
                if (isect_tri(__ldg(p), __ldg(p + 1), __ldg(p + 2), o, d, tt) && tt < t) {
                    t = tt;
                    N = xyz(__ldg(&S.tri_n[s]));
                    any = true;
                }
            }
            return any;
        }
        case 0: {  // SPHERE
            const uint32_t s = __ldg(&S.key_slot[info.y]);
            float4 s0 = __ldg(&S.spheres[2 * (size_t)s]), s1 = __ldg(&S.spheres[2 * (size_t)s + 1]);
            float tt;
            if (!isect_sphere(s0, s1, o, d, tt)) return false;
            t = tt;
            N = normalize((o + tt * d) - xyz(s0));
            return true;
        }
        case 2: {  // QUAD
            const uint32_t s = __ldg(&S.key_slot[info.y]);
            const float4* p = S.quads + 4 * (size_t)s;
            float tt;
            if (!isect_quad(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3), o, d, tt)) return false;
            t = tt;
            N = xyz(__ldg(p + 1));
            return true;
        }
        default: {  // PLANE
            const uint32_t s = __ldg(&S.key_slot[info.y]);
            float4 p0 = __ldg(&S.planes[2 * (size_t)s]), p1 = __ldg(&S.planes[2 * (size_t)s + 1]);
            float tt;
            if (!isect_plane(p0, p1, o, d, tt)) return false;
            t = tt;
            N = xyz(p1);
            return true;
        }
    }
}

// The two float4s of one 32-byte row of a node (lo and hi bounds of one axis)
// in one 256-bit load (128-byte aligned nodes).
__device__ __forceinline__ void ld_row(const float4* p, float4& a, float4& b) {
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(__cvta_generic_to_global(p)));
}

__device__ __forceinline__ SlabRay slab_ray(f3 o, f3 d) { return slab_ray(o.x, o.y, o.z, d.x, d.y, d.z); }
__device__ __forceinline__ bool slab_walks(const SlabRay& r, f3 d) { return slab_walks(r, d.x, d.y, d.z); }

// Slab tests of a 4-wide node's children (t in [0, lim]): entry distances and
// which are hit.  The boxes come as centres and half extents, so entry and
// exit follow from the distance to the centre plane by one fused multiply-add
// each: 12 more of those per node than with the two planes of each slab, and
// 24 fewer minima and maxima, which run at half their rate and kept the
// integer / compare pipe 63 % busy (43 % now).  A node is read with three
// 256-bit loads and one of 128.  Packing two children into one
// fma.rn.f32x2 halves the multiply-adds again, but its operand pairs did not
// fit the register budget (1080p terrain 45.4 -> 47.8 ms).
struct Slab4 {
    float tn[4];
    bool hit[4];
    int32_t ref[4];
};
__device__ __forceinline__ Slab4 slab4(const float4* __restrict__ node, const SlabRay& r, float lim) {
    float4 cx, hx, cy, hy, cz, hz;
    ld_row(node, cx, hx);
    ld_row(node + 2, cy, hy);
    ld_row(node + 4, cz, hz);
    const int4 rf = __ldg(reinterpret_cast<const int4*>(node + 6));
    const float x[4] = {cx.x, cx.y, cx.z, cx.w}, ex[4] = {hx.x, hx.y, hx.z, hx.w};
    const float y[4] = {cy.x, cy.y, cy.z, cy.w}, ey[4] = {hy.x, hy.y, hy.z, hy.w};
    const float z[4] = {cz.x, cz.y, cz.z, cz.w}, ez[4] = {hz.x, hz.y, hz.z, hz.w};
    Slab4 s;
    s.ref[0] = rf.x; s.ref[1] = rf.y; s.ref[2] = rf.z; s.ref[3] = rf.w;
#pragma unroll
    for (int k = 0; k < 4; ++k) s.hit[k] = slab_child(x[k], ex[k], y[k], ey[k], z[k], ez[k], r, lim, s.tn[k]);
    return s;
}

// Traversal stacks.  An entry is (entry distance's bits, child reference):
// entry distances are >= 0, so their bits order as integers; occlusion rays
// keep the reference only.
constexpr int32_t KEY_MISS = 0x7fffffff;
// An entry can still hold a counted hit while its key is at most this.
__device__ __forceinline__ int32_t key_limit(float t_best) { return __float_as_int(t_best) & 0x7fffffff; }

struct LocalStack {
    int2 e[CUPBR_STACK_SIZE];
    int sp;
    __device__ __forceinline__ void clear() { sp = 0; }
    __device__ __forceinline__ bool empty() const { return sp == 0; }
    static constexpr int ROW = 1;
    __device__ __forceinline__ bool near3() const { return sp <= CUPBR_STACK_SIZE - 3; }
    __device__ __forceinline__ void put(int at, int32_t key, int32_t ref) { e[at] = make_int2(key, ref); }
    __device__ __forceinline__ void push(int32_t key, int32_t ref, bool& overflow) {
        if (sp < CUPBR_STACK_SIZE) e[sp++] = make_int2(key, ref);
        else overflow = true;
    }
    __device__ __forceinline__ int2 pop() { return e[--sp]; }
};

// Enters a node: `first` is the child to visit next (nearest first; any order
// for occlusion rays, where any counted hit ends the ray) and the other
// children hit are pushed far-to-near.  False when no child is hit.
template <bool ANY, typename Stack>
__device__ __forceinline__ bool visit4(const float4* __restrict__ node, const SlabRay& r, float lim, int32_t& first,
                                       Stack& st, bool& overflow) {
    const Slab4 s = slab4(node, r, lim);
    if (ANY) {
        const int lowest = s.hit[0] ? 0 : s.hit[1] ? 1 : s.hit[2] ? 2 : s.hit[3] ? 3 : -1;
        if (lowest < 0) return false;
        first = s.hit[0] ? s.ref[0] : s.hit[1] ? s.ref[1] : s.hit[2] ? s.ref[2] : s.ref[3];
        if (st.near3()) {
#pragma unroll
            for (int k = 3; k >= 1; --k)
                if (s.hit[k] && k != lowest) {
                    st.put(st.sp, 0, s.ref[k]);
                    st.sp += Stack::ROW;
                }
        } else {
            for (int k = 3; k >= 1; --k)
                if (s.hit[k] && k != lowest) st.push(0, s.ref[k], overflow);
        }
        return true;
    }
    int32_t k[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) k[c] = s.hit[c] ? __float_as_int(s.tn[c]) : KEY_MISS;
    int32_t k0 = k[0], k1 = k[1], k2 = k[2], k3 = k[3];
    int32_t r0 = s.ref[0], r1 = s.ref[1], r2 = s.ref[2], r3 = s.ref[3];
#define CUPBR_CSWAP(ka, ra, kb, rb)                        \
    {                                                      \
        const bool w_ = kb < ka;                           \
        const int32_t lo_ = min(ka, kb), rl_ = w_ ? rb : ra; \
        kb = max(ka, kb);                                  \
        rb = w_ ? ra : rb;                                 \
        ka = lo_;                                          \
        ra = rl_;                                          \
    }
    CUPBR_CSWAP(k0, r0, k1, r1)
    CUPBR_CSWAP(k2, r2, k3, r3)
    CUPBR_CSWAP(k0, r0, k2, r2)
    CUPBR_CSWAP(k1, r1, k3, r3)
    CUPBR_CSWAP(k1, r1, k2, r2)
#undef CUPBR_CSWAP
    if (k0 == KEY_MISS) return false;
    first = r0;
    if (st.near3()) {
        st.sp += (k3 != KEY_MISS ? 3 : k2 != KEY_MISS ? 2 : k1 != KEY_MISS ? 1 : 0) * Stack::ROW;
        if (k1 != KEY_MISS) st.put(st.sp - Stack::ROW, k1, r1);
        if (k2 != KEY_MISS) st.put(st.sp - 2 * Stack::ROW, k2, r2);
        if (k3 != KEY_MISS) st.put(st.sp - 3 * Stack::ROW, k3, r3);
    } else {
        if (k3 != KEY_MISS) st.push(k3, r3, overflow);
        if (k2 != KEY_MISS) st.push(k2, r2, overflow);
        if (k1 != KEY_MISS) st.push(k1, r1, overflow);
    }
    return true;
}

// Closest hit (ANY = false) or visibility (ANY = true).
//   closest: on return t_best / best_prim / best_key hold the winning hit
//            (t_best = INF, best_prim = HIT_NONE when nothing is hit).
//   any    : returns true when some counted hit has t <= t_limit.
// `overflow` is set when the traversal stack would overflow (the entry is
// dropped; the caller reports it as an error).
// trace_scene_rt takes ANY / COUNT at run time, for kernels that trace
// closest-hit and shadow rays from one call site (one copy of the loop in
// the instruction cache); with constant flags it folds to trace_scene.
__device__ __forceinline__ bool trace_scene_rt(bool ANY, bool COUNT, const DeviceScene& S, f3 o, f3 d, float t_limit,
                                               float& t_best, int32_t& best_prim, uint32_t& best_key, bool& overflow,
                                               TraceCounters& ctr) {
    RefBoxCache cache;
    t_best = ANY ? t_limit : __int_as_float(0x7f800000);
    best_prim = HIT_NONE;
    best_key = 0xFFFFFFFFu;

    // unbounded primitives (planes) are tested for every ray
    for (uint32_t i = 0; i < S.n_planes; ++i) {
        float4 p0 = __ldg(&S.planes[2 * i]), p1 = __ldg(&S.planes[2 * i + 1]);
        float t;
        if (isect_plane(p0, p1, o, d, t)) {
            uint32_t key = __float_as_uint(p0.w);
            if (ANY) {
                if (t <= t_limit) return true;
            } else if (t < t_best || (t == t_best && key < best_key)) {
                t_best = t; best_prim = prim_ref(3, i); best_key = key;
            }
        }
    }
    const SlabRay sr = slab_ray(o, d);
    if (S.n_nodes == 0 || !slab_walks(sr, d)) return ANY ? false : best_prim != HIT_NONE;

    LocalStack st;
    st.clear();
    int32_t cur = 0;
    // A well-formed tree visits every node at most once per ray; the bound
    // turns a malformed node array into a reported error instead of a hang.
    uint32_t guard = 2u * S.n_nodes + 64u;

    for (;;) {
        if (--guard == 0u) {
            overflow = true;
            return ANY ? false : best_prim != HIT_NONE;
        }
        if (cur >= 0) {
            if ((uint32_t)cur >= S.n_nodes) {  // corrupt reference: report and stop
                overflow = true;
                return ANY ? false : best_prim != HIT_NONE;
            }
            if (COUNT) ctr.nodes++;
            int32_t first;
            if (visit4<false>(S.nodes + BVH_NODE_F4 * (size_t)cur, sr, t_best, first, st, overflow)) {
                cur = first;
                continue;
            }
        } else {
            const uint32_t v = ~(uint32_t)cur;
            const uint32_t start = v >> 3, cnt = (v & 7u) + 1u;
            if (start < S.sphere_base) {
                for (uint32_t k = 0; k < cnt; ++k) {
                    const uint32_t s = start + k;
                    const float4* p = S.tris + 3 * (size_t)s;
                    float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
                    if (COUNT) ctr.tris++;
                    float t;
                    if (!isect_tri(a, b, c, o, d, t)) continue;
                    const int32_t obj = __float_as_int(b.w);
                    if (ANY) {
                        if (t <= t_limit && cache.test(S, obj, o, d)) return true;
                    } else {
                        const uint32_t key = __float_as_uint(a.w);
                        if ((t < t_best || (t == t_best && key < best_key)) && cache.test(S, obj, o, d)) {
                            t_best = t; best_prim = prim_ref(0, s); best_key = key;
                        }
                    }
                }
            } else if (start < S.quad_base) {
                for (uint32_t k = 0; k < cnt; ++k) {
                    const uint32_t s = start + k - S.sphere_base;
                    float4 s0 = __ldg(&S.spheres[2 * (size_t)s]), s1 = __ldg(&S.spheres[2 * (size_t)s + 1]);
                    float t;
                    if (!isect_sphere(s0, s1, o, d, t)) continue;
                    const int32_t obj = __float_as_int(s1.z);
                    if (ANY) {
                        if (t <= t_limit && cache.test(S, obj, o, d)) return true;
                    } else {
                        const uint32_t key = __float_as_uint(s0.w);
                        if ((t < t_best || (t == t_best && key < best_key)) && cache.test(S, obj, o, d)) {
                            t_best = t; best_prim = prim_ref(1, s); best_key = key;
                        }
                    }
                }
            } else {
                for (uint32_t k = 0; k < cnt; ++k) {
                    const uint32_t s = start + k - S.quad_base;
                    const float4* p = S.quads + 4 * (size_t)s;
                    float4 q0 = __ldg(p), q1 = __ldg(p + 1), q2 = __ldg(p + 2), q3 = __ldg(p + 3);
                    float t;
                    if (COUNT) ctr.tris++;
                    if (!isect_quad(q0, q1, q2, q3, o, d, t)) continue;
                    if (ANY) {
                        if (t <= t_limit) return true;
                    } else {
                        const uint32_t key = __float_as_uint(q0.w);
                        if (t < t_best || (t == t_best && key < best_key)) {
                            t_best = t; best_prim = prim_ref(2, s); best_key = key;
                        }
                    }
                }
            }
        }
        // pop the next entry that can still hold a counted hit
        const int32_t limit = key_limit(t_best);
        for (;;) {
            if (st.empty()) return ANY ? false : best_prim != HIT_NONE;
            const int2 e = st.pop();
            if (e.x <= limit) { cur = e.y; break; }
        }
    }
}

template <bool ANY, bool COUNT>
__device__ __forceinline__ bool trace_scene(const DeviceScene& S, f3 o, f3 d, float t_limit, float& t_best,
                                            int32_t& best_prim, uint32_t& best_key, bool& overflow,
                                            TraceCounters& ctr) {
    return trace_scene_rt(ANY, COUNT, S, o, d, t_limit, t_best, best_prim, best_key, overflow, ctr);
}

// ------------------------------------------------ resumable traversal ---
// State of one ray's traversal, so a persistent warp can advance its lanes
// step by step, hand finished lanes a new ray and resume the others.  Same
// tests and acceptance rules as trace_scene.  `cur` is an inner node (>= 0), a
// leaf's remaining primitives (< 0, as a child reference), or TRAV_IDLE.
// Occlusion rays keep their limit in t_best, which never shrinks for them.
constexpr int32_t TRAV_IDLE = 0x7fffffff;
struct TravState {
    f3 o, d;
    SlabRay r;
    float t_best;
    int32_t best_prim;
    uint32_t best_key;
    int32_t cur;
    bool hit;
    RefBoxCache cache;
};

template <bool ANY>
__device__ __forceinline__ void trav_init(const DeviceScene& S, TravState& s, f3 o, f3 d, float t_limit) {
    s.o = o;
    s.d = d;
    s.r = slab_ray(o, d);
    s.t_best = ANY ? t_limit : __int_as_float(0x7f800000);
    s.best_prim = HIT_NONE;
    s.best_key = 0xFFFFFFFFu;
    s.cur = S.n_nodes && slab_walks(s.r, d) ? 0 : TRAV_IDLE;
    s.hit = false;
    s.cache.obj = -1;
    s.cache.ok = true;
    for (uint32_t i = 0; i < S.n_planes; ++i) {
        float4 p0 = __ldg(&S.planes[2 * i]), p1 = __ldg(&S.planes[2 * i + 1]);
        float t;
        if (isect_plane(p0, p1, o, d, t)) {
            uint32_t key = __float_as_uint(p0.w);
            if (ANY) {
                if (t <= t_limit) { s.hit = true; s.cur = TRAV_IDLE; return; }
            } else if (t < s.t_best || (t == s.t_best && key < s.best_key)) {
                s.t_best = t; s.best_prim = prim_ref(3, i); s.best_key = key;
            }
        }
    }
}

// Accepts a candidate hit (t, key) of object obj (< 0: no finite box to ask):
// true when an occlusion ray is blocked by it.
template <bool ANY>
__device__ __forceinline__ bool trav_accept(const DeviceScene& S, TravState& s, float t, uint32_t key, int32_t obj,
                                            int32_t prim) {
    if (ANY) return t <= s.t_best && (obj < 0 || s.cache.test(S, obj, s.o, s.d));
    if ((t < s.t_best || (t == s.t_best && key < s.best_key)) && (obj < 0 || s.cache.test(S, obj, s.o, s.d))) {
        s.t_best = t;
        s.best_prim = prim;
        s.best_key = key;
    }
    return false;
}

// Tests the primitives of leaf v (start << 3 | count - 1, one type per leaf)
// against the ray of s; true when an occlusion ray is blocked.
template <bool ANY, bool COUNT>
__device__ __forceinline__ bool trav_leaf(const DeviceScene& S, TravState& s, uint32_t v, TraceCounters& ctr) {
    const uint32_t start = v >> 3, cnt = (v & 7u) + 1u;
    float t;
    if (start < S.sphere_base) {
        const float4* p = S.tris + 3 * (size_t)start;
        for (uint32_t k = 0; k < cnt; ++k, p += 3) {
            if (COUNT) ctr.tris++;
            const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2);
            if (isect_tri(a, b, c, s.o, s.d, t) &&
                trav_accept<ANY>(S, s, t, __float_as_uint(a.w), __float_as_int(b.w), prim_ref(0, start + k)))
                return true;
        }
    } else if (start < S.quad_base) {
        const uint32_t first = start - S.sphere_base;
        const float4* p = S.spheres + 2 * (size_t)first;
        for (uint32_t k = 0; k < cnt; ++k, p += 2) {
            if (COUNT) ctr.tris++;
            const float4 a = __ldg(p), b = __ldg(p + 1);
            if (isect_sphere(a, b, s.o, s.d, t) &&
                trav_accept<ANY>(S, s, t, __float_as_uint(a.w), __float_as_int(b.z), prim_ref(1, first + k)))
                return true;
        }
    } else {
        const uint32_t first = start - S.quad_base;
        const float4* p = S.quads + 4 * (size_t)first;
        for (uint32_t k = 0; k < cnt; ++k, p += 4) {
            if (COUNT) ctr.tris++;
            const float4 a = __ldg(p), b = __ldg(p + 1), c = __ldg(p + 2), d = __ldg(p + 3);
            // a quad's object box is infinite
            if (isect_quad(a, b, c, d, s.o, s.d, t) &&
                trav_accept<ANY>(S, s, t, __float_as_uint(a.w), -1, prim_ref(2, first + k)))
                return true;
        }
    }
    return false;
}

// ------------------------------------------------------ warp packets ---
// Coherent rays (a warp's camera rays over one pixel tile) walk the tree
// as one packet: the node sequence, the stack pointer and the node refs
// are the same in every lane, each lane keeps its own ray, entry
// distances and closest hit.  A child is visited when any lane's slab test
// accepts it, nearest first by the smallest entry distance over the lanes;
// a stack entry is resumed while any lane's own entry distance is still
// within its closest hit.  Because the builder inflated every box
// conservatively, a box that holds a primitive is never entered later than
// that primitive's hit distance, so a ray's closest hit does not depend on
// the order in which nodes are visited and extra leaves tested for other
// lanes cannot change it: each lane ends with the same hit as trace_scene.

// Slab tests of a 4-wide node for every lane (as visit4).  Returns false
// when no lane hits a child; otherwise `first` is the child with the
// nearest entry over the lanes and the other accepted children are pushed
// far-to-near with each lane's own entry distance (INF where it missed).
__device__ __forceinline__ bool packet_visit4(const float4* __restrict__ node, const SlabRay& sr, float lim,
                                              int32_t& first, int32_t* st_ref, float* st_t, int& sp, bool& overflow) {
    const unsigned full = 0xffffffffu;
    const float INF = __int_as_float(0x7f800000);
    const Slab4 s = slab4(node, sr, lim);
    int32_t r[4] = {s.ref[0], s.ref[1], s.ref[2], s.ref[3]};
    float key[4];
    uint32_t wk[4];  // nearest entry over the lanes, as ordered bits (INF: no lane)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        key[k] = s.hit[k] ? s.tn[k] : INF;
        // entry distances are >= 0 (a -0 clears to 0), so their bits order as the values
        wk[k] = __reduce_min_sync(full, __float_as_uint(key[k]) & 0x7fffffffu);
    }
#define CUPBR_PSWAP(a, b)                                                                \
    if (wk[b] < wk[a]) {                                                                 \
        const uint32_t tw = wk[a]; wk[a] = wk[b]; wk[b] = tw;                            \
        const float tk = key[a]; key[a] = key[b]; key[b] = tk;                           \
        const int32_t tr = r[a]; r[a] = r[b]; r[b] = tr;                                 \
    }
    CUPBR_PSWAP(0, 1)
    CUPBR_PSWAP(2, 3)
    CUPBR_PSWAP(0, 2)
    CUPBR_PSWAP(1, 3)
    CUPBR_PSWAP(1, 2)
#undef CUPBR_PSWAP
    const uint32_t inf_bits = 0x7f800000u;
    if (wk[0] >= inf_bits) return false;
    first = r[0];
#pragma unroll
    for (int k = 3; k >= 1; --k) {
        if (wk[k] >= inf_bits) continue;
        if (sp < CUPBR_STACK_SIZE) {
            st_ref[sp] = r[k];
            st_t[sp] = key[k];
            ++sp;
        } else {
            overflow = true;
        }
    }
    return true;
}

// Resumes the top stack entry that some lane can still use; false when the
// stack is empty.
__device__ __forceinline__ bool packet_pop(float t_best, const int32_t* st_ref, const float* st_t, int& sp,
                                           int32_t& cur) {
    while (sp > 0) {
        --sp;
        if (__any_sync(0xffffffffu, st_t[sp] <= t_best)) {
            cur = st_ref[sp];
            return true;
        }
    }
    return false;
}

}  // namespace cupbr_b200
