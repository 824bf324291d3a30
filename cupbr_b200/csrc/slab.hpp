// The slab test of the BVH's traversal: a ray against one child's box, given
// as centre and half extent (k_slab_nodes).  Plain C++ for the device and for
// the host, where a test goes through rays that are no numbers.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define CUPBR_SLAB __host__ __device__ __forceinline__
#else
#define CUPBR_SLAB inline
#endif

namespace cupbr_b200 {

CUPBR_SLAB float max3(float a, float b, float c) {
#ifdef __CUDA_ARCH__
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
#else
    return fmaxf(fmaxf(a, b), c);
#endif
}
CUPBR_SLAB float min3(float a, float b, float c) {
#ifdef __CUDA_ARCH__
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
#else
    return fminf(fminf(a, b), c);
#endif
}

CUPBR_SLAB float safe_inv(float v) { return 1.0f / (fabsf(v) > 1e-20f ? v : copysignf(1e-20f, v)); }

// A ray as the slab tests read it, per axis: 1 / d, o / d and |1 / d|.
struct SlabAxis {
    float i, o, a;
};
struct SlabRay {
    SlabAxis x, y, z;
};
CUPBR_SLAB SlabAxis slab_axis_of(float o, float d) {
    SlabAxis s;
    s.i = safe_inv(d);
    s.o = o * s.i;
    s.a = fabsf(s.i);
    return s;
}
CUPBR_SLAB SlabRay slab_ray(float ox, float oy, float oz, float dx, float dy, float dz) {
    return {slab_axis_of(ox, dx), slab_axis_of(oy, dy), slab_axis_of(oz, dz)};
}
// Whether the ray may walk a tree.  A missing child has centre 0 and half
// extent -inf: an axis of finite o / d and finite d turns it down (entry +inf,
// exit -inf) whatever the other axes say.  Minima and maxima drop a NaN, so
// where no axis does -- an origin of NaN -- a missing child would be entered,
// and its reference leads out of the tables.  A ray with o / d not finite on
// some axis meets no primitive: its distances are NaN, or it runs outside the
// slab.  Asked once per ray, which costs nothing that can be measured (1080p
// terrain 36.88 -> 36.85 ms, Cornell box 7.911 -> 7.913); a bounds check of the leaf instead takes
// 1.5 %, an axis made to turn down every child 1 to 2 %.
CUPBR_SLAB bool slab_walks(const SlabRay& r, float dx, float dy, float dz) {
    return fabsf(r.x.o) < INFINITY && fabsf(r.y.o) < INFINITY && fabsf(r.z.o) < INFINITY &&
           min3(fabsf(dx), fabsf(dy), fabsf(dz)) < INFINITY;
}

// Whether the ray (slab_walks) is inside the box somewhere in [0, lim], and where it enters.
CUPBR_SLAB bool slab_child(float cx, float hx, float cy, float hy, float cz, float hz, const SlabRay& r, float lim,
                           float& entry) {
    const float mx = fmaf(cx, r.x.i, -r.x.o), my = fmaf(cy, r.y.i, -r.y.o), mz = fmaf(cz, r.z.i, -r.z.o);
    entry = fmaxf(max3(fmaf(-hx, r.x.a, mx), fmaf(-hy, r.y.a, my), fmaf(-hz, r.z.a, mz)), 0.0f);
    const float exit = fminf(min3(fmaf(hx, r.x.a, mx), fmaf(hy, r.y.a, my), fmaf(hz, r.z.a, mz)), lim);
    return entry <= exit;
}

}  // namespace cupbr_b200
