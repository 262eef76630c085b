// Device side of the four-wide mesh BVH (wide_bvh.h): one node's children
// against a ray.
#pragma once
#include "tracer_core.cuh"

namespace slim {
namespace dev {

// A ray as the wide walk takes it: the reciprocal direction, and -o * rcp
// with the margin for the planes a ray meets first and last.  The exact test
// rounds plane * rcp + so once; here so -+ margin, origin * rcp + that and
// offset * rcp + that round, all four by at most 2^-24 (extent |rcp| + |so|):
// a margin of eight such units makes every box hit here that the exact test
// hits.
//
// Along an axis the ray is parallel to (an infinite reciprocal) the exact
// test's distances are infinite or NaN, and a NaN leaves the axis out of the
// comparisons: boxes far beside the ray count as hit, though none of their
// triangles is.  The walk takes 1e18 for the reciprocal there, which keeps
// to the boxes beside the ray, and a margin 32 times as wide, against the
// rounding of the triangle tests; a leaf's own box is still tested exactly.
struct WideRay {
    float3 near, far;
    bool parallel;
};
SLIM_D void wide_axis(float o, float rcp, float so, float extent, float &r, float &near, float &far, bool &parallel) {
    const bool along = !(fabsf(rcp) < 1e18f);
    r = along ? copysignf(1e18f, rcp) : rcp;
    const float s = along ? -o * r : so;
    const float e = fmaf(extent, fabsf(r), fabsf(s)) * (along ? 0x1p-16f : 0x1p-21f);
    near = s - e;
    far = s + e;
    parallel |= along;
}
SLIM_D WideRay wide_setup(Ray &r, float extent) {     // r.rcp becomes the walk's
    WideRay w;
    w.parallel = false;
    wide_axis(r.o.x, r.rcp.x, r.so.x, extent, r.rcp.x, w.near.x, w.far.x, w.parallel);
    wide_axis(r.o.y, r.rcp.y, r.so.y, extent, r.rcp.y, w.near.y, w.far.y, w.parallel);
    wide_axis(r.o.z, r.rcp.z, r.so.z, extent, r.rcp.z, w.near.z, w.far.z, w.parallel);
    return w;
}

// Four children of wide node i against the ray: bit s of the result is set
// when box s is hit before tmax, between t0[s] and t1[s].
SLIM_D uint32_t wide_hits(const uint4 *nodes, uint32_t i, const Ray &r, const WideRay &w, float tmax,
                          uint32_t child[4], float t0[4], float t1[4]) {
    const uint4 *n = nodes + 5 * (size_t)i;
    const uint4 a = __ldg(n), b = __ldg(n + 1), c = __ldg(n + 2), d = __ldg(n + 3), e = __ldg(n + 4);
    child[0] = b.x;
    child[1] = b.y;
    child[2] = b.z;
    child[3] = b.w;
    const float3 org = f3(__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z));
    const float3 near = mul_add(org, r.rcp, w.near), far = mul_add(org, r.rcp, w.far);
    const uint32_t nx[2] = {r.nx ? d.z : c.x, r.nx ? d.w : c.y}, fx[2] = {r.nx ? c.x : d.z, r.nx ? c.y : d.w};
    const uint32_t ny[2] = {r.ny ? e.x : c.z, r.ny ? e.y : c.w}, fy[2] = {r.ny ? c.z : e.x, r.ny ? c.w : e.y};
    const uint32_t nz[2] = {r.nz ? e.z : d.x, r.nz ? e.w : d.y}, fz[2] = {r.nz ? d.x : e.z, r.nz ? d.y : e.w};
    uint32_t missed = 0;
#pragma unroll
    for (int s = 3; s >= 0; s--) {
        auto plane = [&](const uint32_t v[2]) { return __uint_as_float(s & 1 ? v[s >> 1] : v[s >> 1] << 16); };
        t0[s] = fmaxf(max3(fmaf(plane(nx), r.rcp.x, near.x), fmaf(plane(ny), r.rcp.y, near.y),
                           fmaf(plane(nz), r.rcp.z, near.z)), 0.0f);
        t1[s] = fminf(min3(fmaf(plane(fx), r.rcp.x, far.x), fmaf(plane(fy), r.rcp.y, far.y),
                           fmaf(plane(fz), r.rcp.z, far.z)), tmax);
        missed = __funnelshift_l(__float_as_uint(t1[s] - t0[s]), missed, 1);   // the difference's sign
    }
    return missed ^ 0xFu;
}

// The exact test of a leaf's box.
SLIM_D bool wide_leaf_box(const Ray &r, const WideRay &w, float4 a, float4 b, float &near, float &far) {
    if (!w.parallel) return hit_box_finite(r, a, b, near, far);
    Ray exact;
    reset(exact, r.o, r.d);
    return hit_node(exact, a, b, near, far);
}

}  // namespace dev
}  // namespace slim
