// A pose's neighbourhood: the triangles nearest its receiver, as a flat list that answers
// the ray queries of a path which stays near the sensor.
//
// In a dense scene most of a path's traversal finds the same place again: on the boxes
// workload (1 M triangles, about 57 overlapping boxes over any point) a segment is 5 cm long on
// average, yet a query descends through the 110-130 nodes whose boxes hold that point. All
// queries of a pose start there. So each pose gets the list of the 64 triangles whose bounding
// boxes are nearest its receiver, and the largest cube around the receiver that no other
// triangle's box reaches (with a margin). A segment inside the cube can only meet listed
// triangles: an occlusion query between two of its points, and a closest-hit query whose
// hit lies inside, are settled by the list; 96-98 % of them on the boxes scene with 64
// triangles (48: 95 %, 32: 91 %, 128: 98 %). A query that leaves the cube unanswered goes
// to the BVH as before. Every lane of a warp tests the same triangle at the same time
// (broadcast loads, no divergence), where a warp's lanes each walk the tree by themselves (14 of 32
// active).
//
// The list is grouped by plane, and a plane is tested first: the segment's end points on one
// side of it, both further than `eps`, and none of its triangles can be met. `eps` covers
// the rounding of tri_test, so that whatever tri_test would accept reaches it.
//
// Whole calls before -> after: 96 poses on 1 M triangles (14 M paths, 4 bounces) 91 -> 17.1 ms,
// 33 poses on 100 k triangles (reference phase) 17 -> 5.1 ms, 1999 short poses on 20 k
// triangles 19.9 -> 12.8 ms (of which 10 on the host). With 32, 48, 64 and 96 triangles, one
// plane each, the first of these took 28.5, 22.1, 19.3 and 20.5 ms; grouping by plane
// took 64 to 17.1. The lists take one warp per pose and 0.13 ms before the launch. Served
// mix (24 requests, two of three scenes dense) 31 -> 12 ms.
#pragma once
#include <math_constants.h>

#include "hsr_common.cuh"
#include "hsr_internal.h"
#include "hsr_traverse.cuh"

namespace hsr {

// Half the cube's edge where the nearest triangle that is not listed has its bounding box
// at Chebyshev distance `next` from the centre: less a margin for the rounding of hit points
// and of box corners formed from v0 + e.
__device__ __forceinline__ float local_half_edge(float next, f3 c) {
    return next - 1e-5f * (next + fmaxf(fabsf(c.x), fmaxf(fabsf(c.y), fabsf(c.z)))) - 1e-6f;
}

// A triangle's plane relative to the centre, and the margin its test needs: tri_test's
// distance comes from products of edges and of vertex differences with a few roundings
// each, so in terms of the distance to the plane its error is at most some 2^-22 of the
// lengths involved, magnified by how acute the triangle is; so is the error of the plane
// formed here in single precision. The margin is 2^-19 of them. A degenerate triangle gets the
// plane 0 = 0, which is always tested. The normal's largest component is positive.
__device__ __forceinline__ float4 local_plane(const DTri &T, f3 c, float h, float &eps) {
    const f3 e1 = mk3(T.e1.x, T.e1.y, T.e1.z), e2 = mk3(T.e2.x, T.e2.y, T.e2.z);
    const f3 v = mk3(T.v0.x - c.x, T.v0.y - c.y, T.v0.z - c.z);
    const f3 n = crs3(e1, e2);
    const float len = nrm3(n), l1 = nrm3(e1), l2 = nrm3(e2);
    float big = n.x;
    if (fabsf(n.y) > fabsf(big)) big = n.y;
    if (fabsf(n.z) > fabsf(big)) big = n.z;
    const float inv = len > 0.f ? (big < 0.f ? -1.f : 1.f) / len : 0.f;
    const f3 u = scl3(inv, n);
    const float acute = fminf(fmaxf(l1 * l2 * fabsf(inv), 1.f), 1e6f);
    eps = 2e-6f * (nrm3(v) + l1 + l2 + h) * acute;
    return make_float4(u.x, u.y, u.z, dot3(u, v));
}

// Whether two planes share a group: they are apart by less than local_merge_margin anywhere
// in the cube, which the pose's eps takes in.
__device__ __forceinline__ bool local_same_plane(float4 a, float4 b, float h) {
    return fabsf(a.x - b.x) <= 1e-6f && fabsf(a.y - b.y) <= 1e-6f && fabsf(a.z - b.z) <= 1e-6f &&
           fabsf(a.w - b.w) <= 1e-6f * h;
}
__device__ __forceinline__ float local_merge_margin(float h) { return 4e-6f * h; }

// Whether a point lies in the list's cube.
__device__ __forceinline__ bool local_holds(const LocalList &L, f3 p) {
    return fmaxf(fabsf(p.x - L.cx), fmaxf(fabsf(p.y - L.cy), fabsf(p.z - L.cz))) <= L.h;
}

// Closest hit of a ray that starts in the cube: the slot and its distance, or -1 where the
// list does not settle it (no listed triangle is hit before the ray leaves the cube).
__device__ __forceinline__ int closest_local(const LocalList &L, const DTri *__restrict__ tris, f3 o, f3 d,
                                             float &t_best) {
    const f3 q = mk3(o.x - L.cx, o.y - L.cy, o.z - L.cz);
    const float ex = (L.h - copysignf(1.f, d.x) * q.x) * fabsf(safe_inv(d.x));
    const float ey = (L.h - copysignf(1.f, d.y) * q.y) * fabsf(safe_inv(d.y));
    const float ez = (L.h - copysignf(1.f, d.z) * q.z) * fabsf(safe_inv(d.z));
    const float t_exit = fminf(ex, fminf(ey, ez)) * 0.999999f;
    const float eps = L.eps;
    t_best = t_exit;
    int best = -1, prim_best = 0x7fffffff;
#pragma unroll 4
    for (int j = 0; j < L.planes; ++j) {
        const float4 n = L.plane[j];
        const float s0 = __fmaf_rn(n.x, q.x, __fmaf_rn(n.y, q.y, __fmaf_rn(n.z, q.z, -n.w)));
        const float s1 = __fmaf_rn(n.x, d.x, __fmaf_rn(n.y, d.y, n.z * d.z));
        const float se = __fmaf_rn(s1, t_best, s0);
        if (fminf(s0, se) > eps || fmaxf(s0, se) < -eps) continue;
        for (int k = L.start[j]; k < L.start[j + 1]; ++k) {
            const int slot = L.slot[k];
            const DTri T = load_tri(tris, slot);
            float t;
            if (tri_test(T, o, d, kEpsilon, CUDART_INF_F, t) && t <= t_best) {
                const int prim = __float_as_int(T.v0.w);
                if (t < t_best || prim < prim_best) {
                    t_best = t;
                    prim_best = prim;
                    best = slot;
                }
            }
        }
    }
    return best;
}

// Any hit in (kEpsilon, dist] of the segment from a point of the cube to the receiver, the
// cube's centre.
__device__ __forceinline__ bool any_local(const LocalList &L, const DTri *__restrict__ tris, f3 o, f3 d, float dist) {
    const f3 q = mk3(o.x - L.cx, o.y - L.cy, o.z - L.cz);
    const float eps = L.eps;
#pragma unroll 4
    for (int j = 0; j < L.planes; ++j) {
        const float4 n = L.plane[j];
        const float s0 = __fmaf_rn(n.x, q.x, __fmaf_rn(n.y, q.y, __fmaf_rn(n.z, q.z, -n.w)));
        if (fminf(s0, -n.w) > eps || fmaxf(s0, -n.w) < -eps) continue;
        for (int k = L.start[j]; k < L.start[j + 1]; ++k) {
            const DTri T = load_tri(tris, L.slot[k]);
            float t;
            if (tri_test(T, o, d, kEpsilon, dist, t)) return true;
        }
    }
    return false;
}

}  // namespace hsr
