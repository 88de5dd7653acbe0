// A pose's neighbourhood: the triangles nearest its receiver, as a flat list that answers
// the ray queries of a path which stays near the sensor.
//
// In a dense scene most of a path's traversal finds the same place again: on the boxes
// workload (1 M triangles, about 57 overlapping boxes over any point) a segment is 5 cm long on
// average, yet a query descends through the 110-130 nodes whose boxes hold that point. All
// queries of a pose start there. So each pose gets the list of the 96 triangles whose bounding
// boxes are nearest its receiver, and the largest cube around the receiver that no other
// triangle's box reaches (with a margin). A segment inside the cube can only meet listed
// triangles: an occlusion query between two of its points, and a closest-hit query whose
// hit lies inside, are settled by the list; 98-99 % of them on the boxes scene (64 triangles:
// 97 %, 32: 91 %). A query that leaves the cube unanswered goes to the BVH as before. Every
// lane of a warp tests the same triangle at the same time (broadcast loads, no divergence),
// where a warp's lanes each walk the tree by themselves (14 of 32 active).
//
// The list is grouped by plane, nearest group first, and a query ends at the first group
// further out than its segment reaches, which shrinks with every hit found. A plane is
// tested first: the segment's end points on one side of it, both further than its margin,
// and none of its triangles can be met. Where the plane is crossed, the crossing's
// barycentric coordinates in its triangles, from two more dot products each, tell hits from
// misses, again with margins that cover the rounding of tri_test. Only what lies within the
// margins, and a ray's final candidate, goes through tri_test itself, whose distance is the
// answer.
//
// Whole calls without and with the lists: 96 poses on 1 M triangles (14 M paths, 4 bounces) 91
// and 13.3 ms, 33 poses on 100 k triangles (reference phase) 17 and 3.7 ms, 1999 short poses on
// 20 k triangles 19.9 (9 of it on the host) and 4.2 ms, served mix of 24 requests (two of three
// scenes dense) 31 and 8.8 ms. On the first two: 128 triangles 13.1 and 3.7; one plane at a
// time instead of groups of 8 (kLocalGroup) 14.5 and 4.0, and so with 64 triangles 15.3 and
// 4.4; every triangle of 64 through tri_test 19.3 and 5.6. The lists take one warp per pose and
// 85 us before the launch.
#pragma once
#include <math_constants.h>

#include "hsr_common.cuh"
#include "hsr_internal.h"
#include "hsr_traverse.cuh"

namespace hsr {

// How far from the centre a point can lie and surely be outside a bounding box at Chebyshev
// distance `dist` from it: less a margin for the rounding of hit points and of box corners
// formed from v0 + e. With the nearest triangle that is not listed, half the cube's edge.
__device__ __forceinline__ float local_clear(float dist, f3 c) {
    return dist - 1e-5f * (dist + fmaxf(fabsf(c.x), fmaxf(fabsf(c.y), fabsf(c.z)))) - 1e-6f;
}

// Chebyshev distance from the centre.
__device__ __forceinline__ float local_radius(f3 q) { return fmaxf(fabsf(q.x), fmaxf(fabsf(q.y), fabsf(q.z))); }

// A triangle's plane and coordinates relative to the centre, and their margins: tri_test's
// distance comes from products of edges and of vertex differences with a few roundings each,
// so in terms of the distance to the plane its error is at most some 2^-22 of the lengths
// involved, magnified by how acute the triangle is; so is the error of what is formed here
// in single precision. The margin is 2^-19 of them, and that distance over the triangle's
// heights for its coordinates. A degenerate triangle gets the plane 0 = 0, which is always
// crossed, at no number. The normal's largest component is positive.
struct LocalTri {
    float4 plane, u, v;
    float plane_eps, uv_eps;
};

__device__ __forceinline__ LocalTri local_tri(const DTri &T, f3 c, float h) {
    const f3 e1 = mk3(T.e1.x, T.e1.y, T.e1.z), e2 = mk3(T.e2.x, T.e2.y, T.e2.z);
    const f3 v = mk3(T.v0.x - c.x, T.v0.y - c.y, T.v0.z - c.z);
    const f3 n = crs3(e1, e2);
    const float len = nrm3(n), l1 = nrm3(e1), l2 = nrm3(e2);
    float big = n.x;
    if (fabsf(n.y) > fabsf(big)) big = n.y;
    if (fabsf(n.z) > fabsf(big)) big = n.z;
    const float size = len > 0.f ? 1.f / len : 0.f;
    const f3 unit = scl3(size, n);
    // u = (p - v0) . (e2 x n) / |n|^2, v = (p - v0) . (n x e1) / |n|^2
    const f3 nu = scl3(size, crs3(e2, unit)), nv = scl3(size, crs3(unit, e1));
    const f3 facing = scl3(big < 0.f ? -1.f : 1.f, unit);
    const float acute = fminf(fmaxf(l1 * l2 * size, 1.f), 1e6f);
    LocalTri t;
    t.plane = make_float4(facing.x, facing.y, facing.z, dot3(facing, v));
    t.u = make_float4(nu.x, nu.y, nu.z, dot3(nu, v));
    t.v = make_float4(nv.x, nv.y, nv.z, dot3(nv, v));
    t.plane_eps = 2e-6f * (nrm3(v) + l1 + l2 + h) * acute;
    t.uv_eps = 2.f * fmaxf(nrm3(nu), nrm3(nv)) * t.plane_eps + 1e-6f;
    return t;
}

// Whether two planes share a group: they are apart by less than local_merge_margin anywhere
// in the cube, which the margins take in.
__device__ __forceinline__ bool local_same_plane(float4 a, float4 b, float h) {
    return fabsf(a.x - b.x) <= 1e-6f && fabsf(a.y - b.y) <= 1e-6f && fabsf(a.z - b.z) <= 1e-6f &&
           fabsf(a.w - b.w) <= 1e-6f * h;
}
__device__ __forceinline__ float local_merge_margin(float h) { return 4e-6f * h; }

// Whether a point lies in the list's cube.
__device__ __forceinline__ bool local_holds(const LocalList &L, f3 p) {
    return fmaxf(fabsf(p.x - L.cx), fmaxf(fabsf(p.y - L.cy), fabsf(p.z - L.cz))) <= L.h;
}

// 1 / x within 2 ulps (0: infinite).
__device__ __forceinline__ float local_inverse(float x) {
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.f / x;
#endif
}

__device__ __forceinline__ int local_lowest(unsigned m) { return __ffs(int(m)) - 1; }

// Planes are tested kLocalGroup at a time for being crossed at all; then each lane takes the
// ones it crosses one by one, its own at the same time as the other lanes theirs (groups of
// 4: 13.2 and 3.8 ms on the workloads above, of 16: 13.4 and 3.7). The list is filled up to
// whole groups with planes that are never crossed.
constexpr int kLocalGroup = 8;
static_assert(kLocalTris % kLocalGroup == 0, "whole groups");
__device__ __forceinline__ void local_fill(LocalList &L, int j) {
    L.plane[j] = make_float4(0.f, 0.f, 0.f, 1.f);
    L.range[j] = make_float2(0.f, CUDART_INF_F);
}

// Where a point of its plane lies in triangle k: -1 outside, 1 inside, 0 too near an edge (or
// no number) to tell. `scale`: the coordinates' margin in units of the list's.
__device__ __forceinline__ int local_inside(const LocalList &L, int k, f3 p, float scale) {
    const float4 a = L.u[k], b = L.v[k];
    const float u = __fmaf_rn(a.x, p.x, __fmaf_rn(a.y, p.y, __fmaf_rn(a.z, p.z, -a.w)));
    const float v = __fmaf_rn(b.x, p.x, __fmaf_rn(b.y, p.y, __fmaf_rn(b.z, p.z, -b.w)));
    const float m = L.uv_eps[k] * scale;
    const float least = fminf(u, fminf(v, 1.f - (u + v)));
    return least < -m ? -1 : least > m ? 1 : 0;
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
    t_best = t_exit;
    int best = -1, prim_best = 0x7fffffff;
    auto verify = [&](int slot) {
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
    };
    // The candidate: a sure hit at about `near` (within `slack`), nearer than any sure hit
    // before it. What cannot be told from it, or is no sure hit, is verified at once.
    int cand = -1;
    float near = t_exit, slack = 0.f;
    const float from = local_radius(q);
    float reach = L.h;  // of the segment up to `near`: what lies further out cannot be met
    for (int j0 = 0; j0 < L.planes && !(L.range[j0].y > reach); j0 += kLocalGroup) {
        unsigned crossed = 0;
#pragma unroll 4
        for (int k = 0; k < kLocalGroup; ++k) {
            const float4 n = L.plane[j0 + k];
            const float eps = L.range[j0 + k].x;
            const float s0 = __fmaf_rn(n.x, q.x, __fmaf_rn(n.y, q.y, __fmaf_rn(n.z, q.z, -n.w)));
            const float s1 = __fmaf_rn(n.x, d.x, __fmaf_rn(n.y, d.y, n.z * d.z));
            const float se = __fmaf_rn(s1, near + slack, s0);
            if (!(fminf(s0, se) > eps || fmaxf(s0, se) < -eps)) crossed |= 1u << k;
        }
        for (; crossed; crossed &= crossed - 1) {
            const int j = j0 + local_lowest(crossed);
            const float4 n = L.plane[j];
            const float s0 = __fmaf_rn(n.x, q.x, __fmaf_rn(n.y, q.y, __fmaf_rn(n.z, q.z, -n.w)));
            const float s1 = __fmaf_rn(n.x, d.x, __fmaf_rn(n.y, d.y, n.z * d.z));
            const float inv = local_inverse(s1), steep = fabsf(inv);
            const float t = -s0 * inv, tol = 2.f * L.range[j].x * steep;
            if (t < kEpsilon - tol || t > near + slack + tol) continue;
            const f3 p = mk3(__fmaf_rn(t, d.x, q.x), __fmaf_rn(t, d.y, q.y), __fmaf_rn(t, d.z, q.z));
            for (int k = L.start[j]; k < L.start[j + 1]; ++k) {
                const int in = local_inside(L, k, p, 1.f + steep);
                if (in < 0) continue;
                if (in > 0 && t > kEpsilon + tol && t + tol < near - slack) {
                    cand = L.slot[k];
                    near = t;
                    slack = tol;
                    reach = fmaxf(from, local_radius(p)) + tol;
                } else {
                    verify(L.slot[k]);
                    if (t_best < near) {
                        near = t_best;
                        slack = 0.f;
                    }
                }
            }
        }
    }
    if (cand >= 0) verify(cand);
    return best;
}

// Any hit in (kEpsilon, dist] of the segment from a point of the cube to the receiver, the
// cube's centre.
__device__ __forceinline__ bool any_local(const LocalList &L, const DTri *__restrict__ tris, f3 o, f3 d, float dist) {
    const f3 q = mk3(o.x - L.cx, o.y - L.cy, o.z - L.cz);
    const float reach = local_radius(q);
    for (int j0 = 0; j0 < L.planes && !(L.range[j0].y > reach); j0 += kLocalGroup) {
        unsigned crossed = 0;
#pragma unroll 4
        for (int k = 0; k < kLocalGroup; ++k) {
            const float4 n = L.plane[j0 + k];
            const float eps = L.range[j0 + k].x;
            const float s0 = __fmaf_rn(n.x, q.x, __fmaf_rn(n.y, q.y, __fmaf_rn(n.z, q.z, -n.w)));
            if (!(fminf(s0, -n.w) > eps || fmaxf(s0, -n.w) < -eps)) crossed |= 1u << k;
        }
        for (; crossed; crossed &= crossed - 1) {
            const int j = j0 + local_lowest(crossed);
            const float4 n = L.plane[j];
            const float s0 = __fmaf_rn(n.x, q.x, __fmaf_rn(n.y, q.y, __fmaf_rn(n.z, q.z, -n.w)));
            const float s1 = __fmaf_rn(n.x, d.x, __fmaf_rn(n.y, d.y, n.z * d.z));
            const float inv = local_inverse(s1), steep = fabsf(inv);
            const float t = -s0 * inv, tol = 2.f * L.range[j].x * steep;
            if (t < kEpsilon - tol || t > dist + tol) continue;
            const f3 p = mk3(__fmaf_rn(t, d.x, q.x), __fmaf_rn(t, d.y, q.y), __fmaf_rn(t, d.z, q.z));
            for (int k = L.start[j]; k < L.start[j + 1]; ++k) {
                const int in = local_inside(L, k, p, 1.f + steep);
                if (in < 0) continue;
                if (in > 0 && t > kEpsilon + tol && t < dist - tol) return true;
                float th;
                if (tri_test(load_tri(tris, L.slot[k]), o, d, kEpsilon, dist, th)) return true;
            }
        }
    }
    return false;
}

}  // namespace hsr
