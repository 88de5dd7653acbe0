// CPU check of the neighbourhood lists' queries, compiled from the product's own header
// (hussar_gb300/csrc/hsr_local.cuh) with host definitions of the CUDA intrinsics
// (host_shim.h). The list of a centre is formed here by brute force (the kLocalTris triangles
// nearest in Chebyshev distance of their bounding boxes, planes and margins by the header's own
// functions); its answers are compared with brute force over every triangle of the mesh,
// same triangle test and tie rule.
//
// Input (binary, little endian): int64 nv, nt, nr; float v[nv][3]; int32 idx[nt][3]; float
// c[3]; per ray 3 + 3 + 1 uniform numbers: origin within the cube [-1, 1]^3 (scaled by the
// cube found), direction, and whether the origin moves onto the nearest triangle hit.
// Output: "half H planes P settled S wrong W missed M any_wrong A occluded O".
#include "host_shim.h"
#include "hsr_local.cuh"

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <vector>

using namespace hsr;

static float axis_gap(float c, float lo, float hi) { return std::max(0.f, std::max(lo - c, c - hi)); }

int main(int argc, char **argv) {
    FILE *f = std::fopen(argv[1], "rb");
    if (!f || argc < 2) return 1;
    int64_t n[3];
    if (std::fread(n, 8, 3, f) != 3) return 1;
    std::vector<float> v(3 * n[0]), rays(7 * n[2]);
    std::vector<int32_t> idx(3 * n[1]);
    float c3[3];
    if (std::fread(v.data(), 4, v.size(), f) != v.size() || std::fread(idx.data(), 4, idx.size(), f) != idx.size() ||
        std::fread(c3, 4, 3, f) != 3 || std::fread(rays.data(), 4, rays.size(), f) != rays.size())
        return 1;
    std::fclose(f);
    const f3 c = mk3(c3[0], c3[1], c3[2]);
    const int nt = int(n[1]);
    std::vector<DTri> tris(nt);
    std::vector<std::pair<float, int>> order(nt);
    for (int i = 0; i < nt; ++i) {
        const float *a = &v[3 * idx[3 * i]], *b = &v[3 * idx[3 * i + 1]], *d = &v[3 * idx[3 * i + 2]];
        DTri T;
        T.v0 = make_float4(a[0], a[1], a[2], __int_as_float(i));
        T.e1 = make_float4(b[0] - a[0], b[1] - a[1], b[2] - a[2], 0.f);
        T.e2 = make_float4(d[0] - a[0], d[1] - a[1], d[2] - a[2], 0.f);
        tris[i] = T;
        float dist = 0.f;
        for (int k = 0; k < 3; ++k)
            dist = std::max(dist, axis_gap(c3[k], std::min(a[k], std::min(b[k], d[k])),
                                           std::max(a[k], std::max(b[k], d[k]))));
        order[i] = {dist, i};
    }
    std::sort(order.begin(), order.end());
    LocalList L{};
    L.cx = c.x;
    L.cy = c.y;
    L.cz = c.z;
    L.h = local_clear(order[kLocalTris].first, c);
    std::vector<std::vector<int>> group;
    for (int j = 0; j < kLocalTris; ++j) {
        const float4 pl = local_tri(tris[order[j].second], c, L.h).plane;
        size_t g = 0;
        while (g < group.size() && !local_same_plane(L.plane[g], pl, L.h)) ++g;
        if (g == group.size()) {
            L.plane[g] = pl;
            L.range[g].y = local_clear(order[j].first, c);
            group.emplace_back();
        }
        group[g].push_back(order[j].second);
    }
    L.planes = int(group.size());
    int at = 0;
    for (size_t g = 0; g < group.size(); ++g) {
        L.start[g] = (unsigned char)at;
        float eps = 0.f;
        for (int s : group[g]) {
            const LocalTri t = local_tri(tris[s], c, L.h);
            L.u[at] = t.u;
            L.v[at] = t.v;
            L.uv_eps[at] = t.uv_eps;
            eps = std::max(eps, t.plane_eps);
            L.slot[at++] = s;
        }
        L.range[g].x = eps + local_merge_margin(L.h);
    }
    L.start[group.size()] = (unsigned char)at;
    for (int j = L.planes; j % kLocalGroup; ++j) local_fill(L, j);

    long settled = 0, wrong = 0, missed = 0, any_wrong = 0, occluded = 0;
    auto brute = [&](f3 o, f3 d, float &t_best) {
        int best = -1;
        t_best = CUDART_INF_F;
        for (int i = 0; i < nt; ++i) {
            float t;
            if (tri_test(tris[i], o, d, kEpsilon, CUDART_INF_F, t) && (t < t_best || (t == t_best && i < best))) {
                t_best = t;
                best = i;
            }
        }
        return best;
    };
    for (int64_t r = 0; L.h > 0.f && r < n[2]; ++r) {
        const float *q = &rays[7 * r];
        f3 o = mk3(c.x + q[0] * L.h, c.y + q[1] * L.h, c.z + q[2] * L.h), d = mk3(q[3], q[4], q[5]);
        if (!local_holds(L, o)) o = c;
        float tb, tl;
        if (q[6] > 0.5f) {  // from a surface, as a path's later segments
            const int s = brute(o, d, tb);
            const f3 hp = add3(o, scl3(tb, d));
            if (s >= 0 && local_holds(L, hp)) {
                const f3 nn = hit_normal(tris[s], d);
                o = hp;
                d = sub3(d, scl3(2.f * dot3(nn, d), nn));
            }
        }
        const int best = brute(o, d, tb);
        const int slot = closest_local(L, tris.data(), o, d, tl);
        const f3 hp = add3(o, scl3(tb * 1.00001f, d));
        if (slot >= 0) {
            ++settled;
            wrong += slot != best || tl != tb;
        } else if (best >= 0) {
            f3 inner = sub3(hp, c);
            missed += std::max(std::fabs(inner.x), std::max(std::fabs(inner.y), std::fabs(inner.z))) < 0.9999f * L.h;
        }
        f3 to = sub3(c, o);
        const float dist = nrm3(to);
        if (dist > 0.f) {
            to = div3(to, dist);
            bool any = false;
            for (int i = 0; i < nt && !any; ++i) {
                float t;
                any = tri_test(tris[i], o, to, kEpsilon, dist, t);
            }
            occluded += any;
            any_wrong += any != any_local(L, tris.data(), o, to, dist);
        }
    }
    std::printf("half %g planes %d settled %ld wrong %ld missed %ld any_wrong %ld occluded %ld\n", double(L.h), L.planes,
                settled, wrong, missed, any_wrong, occluded);
    return 0;
}
