// The neighbourhood lists that the device builds (k_local_build in
// hussar_gb300/csrc/hsr_local.cu, through the library's own launch) against lists formed here
// by brute force over the scene's triangles: which triangles, in which order of planes, the
// cube, and whether the list is kept at all. The functions that form planes and answer queries
// are the product's header's, with host definitions of the CUDA intrinsics (host_shim.h).
//
// Input (binary, little endian): int64 nv, nt, np; float v[nv][3]; int32 idx[nt][3]; per pose
// float tx[3], rx[3]. Output per pose: "planes P want W near N wrong X": planes of the device's
// list (0: none), of the one formed here, rays of 32 that one settles, and what differs (0: nothing).
#include "host_shim.h"
#include "hsr_local.cuh"

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <vector>

using namespace hsr;

static float axis_gap(float c, float lo, float hi) { return std::max(0.f, std::max(lo - c, c - hi)); }

static bool near_equal(float a, float b, float scale) { return std::fabs(a - b) <= 2e-6f * scale; }

int main(int argc, char **argv) {
    FILE *f = argc > 1 ? std::fopen(argv[1], "rb") : nullptr;
    int64_t n[3];
    if (!f || std::fread(n, 8, 3, f) != 3) return 1;
    std::vector<float> v(3 * n[0]), pos(6 * n[2]);
    std::vector<int32_t> idx(3 * n[1]);
    if (std::fread(v.data(), 4, v.size(), f) != v.size() || std::fread(idx.data(), 4, idx.size(), f) != idx.size() ||
        std::fread(pos.data(), 4, pos.size(), f) != pos.size())
        return 1;
    std::fclose(f);
    const int P = int(n[2]), nt = int(n[1]);
    hsr_scene *scene = nullptr;
    if (hsr_scene_create(v.data(), n[0], idx.data(), nt, &scene) != HSR_OK) return 2;
    const SceneDev *dev = scene_device_state(scene);
    std::vector<DTri> tris(nt);
    if (hsr_debug_bvh(scene, nullptr, 0, tris.data(), nt) != HSR_OK) return 2;
    std::vector<hsr_antenna> ant(2 * P);
    for (int p = 0; p < P; ++p)
        for (int k = 0; k < 3; ++k) {
            ant[p].position[k] = pos[6 * p + k];
            ant[P + p].position[k] = pos[6 * p + 3 + k];
        }
    hsr_antenna *d_ant = nullptr;
    LocalList *d_list = nullptr;
    std::vector<LocalList> lists(P);
    TraceParams tp{};
    if (cudaMalloc(&d_ant, sizeof(hsr_antenna) * ant.size()) != cudaSuccess ||
        cudaMalloc(&d_list, sizeof(LocalList) * P) != cudaSuccess ||
        cudaMemcpy(d_ant, ant.data(), sizeof(hsr_antenna) * ant.size(), cudaMemcpyHostToDevice) != cudaSuccess)
        return 2;
    tp.nodes = dev->nodes;
    tp.tris = dev->tris;
    tp.tx = d_ant;
    tp.rx = d_ant + P;
    tp.pose_count = P;
    if (launch_local_build(tp, dev->local_radius, d_list, nullptr) != 0 ||
        cudaMemcpy(lists.data(), d_list, sizeof(LocalList) * P, cudaMemcpyDeviceToHost) != cudaSuccess)
        return 2;
    std::printf("radius %g\n", double(dev->local_radius));

    for (int p = 0; p < P; ++p) {
        const f3 s = mk3(pos[6 * p], pos[6 * p + 1], pos[6 * p + 2]);
        const float c3[3] = {pos[6 * p + 3], pos[6 * p + 4], pos[6 * p + 5]};
        const f3 c = mk3(c3[0], c3[1], c3[2]);
        std::vector<std::pair<float, int>> order(nt);
        for (int i = 0; i < nt; ++i) {
            const DTri &T = tris[i];
            const float a[3] = {T.v0.x, T.v0.y, T.v0.z}, e[3] = {T.e1.x, T.e1.y, T.e1.z}, g[3] = {T.e2.x, T.e2.y, T.e2.z};
            float dist = 0.f;
            for (int k = 0; k < 3; ++k) {
                const float b = a[k] + e[k], d = a[k] + g[k];
                dist = std::max(dist, axis_gap(c3[k], std::min(a[k], std::min(b, d)), std::max(a[k], std::max(b, d))));
            }
            order[i] = {dist, i};
        }
        std::sort(order.begin(), order.end());
        LocalList W{};
        W.cx = c.x;
        W.cy = c.y;
        W.cz = c.z;
        W.h = local_clear(order[kLocalTris].first, c);
        std::vector<std::vector<int>> group;
        for (int j = 0; j < kLocalTris; ++j) {
            const float4 pl = local_tri(tris[order[j].second], c, W.h).plane;
            size_t g = 0;
            while (g < group.size() && !local_same_plane(W.plane[g], pl, W.h)) ++g;
            if (g == group.size()) {
                W.plane[g] = pl;
                W.range[g].y = local_clear(order[j].first, c);
                group.emplace_back();
            }
            group[g].push_back(order[j].second);
        }
        W.planes = int(group.size());
        int at = 0;
        for (size_t g = 0; g < group.size(); ++g) {
            W.start[g] = (unsigned char)at;
            float eps = 0.f;
            for (int slot : group[g]) {
                const LocalTri t = local_tri(tris[slot], c, W.h);
                W.u[at] = t.u;
                W.v[at] = t.v;
                W.uv_eps[at] = t.uv_eps;
                eps = std::max(eps, t.plane_eps);
                W.slot[at++] = slot;
            }
            W.range[g].x = eps + local_merge_margin(W.h);
        }
        W.start[group.size()] = (unsigned char)at;
        for (int j = W.planes; j % kLocalGroup; ++j) local_fill(W, j);
        // the builder keeps a list that settles 8 of 32 rays from the transmitter
        int settled = 0;
        if (W.h > 0.f && local_holds(W, s))
            for (int k = 0; k < 32; ++k) {
                const float y = 1.f - (2.f * k + 1.f) / 32.f, r = std::sqrt(std::max(0.f, 1.f - y * y));
                float t;
                settled += closest_local(W, tris.data(), s, mk3(r * std::cos(2.39996323f * k), y,
                                                                r * std::sin(2.39996323f * k)), t) >= 0;
            }
        const LocalList &L = lists[p];
        int wrong = 0;
        if (L.planes > 0) {
            wrong += L.planes != W.planes;
            wrong += !near_equal(L.h, W.h, W.h) || L.cx != W.cx || L.cy != W.cy || L.cz != W.cz;
            for (int g = 0; g < W.planes && !wrong; ++g) {
                const float size = 1.f + std::fabs(W.plane[g].w);
                wrong += !near_equal(L.plane[g].x, W.plane[g].x, 1.f) || !near_equal(L.plane[g].y, W.plane[g].y, 1.f) ||
                         !near_equal(L.plane[g].z, W.plane[g].z, 1.f) || !near_equal(L.plane[g].w, W.plane[g].w, size);
                wrong += !near_equal(L.range[g].y, W.range[g].y, 1.f + W.h);
                // margins: what covers the rounding may itself be rounded, by a thousandth at most
                wrong += std::fabs(L.range[g].x - W.range[g].x) > 1e-3f * W.range[g].x;
                wrong += L.start[g] != W.start[g] || L.start[g + 1] != W.start[g + 1];
                for (int k = W.start[g]; k < W.start[g + 1]; ++k) {
                    wrong += L.slot[k] != W.slot[k];
                    wrong += std::fabs(L.uv_eps[k] - W.uv_eps[k]) > 1e-3f * W.uv_eps[k];
                    const float su = std::fabs(W.u[k].x) + std::fabs(W.u[k].y) + std::fabs(W.u[k].z) + std::fabs(W.u[k].w);
                    const float sv = std::fabs(W.v[k].x) + std::fabs(W.v[k].y) + std::fabs(W.v[k].z) + std::fabs(W.v[k].w);
                    wrong += !near_equal(L.u[k].x, W.u[k].x, su) || !near_equal(L.u[k].y, W.u[k].y, su) ||
                             !near_equal(L.u[k].z, W.u[k].z, su) || !near_equal(L.u[k].w, W.u[k].w, su);
                    wrong += !near_equal(L.v[k].x, W.v[k].x, sv) || !near_equal(L.v[k].y, W.v[k].y, sv) ||
                             !near_equal(L.v[k].z, W.v[k].z, sv) || !near_equal(L.v[k].w, W.v[k].w, sv);
                }
            }
            // whole groups of planes: the filling is never crossed
            for (int j = L.planes; !wrong && j % kLocalGroup; ++j)
                wrong += L.plane[j].x != 0.f || L.plane[j].y != 0.f || L.plane[j].z != 0.f || L.plane[j].w != 1.f ||
                         L.range[j].x != 0.f;
        }
        std::printf("planes %d want %d near %d wrong %d\n", L.planes, W.planes, settled, wrong);
    }
    cudaFree(d_ant);
    cudaFree(d_list);
    return hsr_scene_destroy(scene) == HSR_OK ? 0 : 2;
}
