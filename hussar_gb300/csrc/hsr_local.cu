// Builds the poses' neighbourhood lists (hsr_local.cuh) before a trace launch, and measures
// whether a scene is dense enough for them.
#include <algorithm>
#include <vector>

#include "hsr_local.cuh"

namespace hsr {

namespace {

constexpr int kFrontier = 1024;    // nodes of one tree level a search holds
constexpr int kCandidates = 1024;  // triangles a search holds
constexpr int kNearest = 3 * kLocalTris;   // triangles that are ranked: at most,
constexpr int kFewNearest = kLocalTris + 32;  // and where their distances allow it
constexpr int kSearchSteps = 14;

// A scene whose point queries visit fewer nodes than this keeps to the BVH: the list's
// plane tests cost as much as some ten divergent node visits per query, and the lists of
// open scenes settle few queries (an urban canyon: 20 %). Batches of 33 poses of 2^13 .. 2^17
// samples (4 bounces, split phase, synthesis) by the BVH alone and with lists, by the visits
// measured here: boxes 127 visits 13.2 and 2.3 ms, 70 visits 7.6 and 2.9, 54 visits 6.0 and
// 3.2, 45 visits 6.1 and 2.5, 37 visits 4.7 and 3.4, 29 visits 3.9 and 3.4, 25 visits 3.4 and
// 3.6, 18 visits 1.9 and 2.7; sphere 22 visits 0.33 and 0.61, urban canyon 23 visits 1.8 and
// 2.4. They break even at 22 to 30; the line keeps clear of that, as only boxes lie above it.
// A refit keeps the build's answer: 100 k triangles of boxes, built dense and pulled 8 x
// apart, run in 130 ms with lists and 240 without (the tree is what costs there).
constexpr float kDenseNodes = 48.f;

struct Search {
    int frontier[2][kFrontier];
    int slot[kCandidates];
    float dist[kCandidates];
    int near_slot[kNearest];
    float near_dist[kNearest];
    int leaf[kCandidates];  // leaf references
};

// Chebyshev distance of a point to a box.
__device__ __forceinline__ float box_distance(f3 c, float lx, float hx, float ly, float hy, float lz, float hz) {
    return fmaxf(0.f, fmaxf(fmaxf(lx - c.x, c.x - hx), fmaxf(fmaxf(ly - c.y, c.y - hy), fmaxf(lz - c.z, c.z - hz))));
}

// The triangles whose bounding boxes come within h of c, by one warp, level by level down
// the tree and then over the leaves met, whose triangles' loads need not wait for one
// another. Returns their number (S.slot, S.dist), or -1 when there are more than fit;
// `visited` counts the nodes whose children were looked at.
__device__ int collect(Search &S, const DNode *__restrict__ nodes, const DTri *__restrict__ tris, f3 c, float h,
                       int &visited) {
    const int lane = threadIdx.x;
    const unsigned before = (1u << lane) - 1u;
    int cur = 0, n = 1, leaves = 0, found = 0;
    visited = 0;
    if (lane == 0) S.frontier[0][0] = 0;
    while (n > 0) {
        __syncwarp();
        visited += n;
        int next = 0;
        for (int i0 = 0; i0 < n; i0 += 32) {
            DNode N;
            float dist[2] = {CUDART_INF_F, CUDART_INF_F};
            if (i0 + lane < n) {
                N = load_node(nodes, S.frontier[cur][i0 + lane]);
                dist[0] = box_distance(c, N.a.x, N.a.y, N.a.z, N.a.w, N.c.x, N.c.y);
                dist[1] = box_distance(c, N.b.x, N.b.y, N.b.z, N.b.w, N.c.z, N.c.w);
            }
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const int child = w == 0 ? N.d.x : N.d.y;
                const bool in = i0 + lane < n && dist[w] <= h;
                const unsigned inner = __ballot_sync(0xffffffffu, in && child >= 0);
                const unsigned leaf = __ballot_sync(0xffffffffu, in && child < 0);
                if (in) {
                    const int k = child >= 0 ? next + __popc(inner & before) : leaves + __popc(leaf & before);
                    if (child >= 0 && k < kFrontier) S.frontier[cur ^ 1][k] = child;
                    if (child < 0 && k < kCandidates) S.leaf[k] = ~child;
                }
                next += __popc(inner);
                leaves += __popc(leaf);
            }
        }
        n = next;
        cur ^= 1;
        if (n > kFrontier || leaves > kCandidates) return -1;
    }
    __syncwarp();
    for (int i0 = 0; i0 < leaves; i0 += 32) {
        const int ref = i0 + lane < leaves ? S.leaf[i0 + lane] : 0, count = i0 + lane < leaves ? (ref & 7) + 1 : 0;
        for (int k = 0; __any_sync(0xffffffffu, k < count); ++k) {
            const int s = (ref >> 3) + k;
            float td = CUDART_INF_F;
            if (k < count) {
                const DTri T = load_tri(tris, s);
                const float ax = T.v0.x + T.e1.x, bx = T.v0.x + T.e2.x;
                const float ay = T.v0.y + T.e1.y, by = T.v0.y + T.e2.y;
                const float az = T.v0.z + T.e1.z, bz = T.v0.z + T.e2.z;
                td = box_distance(c, fminf(T.v0.x, fminf(ax, bx)), fmaxf(T.v0.x, fmaxf(ax, bx)),
                                  fminf(T.v0.y, fminf(ay, by)), fmaxf(T.v0.y, fmaxf(ay, by)),
                                  fminf(T.v0.z, fminf(az, bz)), fmaxf(T.v0.z, fmaxf(az, bz)));
            }
            const bool in = k < count && td <= h;
            const unsigned mask = __ballot_sync(0xffffffffu, in);
            const int at = found + __popc(mask & before);
            if (in && at < kCandidates) {
                S.slot[at] = s;
                S.dist[at] = td;
            }
            found += __popc(mask);
        }
    }
    __syncwarp();
    return found > kCandidates ? -1 : found;
}

// The more than kLocalTris and at most kNearest triangles nearest c (S.near_slot,
// S.near_dist; their number is returned), or 0 where there are no such. A search down the
// tree costs 20 us, most of it latency (25 levels of dependent loads), so it takes in up to 1024
// triangles around a first radius `h` and the radius is then narrowed on their distances:
// one or two searches for most poses. Lists of 96 poses (1 M triangles) took 220 us when
// the search was repeated until 65 to 192 triangles were in reach and 129 with this; with the
// leaves after the descent, slots by ballots instead of shared atomics, and ranks and
// groups in loops that need not wait for their loads, 85. Those of 1999 poses (20 k
// triangles): 228, 188 and 130.
__device__ int find_nearest(Search &S, const DNode *__restrict__ nodes, const DTri *__restrict__ tris, f3 c, float h) {
    const int lane = threadIdx.x;
    float lo = 0.f, hi = 0.f;  // too few within lo, too many within hi (0: not known)
    int n = 0;
    for (int step = 0; step < kSearchSteps && n <= kLocalTris; ++step) {
        int visited;
        n = collect(S, nodes, tris, c, h, visited);
        if (n < 0)
            hi = h;
        else
            lo = h;
        if (n <= kLocalTris) h = lo == 0.f ? 0.4f * hi : hi == 0.f ? 2.5f * lo : sqrtf(lo * hi);
        __syncwarp();
    }
    if (n <= kLocalTris) return 0;
    // bisection for a distance that at most kFewNearest and more than kLocalTris are within, or
    // the nearest to it up to kNearest
    auto within = [&](float t) {
        int m = 0;
        for (int i = lane; i < n; i += 32) m += S.dist[i] <= t;
        return __reduce_add_sync(0xffffffffu, m);
    };
    float below = 0.f, above = h, t = h;
    int m = n;
    for (int step = 0; step < 24 && m > kFewNearest; ++step) {
        const float mid = 0.5f * (below + above);
        const int k = within(mid);
        if (k > kLocalTris) {
            above = t = mid;
            m = k;
        } else {
            below = mid;
        }
    }
    if (m > kNearest) return 0;  // too many at one distance
    int at = 0;
    for (int i = lane; i - lane < n; i += 32) {
        const bool in = i < n && S.dist[i] <= t;
        const unsigned mask = __ballot_sync(0xffffffffu, in);
        if (in) {
            const int k = at + __popc(mask & ((1u << lane) - 1u));
            S.near_slot[k] = S.slot[i];
            S.near_dist[k] = S.dist[i];
        }
        at += __popc(mask);
    }
    __syncwarp();
    return m;
}

// The rank of one of the n nearest.
__device__ __forceinline__ int rank_of(const Search &S, int n, int i) {
    const float di = S.near_dist[i];
    const int si = S.near_slot[i];
    int rank = 0;
#pragma unroll 8
    for (int k = 0; k < n; ++k) {
        const float dk = S.near_dist[k];
        rank += int(dk < di) | (int(dk == di) & int(S.near_slot[k] < si));
    }
    return rank;
}

// One warp per pose. The list is left empty (planes 0: the pose's queries all go to the
// BVH) where the transmitter lies outside the cube or fewer than a quarter of 32 rays from
// it, spread over the sphere, are settled by the list.
__global__ void __launch_bounds__(32) k_local_build(const PoseJob *__restrict__ jobs, const DNode *nodes,
                                                    const DTri *tris, const hsr_antenna *__restrict__ tx,
                                                    const hsr_antenna *__restrict__ rx, float guess,
                                                    LocalList *__restrict__ out) {
    __shared__ Search S;
    __shared__ LocalList L;
    __shared__ int near_slot[kLocalTris];
    __shared__ float near_dist[kLocalTris];
    __shared__ float4 near_plane[kLocalTris];
    __shared__ unsigned char near_group[kLocalTris], next[kLocalTris];
    const int pose = blockIdx.x, lane = threadIdx.x;
    if (jobs) {
        nodes = jobs[pose].nodes;
        tris = jobs[pose].tris;
        guess = jobs[pose].local_radius;
    }
    const f3 c = mk3(rx[pose].position[0], rx[pose].position[1], rx[pose].position[2]);
    const f3 s = mk3(tx[pose].position[0], tx[pose].position[1], tx[pose].position[2]);
    const int n = guess > 0.f ? find_nearest(S, nodes, tris, c, guess) : 0;
    if (n <= kLocalTris) {
        if (lane == 0) out[pose].planes = 0;
        return;
    }
    // the kLocalTris nearest in order, and the cube up to the next triangle's box
    for (int i = lane; i < n; i += 32) {
        const int rank = rank_of(S, n, i);
        if (rank < kLocalTris) {
            near_slot[rank] = S.near_slot[i];
            near_dist[rank] = S.near_dist[i];
        }
        if (rank == kLocalTris) L.h = local_clear(S.near_dist[i], c);
    }
    __syncwarp();
    const float half = L.h;
    for (int j = lane; j < kLocalTris; j += 32) near_plane[j] = local_tri(load_tri(tris, near_slot[j]), c, half).plane;
    __syncwarp();
    // the planes in order of their nearest triangle: each triangle joins the first group
    // whose plane it shares. First every triangle's earlier likenesses, as bits (a lane has
    // the triangles l, l + 32, ...), then which of them lead a group, one after the other.
    constexpr int kPerLane = kLocalTris / 32;
    static_assert(kLocalTris % 32 == 0 && kLocalTris < 256, "whole lanes of triangles, offsets in a byte");
    unsigned like[kPerLane][kPerLane] = {};
#pragma unroll
    for (int w = 0; w < kPerLane; ++w) {
        const float4 mine = near_plane[lane + 32 * w];
#pragma unroll
        for (int v = 0; v <= w; ++v) {
            unsigned bits = 0;
#pragma unroll 8
            for (int i = 0; i < 32; ++i)
                bits |= unsigned(local_same_plane(near_plane[32 * v + i], mine, half)) << i;
            like[w][v] = v == w ? bits & ((1u << lane) - 1u) : bits;
        }
    }
    unsigned leads[kPerLane] = {};
    int groups = 0, size[kPerLane] = {};
#pragma unroll
    for (int w = 0; w < kPerLane; ++w)
        for (int i = 0; i < 32; ++i) {
            int lead = 32 * w + i;  // its own, unless an earlier leader is like it
#pragma unroll
            for (int v = w; v >= 0; --v) {
                const unsigned m = __shfl_sync(0xffffffffu, like[w][v], i) & leads[v];
                if (m) lead = 32 * v + __ffs(int(m)) - 1;
            }
            int g = groups;
            if (lead == 32 * w + i) {
                leads[w] |= 1u << i;
                if (lane == 0) {
                    L.plane[g] = near_plane[lead];
                    L.range[g].y = local_clear(near_dist[lead], c);
                }
                ++groups;
            } else {
                g = 0;
#pragma unroll
                for (int v = 0; v < kPerLane; ++v)
                    g += lead >= 32 * v + 32 ? __popc(leads[v])
                         : lead >= 32 * v    ? __popc(leads[v] & ((1u << (lead & 31)) - 1u))
                                             : 0;
            }
            if (lane == 0) near_group[32 * w + i] = (unsigned char)g;
#pragma unroll
            for (int v = 0; v < kPerLane; ++v)
                if (lane + 32 * v == g) ++size[v];
        }
    __syncwarp();
    // where each group starts, then its triangles
    int total = 0;
#pragma unroll
    for (int w = 0; w < kPerLane; ++w) {
        int sum = size[w];
        for (int off = 1; off < 32; off <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, sum, off);
            if (lane >= off) sum += v;
        }
        const int before = total + sum - size[w];
        total += __shfl_sync(0xffffffffu, sum, 31);
        L.start[lane + 32 * w] = (unsigned char)before;
        next[lane + 32 * w] = (unsigned char)before;
    }
    if (lane == 0) L.start[kLocalTris] = (unsigned char)kLocalTris;
    for (int j = 0; j < kLocalTris; ++j) {
        const int g = near_group[j];
        if (lane == (g & 31)) L.slot[next[g]++] = near_slot[j];
    }
    __syncwarp();
    for (int j = lane; j < groups; j += 32) {
        float eps = 0.f;
        for (int k = L.start[j]; k < L.start[j + 1]; ++k) {
            const LocalTri t = local_tri(load_tri(tris, L.slot[k]), c, half);
            L.u[k] = t.u;
            L.v[k] = t.v;
            L.uv_eps[k] = t.uv_eps;
            eps = fmaxf(eps, t.plane_eps);
        }
        L.range[j].x = eps + local_merge_margin(half);
    }
    const int whole = (groups + kLocalGroup - 1) / kLocalGroup * kLocalGroup;
    if (groups + lane < whole) local_fill(L, groups + lane);
    if (lane == 0) {
        L.cx = c.x;
        L.cy = c.y;
        L.cz = c.z;
        L.planes = groups;
    }
    __syncwarp();
    bool settled = false;
    if (L.h > 0.f && local_holds(L, s)) {
        // 32 directions spread evenly over the sphere (a Fibonacci lattice)
        const float y = 1.f - (2.f * lane + 1.f) / 32.f, r = sqrtf(fmaxf(0.f, 1.f - y * y));
        float sn, cs;
        sincosf(2.39996323f * lane, &sn, &cs);
        float t;
        settled = closest_local(L, tris, s, mk3(r * cs, y, r * sn), t) >= 0;
    }
    const int hits = __popc(__ballot_sync(0xffffffffu, settled));
    if (lane == 0 && hits < 8) L.planes = 0;
    __syncwarp();
    const int *src = reinterpret_cast<const int *>(&L);
    int *dst = reinterpret_cast<int *>(out + pose);
    for (int k = lane; k < int(sizeof(LocalList) / sizeof(int)); k += 32) dst[k] = src[k];
}

// At kDensityPoints triangle centroids spread over the scene: the nodes a point query
// visits and the distance of the first triangle that a list there would not hold.
constexpr int kDensityPoints = 128;

__global__ void __launch_bounds__(32) k_density(const DNode *__restrict__ nodes, const DTri *__restrict__ tris,
                                                int64_t nt, float guess, float2 *__restrict__ out) {
    __shared__ Search S;
    const DTri T = load_tri(tris, int(nt * blockIdx.x / gridDim.x));
    const f3 c = mk3(T.v0.x + (T.e1.x + T.e2.x) / 3.f, T.v0.y + (T.e1.y + T.e2.y) / 3.f,
                     T.v0.z + (T.e1.z + T.e2.z) / 3.f);
    int visited;
    collect(S, nodes, tris, c, 0.f, visited);
    __syncwarp();
    const int n = float(visited) >= 0.5f * kDenseNodes ? find_nearest(S, nodes, tris, c, guess) : 0;
    for (int i = threadIdx.x; i < n; i += 32)
        if (rank_of(S, n, i) == kLocalTris) out[blockIdx.x] = make_float2(float(visited), S.near_dist[i]);
    if (n == 0 && threadIdx.x == 0) out[blockIdx.x] = make_float2(float(visited), 0.f);
}

}  // namespace

int measure_density(SceneDev &s, cudaStream_t st, std::string &err) {
    s.local_radius = 0.f;
    if (s.node_count < 4 * kDenseNodes) return 0;
    DNode root;
    float2 *d = nullptr;
    if (!dev_alloc(&d, sizeof(float2) * kDensityPoints, err)) return 3;
    cudaError_t e = cudaMemcpyAsync(&root, s.nodes, sizeof(root), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    std::vector<float2> v(kDensityPoints);
    if (e == cudaSuccess) {
        // a first radius: the cube that would hold a neighbourhood were the triangles
        // spread evenly over the scene's box
        const float ex = std::max(root.a.y, root.b.y) - std::min(root.a.x, root.b.x);
        const float ey = std::max(root.a.w, root.b.w) - std::min(root.a.z, root.b.z);
        const float ez = std::max(root.c.y, root.c.w) - std::min(root.c.x, root.c.z);
        const float guess = 0.5f * std::max(ex, std::max(ey, ez)) * std::cbrt(float(kLocalTris) / float(s.tri_count));
        k_density<<<kDensityPoints, 32, 0, st>>>(s.nodes, s.tris, s.tri_count, guess > 0.f ? guess : 1.f, d);
        note_launches(1);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(v.data(), d, sizeof(float2) * kDensityPoints, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(d);
    if (e != cudaSuccess) {
        err = std::string("density: ") + cudaGetErrorString(e);
        return 2;
    }
    float visited = 0.f;
    std::vector<float> radius;
    for (const float2 &x : v) {
        visited += x.x / kDensityPoints;
        if (x.y > 0.f) radius.push_back(x.y);
    }
    if (visited < kDenseNodes || radius.size() < kDensityPoints / 4) return 0;
    std::nth_element(radius.begin(), radius.begin() + radius.size() / 2, radius.end());
    // twice the usual distance: some 200 to 500 triangles in reach, a single search mostly
    s.local_radius = 2.f * radius[radius.size() / 2];
    return 0;
}

int launch_local_build(const TraceParams &p, float radius, LocalList *out, cudaStream_t st) {
    k_local_build<<<p.pose_count, 32, 0, st>>>(p.jobs, p.nodes, p.tris, p.tx, p.rx, radius, out);
    note_launches(1);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // namespace hsr
