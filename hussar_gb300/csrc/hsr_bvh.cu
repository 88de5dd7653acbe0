// Device BVH build: replaces Embree's rtcCommitScene (libhussar/src/arch/cpu.cpp:32-47)
// and OptiX's optixAccelBuild + compaction (src/arch/gpu.cpp:82-207).
//
//   1. per-triangle bounds and centroids, scene centroid bounds (k_bounds)
//   2. 63-bit Morton code of each centroid, 21 bits per axis (k_morton)
//   3. radix sort of (code, triangle id) pairs (CUB DeviceRadixSort)
//   4. triangle records written in sorted order (k_write_tris)
//   5. topology, one of:
//      PLOC (default): parallel locally-ordered clustering over the Morton order
//        (Meister and Bittner 2018): every cluster finds, within +-256 positions, the
//        neighbour whose merged box has the smallest surface area; mutual nearest pairs
//        merge; survivors are compacted in order; repeat until one cluster is left.
//        Surface-area-driven like an SAH build, robust to large overlapping triangles.
//      LBVH: binary radix tree from the sorted codes (Karras 2012, k_karras) and a
//        bottom-up box refit (k_refit).
//   6. insertion passes (up to 32, hsr_set_bvh_optimize): every subtree is re-placed in
//      parallel where the surface-area cost falls most (k_reins_*, below)
//   7. leaves: a bottom-up surface-area cost pass turns subtrees of at most the leaf size
//      (default 4, hsr_set_bvh_leaf_size) into leaves when testing their triangles is
//      cheaper than visiting their nodes (k_leaf_cost); the triangle records are reordered so that every
//      leaf's triangles are contiguous (k_leaf_group, radix sort, k_permute_tris) and
//      the links of the remaining nodes rewritten (k_relink).
//   8. the reachable nodes renumbered depth first and the array shrunk to them.
// Node i stores the boxes of both its children; node 0 is the root. A child reference
// c >= 0 is an internal node; c < 0 a leaf of ((~c) & 7) + 1 triangles from slot
// (~c) >> 3. A node's first child, when internal, is node i + 1.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_select.cuh>

#include <limits>
#include <vector>

#include "hsr_common.cuh"
#include "hsr_internal.h"

namespace hsr {

namespace {

__device__ __forceinline__ unsigned f2ord(float f) {
    unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// Triangle AABB, padded so the FMA slab test stays conservative.
__global__ void k_bounds(const float *__restrict__ v, const int32_t *__restrict__ idx, int64_t nt, float *__restrict__ lo,
                         float *__restrict__ hi, unsigned *__restrict__ cbounds) {
    int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (t >= nt) return;
    float c[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float x0 = v[3 * int64_t(idx[3 * t + 0]) + a];
        float x1 = v[3 * int64_t(idx[3 * t + 1]) + a];
        float x2 = v[3 * int64_t(idx[3 * t + 2]) + a];
        float mn = fminf(x0, fminf(x1, x2)), mx = fmaxf(x0, fmaxf(x1, x2));
        float pad = fmaxf(fabsf(mn), fabsf(mx)) * 4e-6f + 1e-6f;
        lo[3 * t + a] = mn - pad;
        hi[3 * t + a] = mx + pad;
        c[a] = 0.5f * mn + 0.5f * mx;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        atomicMin(&cbounds[a], f2ord(c[a]));
        atomicMax(&cbounds[3 + a], f2ord(c[a]));
    }
}

__device__ __forceinline__ uint64_t expand21(uint64_t x) {
    x &= 0x1fffffull;
    x = (x | x << 32) & 0x1f00000000ffffull;
    x = (x | x << 16) & 0x1f0000ff0000ffull;
    x = (x | x << 8) & 0x100f00f00f00f00full;
    x = (x | x << 4) & 0x10c30c30c30c30c3ull;
    x = (x | x << 2) & 0x1249249249249249ull;
    return x;
}

__global__ void k_morton(const float *__restrict__ lo, const float *__restrict__ hi, int64_t nt,
                         const unsigned *__restrict__ cbounds, uint64_t *__restrict__ keys, int32_t *__restrict__ ids) {
    int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (t >= nt) return;
    uint64_t code = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        float cmin = ord2f(cbounds[a]), cmax = ord2f(cbounds[3 + a]);
        float c = 0.5f * lo[3 * t + a] + 0.5f * hi[3 * t + a];
        float ext = cmax - cmin;
        float u = ext > 0.f ? (c - cmin) / ext : 0.5f;
        u = fminf(fmaxf(u, 0.f), 1.f);
        uint64_t q = uint64_t(fminf(u * 2097152.f, 2097151.f));
        code |= expand21(q) << (2 - a);
    }
    keys[t] = code;
    ids[t] = int32_t(t);
}

__global__ void k_write_tris(const float *__restrict__ v, const int32_t *__restrict__ idx,
                             const int32_t *__restrict__ sorted_ids, int64_t nt, DTri *__restrict__ tris) {
    int64_t s = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (s >= nt) return;
    int64_t t = sorted_ids[s];
    const float *p0 = v + 3 * int64_t(idx[3 * t + 0]);
    const float *p1 = v + 3 * int64_t(idx[3 * t + 1]);
    const float *p2 = v + 3 * int64_t(idx[3 * t + 2]);
    DTri T;
    T.v0 = make_float4(p0[0], p0[1], p0[2], __int_as_float(int(t)));
    T.e1 = make_float4(p1[0] - p0[0], p1[1] - p0[1], p1[2] - p0[2], 0.f);
    T.e2 = make_float4(p2[0] - p0[0], p2[1] - p0[1], p2[2] - p0[2], 0.f);
    tris[s] = T;
}

// common prefix length of sorted keys i and j, with the index as a tie-breaker
__device__ __forceinline__ int delta(const uint64_t *__restrict__ k, int64_t n, int64_t i, int64_t j) {
    if (j < 0 || j >= n) return -1;
    uint64_t a = k[i], b = k[j];
    if (a == b) return 64 + __clzll((unsigned long long)(i ^ j));
    return __clzll((unsigned long long)(a ^ b));
}

// Karras 2012: internal node i covers a key range; its split is the highest differing bit.
__global__ void k_karras(const uint64_t *__restrict__ k, int64_t n, DNode *__restrict__ nodes,
                         int32_t *__restrict__ parent_internal, int32_t *__restrict__ parent_leaf) {
    int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= n - 1) return;
    int d = (delta(k, n, i, i + 1) - delta(k, n, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = delta(k, n, i, i - d);
    int64_t lmax = 2;
    while (delta(k, n, i, i + lmax * d) > dmin) lmax <<= 1;
    int64_t l = 0;
    for (int64_t t = lmax >> 1; t >= 1; t >>= 1)
        if (delta(k, n, i, i + (l + t) * d) > dmin) l += t;
    int64_t j = i + l * d;
    int dnode = delta(k, n, i, j);
    int64_t s = 0;
    int64_t len = l;
    int64_t t = (len + 1) >> 1;
    while (true) {
        if (delta(k, n, i, i + (s + t) * d) > dnode) s += t;
        if (t == 1) break;
        t = (t + 1) >> 1;
    }
    int64_t gamma = i + s * d + (d < 0 ? -1 : 0);
    int64_t first = i < j ? i : j, last = i < j ? j : i;
    int c0, c1;
    if (first == gamma) {
        c0 = ~int(gamma);
        parent_leaf[gamma] = int(i);
    } else {
        c0 = int(gamma);
        parent_internal[gamma] = int(i);
    }
    if (last == gamma + 1) {
        c1 = ~int(gamma + 1);
        parent_leaf[gamma + 1] = int(i);
    } else {
        c1 = int(gamma + 1);
        parent_internal[gamma + 1] = int(i);
    }
    nodes[i].d = make_int4(c0, c1, 0, 0);
}

struct Box {
    float lo[3], hi[3];
};

__device__ __forceinline__ Box child_box(const DNode &n, int which) {
    Box b;
    if (which == 0) {
        b.lo[0] = n.a.x; b.hi[0] = n.a.y; b.lo[1] = n.a.z; b.hi[1] = n.a.w; b.lo[2] = n.c.x; b.hi[2] = n.c.y;
    } else {
        b.lo[0] = n.b.x; b.hi[0] = n.b.y; b.lo[1] = n.b.z; b.hi[1] = n.b.w; b.lo[2] = n.c.z; b.hi[2] = n.c.w;
    }
    return b;
}

// Bottom-up refit: a leaf's thread climbs while it is the second child to arrive.
__global__ void k_refit(int64_t n, const int32_t *__restrict__ sorted_ids, const float *__restrict__ lo,
                        const float *__restrict__ hi, DNode *nodes, const int32_t *__restrict__ parent_internal,
                        const int32_t *__restrict__ parent_leaf, int *counters, int *depth_out) {
    int64_t leaf = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (leaf >= n) return;
    int p = parent_leaf[leaf];
    int depth = 1;
    while (p >= 0) {
        __threadfence();
        int prev = atomicAdd(&counters[p], 1);
        if (prev == 0) return;  // the sibling subtree is not finished; its thread continues
        __threadfence();
        volatile DNode *vn = nodes;
        int c[2] = {vn[p].d.x, vn[p].d.y};
        Box bx[2];
        for (int w = 0; w < 2; ++w) {
            if (c[w] < 0) {
                int64_t t = sorted_ids[~c[w]];
                for (int a = 0; a < 3; ++a) {
                    bx[w].lo[a] = lo[3 * t + a];
                    bx[w].hi[a] = hi[3 * t + a];
                }
            } else {
                DNode cn;
                cn.a = make_float4(vn[c[w]].a.x, vn[c[w]].a.y, vn[c[w]].a.z, vn[c[w]].a.w);
                cn.b = make_float4(vn[c[w]].b.x, vn[c[w]].b.y, vn[c[w]].b.z, vn[c[w]].b.w);
                cn.c = make_float4(vn[c[w]].c.x, vn[c[w]].c.y, vn[c[w]].c.z, vn[c[w]].c.w);
                Box b0 = child_box(cn, 0), b1 = child_box(cn, 1);
                for (int a = 0; a < 3; ++a) {
                    bx[w].lo[a] = fminf(b0.lo[a], b1.lo[a]);
                    bx[w].hi[a] = fmaxf(b0.hi[a], b1.hi[a]);
                }
            }
        }
        vn[p].a.x = bx[0].lo[0]; vn[p].a.y = bx[0].hi[0]; vn[p].a.z = bx[0].lo[1]; vn[p].a.w = bx[0].hi[1];
        vn[p].b.x = bx[1].lo[0]; vn[p].b.y = bx[1].hi[0]; vn[p].b.z = bx[1].lo[1]; vn[p].b.w = bx[1].hi[1];
        vn[p].c.x = bx[0].lo[2]; vn[p].c.y = bx[0].hi[2]; vn[p].c.z = bx[1].lo[2]; vn[p].c.w = bx[1].hi[2];
        p = parent_internal[p];
        depth++;
    }
    atomicMax(depth_out, depth);
}

// Leaf depth statistics: each leaf walks to the root.
__global__ void k_leaf_depth(int64_t n, const int32_t *__restrict__ parent_internal,
                             const int32_t *__restrict__ parent_leaf, int *depth_out) {
    int64_t leaf = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (leaf >= n) return;
    int p = parent_leaf[leaf];
    int depth = 1;
    while (p >= 0 && depth < 1 << 20) {
        p = parent_internal[p];
        depth++;
    }
    atomicMax(depth_out, depth);
}

// ---------------- PLOC ----------------
constexpr int kPlocRadius = 256;
constexpr int kPlocLanes = 8;  // per cluster in k_ploc_nearest

struct Cluster {
    int id;       // node encoding: >= 0 internal node, < 0 leaf slot (~slot)
    float b[6];   // lo.xyz, hi.xyz
};

__global__ void k_ploc_init(int64_t n, const int32_t *__restrict__ sorted_ids, const float *__restrict__ lo,
                            const float *__restrict__ hi, Cluster *__restrict__ cl) {
    int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const int64_t t = sorted_ids[i];
    Cluster c;
    c.id = ~int(i);
    for (int a = 0; a < 3; ++a) {
        c.b[a] = lo[3 * t + a];
        c.b[3 + a] = hi[3 * t + a];
    }
    cl[i] = c;
}

__device__ __forceinline__ float merged_area(const float *a, const float *b) {
    const float dx = fmaxf(a[3], b[3]) - fminf(a[0], b[0]);
    const float dy = fmaxf(a[4], b[4]) - fminf(a[1], b[1]);
    const float dz = fmaxf(a[5], b[5]) - fminf(a[2], b[2]);
    return dx * dy + dy * dz + dz * dx;
}

// nearest[i]: the cluster within +-R whose union with i has the smallest surface area
// (ties: the lower index), read through a shared-memory window by eight lanes per cluster.
// Bound by instruction issue while many clusters are left, then by the window's chain of
// comparisons, which eight lanes make an eighth as long. One lane per cluster: 114 us at
// 250 k clusters and 32 us at any count from 500 to 37 k; this 109, 20 at 37 k and 7 from
// 5 k down (a build of 250 k triangles, 69 iterations: 2.39 -> 0.95 ms).
__global__ void __launch_bounds__(256) k_ploc_nearest(int n, const Cluster *__restrict__ cl, int *__restrict__ nearest) {
    constexpr int L = kPlocLanes, kClusters = 256 / L, kRows = kClusters + 2 * kPlocRadius;
    __shared__ float2 sb[kRows][3];
    const int base = blockIdx.x * kClusters;
    for (int k = threadIdx.x; k < kRows; k += 256) {
        const int j = base - kPlocRadius + k;
        if (j >= 0 && j < n) {
#pragma unroll
            for (int a = 0; a < 3; ++a) sb[k][a] = make_float2(cl[j].b[2 * a], cl[j].b[2 * a + 1]);
        }
    }
    __syncthreads();
    const int own = threadIdx.x / L, lane = threadIdx.x % L, i = base + own;
    float best = __int_as_float(0x7f800000);
    int bj = -1;
    if (i < n) {
        const float2 *si = sb[own + kPlocRadius];
        const float bi[6] = {si[0].x, si[0].y, si[1].x, si[1].y, si[2].x, si[2].y};
        const int j0 = max(0, i - kPlocRadius), j1 = min(n - 1, i + kPlocRadius);
#pragma unroll 4
        for (int j = j0 + lane; j <= j1; j += L) {
            if (j == i) continue;
            const float2 *sj = sb[j - base + kPlocRadius];
            const float2 u = sj[0], v = sj[1], w = sj[2];
            const float bb[6] = {u.x, u.y, v.x, v.y, w.x, w.y};
            const float a = merged_area(bi, bb);
            if (a < best) {
                best = a;
                bj = j;
            }
        }
    }
#pragma unroll
    for (int o = L / 2; o > 0; o /= 2) {
        const float a = __shfl_xor_sync(~0u, best, o);
        const int j = __shfl_xor_sync(~0u, bj, o);
        if (a < best || (a == best && unsigned(j) < unsigned(bj))) {
            best = a;
            bj = j;
        }
    }
    if (i < n && lane == 0) nearest[i] = bj;
}

// Mutual nearest pairs merge into a new internal node (allocated from the top so that the
// last merge, the root, is node 0); the lower index keeps the merged cluster.
__global__ void k_ploc_merge(int n, const int *__restrict__ nearest, Cluster *cl, char *__restrict__ keep,
                             DNode *__restrict__ nodes, int *__restrict__ node_counter, int internal_total,
                             int32_t *__restrict__ parent_internal, int32_t *__restrict__ parent_leaf) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int j = nearest[i];
    if (j < 0 || nearest[j] != i) {
        keep[i] = 1;
        return;
    }
    if (i > j) {
        keep[i] = 0;
        return;
    }
    const Cluster a = cl[i], b = cl[j];
    const int id = internal_total - 1 - atomicAdd(node_counter, 1);
    DNode nd;
    nd.a = make_float4(a.b[0], a.b[3], a.b[1], a.b[4]);
    nd.b = make_float4(b.b[0], b.b[3], b.b[1], b.b[4]);
    nd.c = make_float4(a.b[2], a.b[5], b.b[2], b.b[5]);
    nd.d = make_int4(a.id, b.id, 0, 0);
    nodes[id] = nd;
    if (a.id >= 0) parent_internal[a.id] = id; else parent_leaf[~a.id] = id;
    if (b.id >= 0) parent_internal[b.id] = id; else parent_leaf[~b.id] = id;
    Cluster m;
    m.id = id;
    for (int k = 0; k < 3; ++k) {
        m.b[k] = fminf(a.b[k], b.b[k]);
        m.b[3 + k] = fmaxf(a.b[3 + k], b.b[3 + k]);
    }
    cl[i] = m;
    keep[i] = 1;
}

inline unsigned blocks_for(int64_t n, int t) { return unsigned((n + t - 1) / t); }

// ---------------- leaves of several triangles ----------------
// Costs of the leaf decision per unit of a node's surface area: one node visit (two child
// boxes, 64 bytes) and one triangle test (48 bytes and the Moller-Trumbore arithmetic with
// its divide). Measured with leaves of up to 4: a triangle test costing 1 node visit made
// the boxes workload 6 % slower than one triangle per leaf, 2 made it 2 % faster, 3 and 4
// 3 % faster (urban +6 %, sphere +7 %).
constexpr float kCostNode = 1.0f;
constexpr float kCostTri = 3.0f;

__device__ __forceinline__ float box_area(const Box &b) {
    const float dx = b.hi[0] - b.lo[0], dy = b.hi[1] - b.lo[1], dz = b.hi[2] - b.lo[2];
    return dx * dy + dy * dz + dz * dx;
}

// Bottom-up (a leaf's thread climbs while it is the second child to arrive): per node the
// triangle count and the cheaper of its two costs; a node (not the root) whose triangles
// fit a leaf and cost no more as one is marked collapsible.
__global__ void k_leaf_cost(int64_t n, const DNode *__restrict__ nodes, const int32_t *__restrict__ parent_internal,
                            const int32_t *__restrict__ parent_leaf, int *counters, int *count, float *cost,
                            char *collapse, int leaf_max) {
    const int64_t leaf = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (leaf >= n) return;
    int p = parent_leaf[leaf];
    while (p >= 0) {
        __threadfence();
        if (atomicAdd(&counters[p], 1) == 0) return;  // the sibling's thread continues
        __threadfence();
        const DNode nd = nodes[p];
        const int c[2] = {nd.d.x, nd.d.y};
        const volatile int *vcount = count;
        const volatile float *vcost = cost;
        int cnt = 0;
        float sum = 0.f;
        Box u;
        for (int w = 0; w < 2; ++w) {
            const Box b = child_box(nd, w);
            const int cc = c[w] < 0 ? 1 : vcount[c[w]];
            const float cw = c[w] < 0 ? kCostTri : vcost[c[w]];
            cnt += cc;
            sum += box_area(b) * cw;
            for (int a = 0; a < 3; ++a) {
                u.lo[a] = w ? fminf(u.lo[a], b.lo[a]) : b.lo[a];
                u.hi[a] = w ? fmaxf(u.hi[a], b.hi[a]) : b.hi[a];
            }
        }
        const float area = box_area(u);
        const float as_node = kCostNode + (area > 0.f ? sum / area : 0.f);
        const float as_leaf = kCostTri * float(cnt);
        const bool leafy = p != 0 && cnt <= leaf_max && as_leaf <= as_node;
        count[p] = cnt;
        cost[p] = leafy ? as_leaf : as_node;
        collapse[p] = leafy ? 1 : 0;
        p = parent_internal[p];
    }
}

// Per triangle slot: the topmost collapsible ancestor within the leaf-sized part of the
// tree above it (-1: a leaf of its own), and the group's smallest slot.
__global__ void k_leaf_group(int64_t n, const int32_t *__restrict__ parent_internal,
                             const int32_t *__restrict__ parent_leaf, const int *__restrict__ count,
                             const char *__restrict__ collapse, int leaf_max, int32_t *__restrict__ group,
                             int *__restrict__ group_min, char *__restrict__ is_root) {
    const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (t >= n) return;
    int p = parent_leaf[t], root = -1;
    while (p >= 0 && count[p] <= leaf_max) {
        if (collapse[p]) root = p;
        p = parent_internal[p];
    }
    group[t] = root;
    if (root >= 0) {
        atomicMin(&group_min[root], int(t));
        is_root[root] = 1;
    }
}

// sort key: the group's smallest slot, then the slot (groups stay in the Morton order)
__global__ void k_leaf_keys(int64_t n, const int32_t *__restrict__ group, const int *__restrict__ group_min,
                            uint64_t *__restrict__ keys, int32_t *__restrict__ ids) {
    const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (t >= n) return;
    const uint64_t g = group[t] >= 0 ? uint64_t(group_min[group[t]]) : uint64_t(t);
    keys[t] = (g << 32) | uint64_t(t);
    ids[t] = int32_t(t);
}

// new slot of every old slot; records moved; each group's first new slot
__global__ void k_permute_tris(int64_t n, const int32_t *__restrict__ sorted_old, const DTri *__restrict__ src,
                               DTri *__restrict__ dst, int32_t *__restrict__ new_slot) {
    const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const int32_t old = sorted_old[i];
    dst[i] = src[old];
    new_slot[old] = int32_t(i);
}

__global__ void k_leaf_start(int64_t n, const int32_t *__restrict__ group, const int32_t *__restrict__ new_slot,
                             int *__restrict__ start) {
    const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (t >= n || group[t] < 0) return;
    atomicMin(&start[group[t]], new_slot[t]);
}

// child references in the leaf encoding: a collapsed subtree becomes its leaf, a single
// triangle moves to its new slot
__global__ void k_relink(int64_t n_nodes, DNode *nodes, const int32_t *__restrict__ new_slot,
                         const char *__restrict__ is_root, const int *__restrict__ start,
                         const int *__restrict__ count) {
    const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= n_nodes) return;
    int c[2] = {nodes[i].d.x, nodes[i].d.y};
    for (int w = 0; w < 2; ++w) {
        if (c[w] < 0)
            c[w] = ~(new_slot[~c[w]] << 3);
        else if (is_root[c[w]])
            c[w] = ~((start[c[w]] << 3) | (count[c[w]] - 1));
    }
    nodes[i].d.x = c[0];
    nodes[i].d.y = c[1];
}

// ---------------- insertion-based optimisation ----------------
// Bittner, Hapala and Havran (2013): take a subtree out and insert it as the sibling of
// the node where the tree's surface-area cost grows least. Every node searches in
// parallel on a snapshot of the tree (Meister and Bittner 2018); the moves that lower the
// cost claim the six nodes they rewire (the subtree N, its parent P and sibling S, its
// grandparent G, the target X and X's parent) with 64-bit priority locks (gain, node); a
// winner whose target lies inside another winner's subtree withdraws, so no move closes a
// cycle; the winners are applied and the boxes refitted. Index space: internal nodes
// [0, M), triangle slot t at M + t. The root stays node 0 (never moved, never a target,
// never removed). The build's DNodes are written back only when the result passes its
// checks (every node's parent chain ends at node 0; leaves at most 60 deep).
constexpr int kReinsPath = 96;       // deepest parent chain a search handles
constexpr int kReinsStack = 96;      // a search's deferred subtrees
constexpr int kReinsVisits = 8192;   // most subtrees it opens
constexpr int kReinsMaxDepth = 60;   // the traversal stack holds 64 entries

__device__ __forceinline__ Box box_union(const Box &a, const Box &b) {
    Box u;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        u.lo[k] = fminf(a.lo[k], b.lo[k]);
        u.hi[k] = fmaxf(a.hi[k], b.hi[k]);
    }
    return u;
}

// A node of the tree under optimisation: box and children (leaf: kx = -1), one sector.
struct __align__(32) ReinsNode {
    float lo[3];
    int kx;
    float hi[3];
    int ky;
};

__device__ __forceinline__ ReinsNode reins_load(const ReinsNode *__restrict__ t, int i) {
    const float4 *p = reinterpret_cast<const float4 *>(t + i);
    const float4 a = __ldg(p), b = __ldg(p + 1);
    return ReinsNode{{a.x, a.y, a.z}, __float_as_int(a.w), {b.x, b.y, b.z}, __float_as_int(b.w)};
}

__device__ __forceinline__ ReinsNode reins_node(const Box &b, int kx, int ky) {
    return ReinsNode{{b.lo[0], b.lo[1], b.lo[2]}, kx, {b.hi[0], b.hi[1], b.hi[2]}, ky};
}

__device__ __forceinline__ Box box_of(const ReinsNode &n) {
    Box b;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        b.lo[k] = n.lo[k];
        b.hi[k] = n.hi[k];
    }
    return b;
}

__global__ void k_reins_init(int m, const DNode *__restrict__ nodes, const int32_t *__restrict__ par_i, int *rpar,
                             ReinsNode *tree) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const DNode nd = nodes[i];
    const int c[2] = {nd.d.x, nd.d.y};
    int k[2];
    for (int w = 0; w < 2; ++w) {
        k[w] = c[w] >= 0 ? c[w] : m + ~c[w];
        if (c[w] < 0) {
            tree[k[w]] = reins_node(child_box(nd, w), -1, -1);
            rpar[k[w]] = i;
        }
    }
    rpar[i] = par_i[i];
    tree[i] = reins_node(box_union(child_box(nd, 0), child_box(nd, 1)), k[0], k[1]);
}

// The deepest leaf (the root's depth is 0); bad: a parent chain that does not end at node 0
// within the bound.
__global__ void k_reins_depth(int total, int m, const int *__restrict__ rpar, int *max_depth, int *bad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    int d = 0, x = i;
    while (rpar[x] >= 0 && d < 1024) {
        x = rpar[x];
        ++d;
    }
    if (x != 0 || d >= 1024) atomicOr(bad, 1);
    if (i >= m) atomicMax(max_depth, d);
}

// The best place for subtree n: mv_x[n] (-1: none lowers the cost by min_gain) and the
// cost it saves, mv_gain[n]. Taking n out removes its parent P and shrinks the ancestors
// below the one, y, whose other child's subtree (or which itself) receives it; from y up
// nothing changes. So the search climbs from n: `saved` is what the removal saves up to
// here, and each subtree hanging off the path is searched depth first, the child that grows
// less first, with the best place so far as the bound (Meister and Bittner 2018). An open
// subtree is a node and the growth of its ancestors; it is left where even a new parent no
// larger than n would not pay.
// A best-first search of the same space from the root, with the removal's shrunk boxes and
// a 384-entry heap in local memory (5.8 KB per thread), visited fewer nodes but took 2.4 ms
// per pass on 250 k triangles; this one 0.37 (0.39 with a stack of nodes whose children a
// visit has to look up first, 0.65 with the descent as a loop inside the climb), to trees of
// the same node visits per ray (boxes 126, urban 18.6).
__global__ void __launch_bounds__(128) k_reins_search(int total, const int *__restrict__ rpar,
                                                      const ReinsNode *__restrict__ tree, float min_gain, int *mv_x,
                                                      float *mv_gain) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= total) return;
    mv_x[n] = -1;
    const int P = rpar[n];
    if (P < 0) return;
    const int G = rpar[P];
    if (G < 0) return;
    const Box bn = box_of(reins_load(tree, n));
    const float an = box_area(bn);
    const ReinsNode pn = reins_load(tree, P);
    const int S = pn.kx == n ? pn.ky : pn.kx;
    float saved = box_area(box_of(pn)), best = min_gain;
    int bx = -1, visits = 0;
    int2 stack[kReinsStack];  // an open node's children: known when it is opened, so that a
    float grown[kReinsStack]; // visit waits for one load only
    int sp = 0;
    // node x as a place under ancestors that grow by d; its own growth added to d tells
    // whether its subtree is opened
    auto consider = [&](int x, const ReinsNode &t, float &d) {
        const Box b = box_of(t);
        const float au = box_area(box_union(b, bn));
        const float gain = saved - (d + au);
        if (gain > best) {
            best = gain;
            bx = x;
        }
        d += au - box_area(b);
        return t.kx >= 0;
    };
    auto open = [&](const ReinsNode &t, float d) {
        if (sp < kReinsStack && saved - d - an > best) {
            stack[sp] = make_int2(t.kx, t.ky);
            grown[sp++] = d;
        }
    };
    const ReinsNode sn = reins_load(tree, S);
    Box cur = box_of(sn);  // the path's box without n
    if (sn.kx >= 0) open(sn, saved - box_area(cur));  // below the sibling (beside it is where n is)
    int child = P, y = G, steps = 0;
    float saved_next = saved;  // `saved` once the open subtrees are done
    // one loop for both kinds of step, so that a lane that climbs does not wait for one that
    // descends
    while (true) {
        if (sp > 0 && visits < kReinsVisits) {
            const int2 t = stack[--sp];
            const float d = grown[sp];
            if (!(saved - d - an > best)) continue;
            ++visits;
            const ReinsNode l = reins_load(tree, t.x), r = reins_load(tree, t.y);
            float dl = d, dr = d;
            const bool kl = consider(t.x, l, dl), kr = consider(t.y, r, dr);
            if (dl < dr) {
                if (kr) open(r, dr);
                if (kl) open(l, dl);
            } else {
                if (kl) open(l, dl);
                if (kr) open(r, dr);
            }
            continue;
        }
        sp = 0;
        saved = saved_next;
        if (steps > 0 && child != 0) {  // beside the ancestor passed last
            const float gain = saved - box_area(box_union(cur, bn));
            if (gain > best) {
                best = gain;
                bx = child;
            }
        }
        if (y < 0) break;
        if (++steps > kReinsPath) return;
        const ReinsNode yn = reins_load(tree, y);
        const int c = yn.kx == child ? yn.ky : yn.kx;
        const ReinsNode cn = reins_load(tree, c);
        float d = 0.f;
        if (consider(c, cn, d)) open(cn, d);
        cur = box_union(cur, box_of(cn));
        saved_next = saved + (box_area(box_of(yn)) - box_area(cur));
        child = y;
        y = rpar[y];
    }
    if (bx >= 0) {
        mv_x[n] = bx;
        mv_gain[n] = best;
    }
}

// The nodes a move rewires: n, P, S, G, X, X's parent.
__device__ __forceinline__ void reins_touched(int n, int x, const int *rpar, const ReinsNode *tree, int *t) {
    const int P = rpar[n];
    t[0] = n;
    t[1] = P;
    t[2] = tree[P].kx == n ? tree[P].ky : tree[P].kx;
    t[3] = rpar[P];
    t[4] = x;
    t[5] = rpar[x];
}

__global__ void k_reins_lock(int total, const int *__restrict__ rpar, const ReinsNode *__restrict__ tree,
                             const int *__restrict__ mv_x, const float *__restrict__ mv_gain,
                             unsigned long long *lock) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= total || mv_x[n] < 0) return;
    int t[6];
    reins_touched(n, mv_x[n], rpar, tree, t);
    for (int k = 0; k < 6; ++k)
        if (t[k] < 0 || t[k] >= total) return;
    const unsigned long long key = (static_cast<unsigned long long>(__float_as_uint(mv_gain[n])) << 32) | unsigned(n);
    for (int k = 0; k < 6; ++k) atomicMax(&lock[t[k]], key);
}

__global__ void k_reins_claim(int total, const int *__restrict__ rpar, const ReinsNode *__restrict__ tree,
                              const int *__restrict__ mv_x, const float *__restrict__ mv_gain,
                              const unsigned long long *__restrict__ lock, char *moving) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= total) return;
    moving[n] = 0;
    if (mv_x[n] < 0) return;
    int t[6];
    reins_touched(n, mv_x[n], rpar, tree, t);
    const unsigned long long key = (static_cast<unsigned long long>(__float_as_uint(mv_gain[n])) << 32) | unsigned(n);
    for (int k = 0; k < 6; ++k)
        if (t[k] < 0 || t[k] >= total || lock[t[k]] != key) return;
    moving[n] = 1;
}

// A winner stays unless its target is inside another winner's subtree.
__global__ void k_reins_keep(int total, const int *__restrict__ rpar, const int *__restrict__ mv_x,
                             const char *__restrict__ moving, char *keep) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= total) return;
    keep[n] = 0;
    if (!moving[n]) return;
    int x = mv_x[n];
    for (int steps = 0; x >= 0; x = rpar[x], ++steps)
        if (steps >= 1024 || (x != n && moving[x])) return;
    keep[n] = 1;
}

__global__ void k_reins_apply(int total, int *rpar, ReinsNode *tree, const int *__restrict__ mv_x,
                              const char *__restrict__ keep, int *applied) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n >= total || !keep[n]) return;
    auto replace = [&](int parent, int from, int to) {
        if (tree[parent].kx == from)
            tree[parent].kx = to;
        else
            tree[parent].ky = to;
    };
    const int X = mv_x[n];
    const int P = rpar[n], G = rpar[P];
    const int S = tree[P].kx == n ? tree[P].ky : tree[P].kx;
    // take n out: S replaces P below G
    replace(G, P, S);
    rpar[S] = G;
    // P becomes the parent of X and n, in X's place
    const int XP = rpar[X];
    replace(XP, X, P);
    rpar[P] = XP;
    tree[P].kx = X;
    tree[P].ky = n;
    rpar[X] = P;
    rpar[n] = P;
    atomicAdd(applied, 1);
}

// Boxes from the leaves up: a leaf's thread climbs while it is the second child to arrive.
// A child's box comes from another SM: read and written in the L2.
__global__ void k_reins_refit(int total, int m, const int *__restrict__ rpar, ReinsNode *tree, int *counters,
                              int *bad) {
    const int leaf = m + blockIdx.x * blockDim.x + threadIdx.x;
    if (leaf >= total) return;
    int p = rpar[leaf];
    for (int steps = 0; p >= 0; p = rpar[p], ++steps) {
        if (steps >= 1024) {
            atomicOr(bad, 1);
            return;
        }
        __threadfence();
        if (atomicAdd(&counters[p], 1) == 0) return;
        __threadfence();
        float4 *t = reinterpret_cast<float4 *>(tree);
        const float4 w0 = __ldcg(t + 2 * p), w1 = __ldcg(t + 2 * p + 1);
        const int kx = __float_as_int(w0.w), ky = __float_as_int(w1.w);
        const float4 a0 = __ldcg(t + 2 * kx), a1 = __ldcg(t + 2 * kx + 1);
        const float4 b0 = __ldcg(t + 2 * ky), b1 = __ldcg(t + 2 * ky + 1);
        __stcg(t + 2 * p, make_float4(fminf(a0.x, b0.x), fminf(a0.y, b0.y), fminf(a0.z, b0.z), w0.w));
        __stcg(t + 2 * p + 1, make_float4(fmaxf(a1.x, b1.x), fmaxf(a1.y, b1.y), fmaxf(a1.z, b1.z), w1.w));
    }
}

// Back to the build's layout: DNodes with child boxes and references (leaf: ~slot),
// internal and leaf parent links.
__global__ void k_reins_write(int m, const int *__restrict__ rpar, const ReinsNode *__restrict__ tree, DNode *nodes,
                              int32_t *par_i, int32_t *par_l) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const int kx = tree[i].kx, ky = tree[i].ky;
    const Box l = box_of(tree[kx]), r = box_of(tree[ky]);
    DNode nd;
    nd.a = make_float4(l.lo[0], l.hi[0], l.lo[1], l.hi[1]);
    nd.b = make_float4(r.lo[0], r.hi[0], r.lo[1], r.hi[1]);
    nd.c = make_float4(l.lo[2], l.hi[2], r.lo[2], r.hi[2]);
    nd.d = make_int4(kx < m ? kx : ~(kx - m), ky < m ? ky : ~(ky - m), 0, 0);
    nodes[i] = nd;
    par_i[i] = rpar[i];
    if (kx >= m) par_l[kx - m] = i;
    if (ky >= m) par_l[ky - m] = i;
}

}  // namespace

int g_bvh_builder = 0;  // 0: PLOC, 1: LBVH (Karras)
int g_bvh_leaf_max = 4;  // triangles per leaf (1..8)
int g_bvh_optimize = 32;  // largest number of insertion passes after the build (0: none)

// The temporaries of one stage of the build, in one allocation (each piece on a 256-byte
// boundary). With one each, 47 allocations and their releases took 2.3 ms of a build of
// 250 k triangles.
struct Temps {
    void *block = nullptr;
    std::vector<std::pair<void **, size_t>> parts;
    template <typename T> void want(T **p, size_t bytes) {
        parts.emplace_back(reinterpret_cast<void **>(p), (bytes + 255) & ~size_t(255));
    }
    bool get(std::string &err) {
        size_t sum = 0;
        for (const auto &q : parts) sum += q.second;
        if (!dev_alloc(&block, sum, err)) return false;
        char *at = static_cast<char *>(block);
        for (const auto &q : parts) {
            *q.first = at;
            at += q.second;
        }
        return true;
    }
    ~Temps() { cudaFree(block); }
};

// Insertion passes over the binary tree of a build (par_i/par_l and the DNodes, leaves
// referenced as ~slot); stops when a pass moves fewer than 1 in 20,000 nodes (stopping
// at 1 in 4,000 left the urban scene 8 % more node visits per ray; searching every node in the
// first and last passes only and a quarter of the rest between built 250 k triangles in 18.8
// ms instead of 23.1, to trees in which the urban frame took 0-8 % longer). Returns 0
// (also when the result failed its checks and the build's tree was kept), 2 or 3.
static int optimize_tree(SceneDev &s, int64_t nt, int32_t *par_i, int32_t *par_l, cudaStream_t st,
                         std::string &err) {
    if (g_bvh_optimize <= 0 || nt < 4 || nt >= (int64_t(1) << 30)) return 0;
    const int m = int(nt - 1), total = int(2 * nt - 1);
    int *rpar = nullptr, *mv_x = nullptr, *counters = nullptr, *scal = nullptr;
    ReinsNode *tree = nullptr;
    float *mv_gain = nullptr;
    unsigned long long *lock = nullptr;
    char *moving = nullptr, *keep = nullptr;
    int rc = 0;
    Temps t;
    do {
        t.want(&rpar, sizeof(int) * total);
        t.want(&mv_x, sizeof(int) * total);
        t.want(&counters, sizeof(int) * m);
        t.want(&scal, sizeof(int) * 4);
        t.want(&tree, sizeof(ReinsNode) * total);
        t.want(&mv_gain, sizeof(float) * total);
        t.want(&lock, sizeof(unsigned long long) * total);
        t.want(&moving, size_t(total));
        t.want(&keep, size_t(total));
        if (!t.get(err)) {
            rc = 3;
            break;
        }
        const int T = 256;
        k_reins_init<<<blocks_for(m, T), T, 0, st>>>(m, s.nodes, par_i, rpar, tree);
        note_launches(1);
        ReinsNode root;
        if (cudaMemcpyAsync(&root, tree, sizeof(root), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess) {
            err = "BVH optimisation: reading the root box failed";
            rc = 2;
            break;
        }
        const float dx = root.hi[0] - root.lo[0], dy = root.hi[1] - root.lo[1], dz = root.hi[2] - root.lo[2];
        const float min_gain = 1e-6f * (dx * dy + dy * dz + dz * dx);
        int h[4] = {0, 0, 0, 0};
        for (int pass = 0; pass < g_bvh_optimize; ++pass) {
            cudaMemsetAsync(scal, 0, sizeof(int) * 4, st);
            cudaMemsetAsync(lock, 0, sizeof(unsigned long long) * total, st);
            cudaMemsetAsync(counters, 0, sizeof(int) * m, st);
            k_reins_search<<<blocks_for(total, 128), 128, 0, st>>>(total, rpar, tree, min_gain, mv_x, mv_gain);
            k_reins_lock<<<blocks_for(total, T), T, 0, st>>>(total, rpar, tree, mv_x, mv_gain, lock);
            k_reins_claim<<<blocks_for(total, T), T, 0, st>>>(total, rpar, tree, mv_x, mv_gain, lock, moving);
            k_reins_keep<<<blocks_for(total, T), T, 0, st>>>(total, rpar, mv_x, moving, keep);
            k_reins_apply<<<blocks_for(total, T), T, 0, st>>>(total, rpar, tree, mv_x, keep, scal);
            k_reins_refit<<<blocks_for(nt, T), T, 0, st>>>(total, m, rpar, tree, counters, scal + 1);
            note_launches(6);
            if (cudaMemcpyAsync(h, scal, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                cudaStreamSynchronize(st) != cudaSuccess) {
                err = "BVH optimisation pass failed";
                rc = 2;
                break;
            }
            if (h[1] || h[0] < std::max(1, total / 20000)) break;
        }
        // a failed check keeps the build's own tree (every loop of a pass is bounded on any links)
        if (rc || h[1]) break;
        cudaMemsetAsync(scal, 0, sizeof(int) * 4, st);
        k_reins_depth<<<blocks_for(total, T), T, 0, st>>>(total, m, rpar, scal + 2, scal + 1);
        note_launches(1);
        if (cudaMemcpyAsync(h, scal, sizeof(h), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
            cudaStreamSynchronize(st) != cudaSuccess) {
            err = "BVH optimisation check failed";
            rc = 2;
            break;
        }
        if (h[1] || h[2] > kReinsMaxDepth) break;
        k_reins_write<<<blocks_for(m, T), T, 0, st>>>(m, rpar, tree, s.nodes, par_i, par_l);
        note_launches(1);
        if (cudaStreamSynchronize(st) != cudaSuccess) {
            err = "BVH optimisation write-back failed";
            rc = 2;
        }
    } while (false);
    return rc;
}

// Leaves of several triangles over a built binary topology (parent links of the build).
static int collapse_leaves(SceneDev &s, int64_t nt, const int32_t *par_i, const int32_t *par_l, int *counters,
                           cudaStream_t st, std::string &err) {
    const int64_t n_nodes = s.node_count;
    const int leaf_max = std::min(std::max(g_bvh_leaf_max, 1), 8);
    int *count = nullptr, *group_min = nullptr, *start = nullptr;
    float *cost = nullptr;
    char *collapse = nullptr, *is_root = nullptr;
    int32_t *group = nullptr, *ids = nullptr, *ids2 = nullptr, *new_slot = nullptr;
    uint64_t *keys = nullptr, *keys2 = nullptr;
    DTri *tris2 = nullptr;
    void *tmp = nullptr;
    size_t tmp_bytes = 0;
    int rc = 0;
    Temps t;
    do {
        if (cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, keys, keys2, ids, ids2, int(nt), 0, 64, st) !=
            cudaSuccess) {
            err = "leaf sort size query failed";
            rc = 2;
            break;
        }
        t.want(&tmp, tmp_bytes);
        t.want(&count, sizeof(int) * n_nodes);
        t.want(&cost, sizeof(float) * n_nodes);
        t.want(&collapse, size_t(n_nodes));
        t.want(&is_root, size_t(n_nodes));
        t.want(&group_min, sizeof(int) * n_nodes);
        t.want(&start, sizeof(int) * n_nodes);
        t.want(&group, sizeof(int32_t) * nt);
        t.want(&ids, sizeof(int32_t) * nt);
        t.want(&ids2, sizeof(int32_t) * nt);
        t.want(&new_slot, sizeof(int32_t) * nt);
        t.want(&keys, sizeof(uint64_t) * nt);
        t.want(&keys2, sizeof(uint64_t) * nt);
        if (!t.get(err) || !dev_alloc(&tris2, sizeof(DTri) * nt, err)) {
            rc = 3;
            break;
        }
        cudaMemsetAsync(counters, 0, sizeof(int) * n_nodes, st);
        cudaMemsetAsync(count, 0x7f, sizeof(int) * n_nodes, st);  // > leaf_max until written
        cudaMemsetAsync(collapse, 0, size_t(n_nodes), st);
        cudaMemsetAsync(is_root, 0, size_t(n_nodes), st);
        cudaMemsetAsync(group_min, 0x7f, sizeof(int) * n_nodes, st);
        cudaMemsetAsync(start, 0x7f, sizeof(int) * n_nodes, st);
        const int T = 256;
        if (leaf_max > 1) {
            k_leaf_cost<<<blocks_for(nt, T), T, 0, st>>>(nt, s.nodes, par_i, par_l, counters, count, cost, collapse,
                                                          leaf_max);
            note_launches(1);
        }
        k_leaf_group<<<blocks_for(nt, T), T, 0, st>>>(nt, par_i, par_l, count, collapse, leaf_max, group, group_min,
                                                       is_root);
        k_leaf_keys<<<blocks_for(nt, T), T, 0, st>>>(nt, group, group_min, keys, ids);
        note_launches(2);
        if (cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, keys, keys2, ids, ids2, int(nt), 0, 64, st) !=
            cudaSuccess) {
            err = "leaf sort failed";
            rc = 2;
            break;
        }
        k_permute_tris<<<blocks_for(nt, T), T, 0, st>>>(nt, ids2, s.tris, tris2, new_slot);
        k_leaf_start<<<blocks_for(nt, T), T, 0, st>>>(nt, group, new_slot, start);
        k_relink<<<blocks_for(n_nodes, T), T, 0, st>>>(n_nodes, s.nodes, new_slot, is_root, start, count);
        note_launches(4);
        const cudaError_t e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) {
            err = std::string("BVH leaves: ") + cudaGetErrorString(e);
            rc = 2;
            break;
        }
        std::swap(s.tris, tris2);
    } while (false);
    cudaFree(tris2);
    return rc;
}

// PLOC topology over the sorted leaves. Returns 0 or an hsr_status-like code.
static int build_ploc(SceneDev &s, int64_t nt, const int32_t *ids2, const float *lo, const float *hi,
                      int32_t *par_i, int32_t *par_l, int *depth, cudaStream_t st, std::string &err) {
    const int n0 = int(nt);
    Cluster *c0 = nullptr, *c1 = nullptr;
    int *nearest = nullptr, *counter = nullptr, *num_sel = nullptr;
    char *keep = nullptr;
    void *tmp = nullptr;
    size_t tmp_bytes = 0;
    int rc = 0;
    Temps t;
    do {
        cub::DeviceSelect::Flagged(nullptr, tmp_bytes, c0, keep, c1, num_sel, n0, st);
        t.want(&tmp, tmp_bytes);
        t.want(&c0, sizeof(Cluster) * n0);
        t.want(&c1, sizeof(Cluster) * n0);
        t.want(&nearest, sizeof(int) * n0);
        t.want(&counter, sizeof(int) * 2);
        t.want(&num_sel, sizeof(int) * 2);
        t.want(&keep, size_t(n0));
        if (!t.get(err)) {
            rc = 3;
            break;
        }
        cudaMemsetAsync(counter, 0, sizeof(int), st);
        k_ploc_init<<<blocks_for(nt, 256), 256, 0, st>>>(nt, ids2, lo, hi, c0);
        note_launches(1);
        int n = n0;
        int iterations = 0;
        while (n > 1 && iterations < 100000) {
            k_ploc_nearest<<<blocks_for(n, 256 / kPlocLanes), 256, 0, st>>>(n, c0, nearest);
            k_ploc_merge<<<blocks_for(n, 256), 256, 0, st>>>(n, nearest, c0, keep, s.nodes, counter, n0 - 1, par_i,
                                                             par_l);
            if (cub::DeviceSelect::Flagged(tmp, tmp_bytes, c0, keep, c1, num_sel, n, st) != cudaSuccess) {
                err = "PLOC compaction failed";
                rc = 2;
                break;
            }
            note_launches(3);
            int h = 0;
            if (cudaMemcpyAsync(&h, num_sel, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                cudaStreamSynchronize(st) != cudaSuccess) {
                err = "PLOC iteration failed";
                rc = 2;
                break;
            }
            if (h >= n) {  // no pair merged: impossible for a correct nearest search; stop safely
                err = "PLOC made no progress";
                rc = 2;
                break;
            }
            std::swap(c0, c1);
            n = h;
            ++iterations;
        }
        if (rc) break;
        k_leaf_depth<<<blocks_for(nt, 256), 256, 0, st>>>(nt, par_i, par_l, depth + 1);
        note_launches(1);
    } while (false);
    cudaStreamSynchronize(st);
    return rc;
}

namespace {

// Nodes of every subtree, from the nodes with two leaves up: the second of two internal
// children to arrive goes on. Climbs out of a collapsed leaf end where the parent no longer
// refers to the node. A tree can be as deep as it has nodes (triangles on one place merge one
// by one, and a tree that deep keeps no insertion pass), so that bounds the climb; at any
// depth it is one visit per node.
__global__ void k_tree_sizes(int64_t n, const DNode *__restrict__ nodes, const int32_t *__restrict__ par_i, int *size,
                             int *arrived) {
    const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (t >= n || nodes[t].d.x >= 0 || nodes[t].d.y >= 0) return;
    int i = int(t), s = 1;
    for (int64_t steps = 0; steps < n; ++steps) {
        __stcg(&size[i], s);
        if (i == 0) return;
        const int p = par_i[i];
        if (p < 0) return;
        const int4 d = nodes[p].d;
        if (d.x != i && d.y != i) return;
        if (d.x >= 0 && d.y >= 0) {
            __threadfence();
            if (atomicAdd(&arrived[p], 1) == 0) return;
            __threadfence();
        }
        s = 1 + (d.x >= 0 ? __ldcg(&size[d.x]) : 0) + (d.y >= 0 ? __ldcg(&size[d.y]) : 0);
        i = p;
    }
}

// A reachable node's place in depth-first order: a first child follows its parent, a second
// one its sibling's subtree; summed over the path to the root. placed: how many there were.
// The climbs add up to half the depth squared on a chain, as k_leaf_depth's do; one of 20,000
// triangles on one place builds in 0.81 s, with the host's walk it took 1.31.
__global__ void k_tree_place(int64_t n, const DNode *__restrict__ nodes, const int32_t *__restrict__ par_i,
                             const int *__restrict__ size, int64_t out_count, DNode *__restrict__ out, int *placed) {
    const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (t >= n) return;
    auto first = [&](const int4 &d) { return d.x >= 0 ? size[d.x] : 0; };
    int64_t id = 0;
    int c = int(t);
    for (int64_t steps = 0; c != 0; ++steps) {
        const int p = par_i[c];
        if (p < 0 || steps >= n) return;
        const int4 d = nodes[p].d;
        if (d.x == c)
            id += 1;
        else if (d.y == c)
            id += 1 + first(d);
        else
            return;
        c = p;
    }
    if (id >= out_count) return;
    DNode nd = nodes[t];
    const int skip = first(nd.d);
    if (nd.d.x >= 0) nd.d.x = int(id) + 1;
    if (nd.d.y >= 0) nd.d.y = int(id) + 1 + skip;
    out[id] = nd;
    atomicAdd(placed, 1);
}

}  // namespace

// The reachable nodes renumbered in depth-first order from the root (each node's first
// child follows it in memory, so a descent reads neighbouring nodes), the nodes inside
// collapsed leaves dropped: the node array shrinks to the reachable nodes. `counters` holds
// one int per node. (The host's walk over a downloaded copy took 15 ms of the 49 of a
// build of 250 k triangles.)
static int renumber_depth_first(SceneDev &s, const int32_t *par_i, int *counters, cudaStream_t st, std::string &err) {
    const int64_t n = s.node_count;
    if (n < 2) return 0;
    int *size = nullptr;
    DNode *compact = nullptr;
    if (!dev_alloc(&size, sizeof(int) * size_t(n + 1), err)) return 3;
    auto fail = [&](int rc, const char *what) {
        if (rc == 2) err = what;
        cudaFree(size);
        cudaFree(compact);
        return rc;
    };
    const int T = 256;
    cudaMemsetAsync(counters, 0, sizeof(int) * size_t(n), st);
    cudaMemsetAsync(size, 0, sizeof(int) * size_t(n + 1), st);
    k_tree_sizes<<<blocks_for(n, T), T, 0, st>>>(n, s.nodes, par_i, size, counters);
    note_launches(1);
    int count = 0, placed = 0;
    if (cudaMemcpyAsync(&count, size, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return fail(2, "BVH layout: subtree sizes failed");
    if (count < 1 || count > n) return fail(2, "BVH layout: the tree is not a tree");
    // the array shrinks to the reachable nodes
    if (!dev_alloc(&compact, sizeof(DNode) * size_t(count), err)) return fail(3, "");
    k_tree_place<<<blocks_for(n, T), T, 0, st>>>(n, s.nodes, par_i, size, count, compact, size + n);
    note_launches(1);
    if (cudaMemcpyAsync(&placed, size + n, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
        return fail(2, "BVH layout failed");
    if (placed != count) return fail(2, "BVH layout: the tree is not a tree");
    cudaFree(size);
    cudaFree(s.nodes);
    s.nodes = compact;
    s.node_count = count;
    return 0;
}

// Builds tris/nodes for `scene` from device vertex/index arrays. Returns 0, 2 (CUDA
// error), 3 (out of memory) or 4 (too many triangles).
int bvh_build(SceneDev &s, const float *d_v, int64_t nv, const int32_t *d_idx, int64_t nt, cudaStream_t st,
              std::string &err) {
    (void)nv;
    if (nt >= (int64_t(1) << 28)) {  // a leaf reference holds the slot in 28 bits
        err = "scenes are limited to 2^28 - 1 triangles";
        return 4;
    }
    s.tri_count = nt;
    const int64_t n_nodes = nt >= 2 ? nt - 1 : 1;
    s.node_count = n_nodes;
    if (!dev_alloc(&s.tris, sizeof(DTri) * (size_t)std::max<int64_t>(nt, 1), err)) return 3;
    if (!dev_alloc(&s.nodes, sizeof(DNode) * (size_t)n_nodes, err)) return 3;
    if (nt < 2) {
        // 0 or 1 triangle: one root whose two children are both slot 0. With no triangle,
        // slot 0 is all zeros (zero determinant: never hit). A second visit of the only
        // triangle is harmless. (An inverted box is not empty under the min/max slab test.)
        if (cudaMemsetAsync(s.tris, 0, sizeof(DTri), st) != cudaSuccess) return 2;
        DNode root;
        const float inf = std::numeric_limits<float>::infinity();
        root.a = make_float4(inf, -inf, inf, -inf);
        root.b = make_float4(inf, -inf, inf, -inf);
        root.c = make_float4(inf, -inf, inf, -inf);
        root.d = make_int4(-1, -1, 0, 0);  // ~0 = slot 0
        if (nt == 1) {
            float hv[9];
            int32_t hi[3];
            if (cudaMemcpyAsync(hi, d_idx, sizeof(hi), cudaMemcpyDeviceToHost, st) != cudaSuccess) return 2;
            cudaStreamSynchronize(st);
            for (int k = 0; k < 3; ++k)
                if (cudaMemcpyAsync(hv + 3 * k, d_v + 3 * (int64_t)hi[k], 3 * sizeof(float), cudaMemcpyDeviceToHost,
                                    st) != cudaSuccess)
                    return 2;
            cudaStreamSynchronize(st);
            float lo[3], hiB[3];
            for (int a = 0; a < 3; ++a) {
                float mn = std::min(hv[a], std::min(hv[3 + a], hv[6 + a]));
                float mx = std::max(hv[a], std::max(hv[3 + a], hv[6 + a]));
                float pad = std::max(std::fabs(mn), std::fabs(mx)) * 4e-6f + 1e-6f;
                lo[a] = mn - pad;
                hiB[a] = mx + pad;
            }
            root.a = make_float4(lo[0], hiB[0], lo[1], hiB[1]);
            root.c.x = lo[2];
            root.c.y = hiB[2];
            DTri T;
            T.v0 = make_float4(hv[0], hv[1], hv[2], 0.f);  // bit pattern of int 0
            T.e1 = make_float4(hv[3] - hv[0], hv[4] - hv[1], hv[5] - hv[2], 0.f);
            T.e2 = make_float4(hv[6] - hv[0], hv[7] - hv[1], hv[8] - hv[2], 0.f);
            if (cudaMemcpyAsync(s.tris, &T, sizeof(T), cudaMemcpyHostToDevice, st) != cudaSuccess) return 2;
        }
        if (cudaMemcpyAsync(s.nodes, &root, sizeof(root), cudaMemcpyHostToDevice, st) != cudaSuccess) return 2;
        cudaStreamSynchronize(st);
        s.max_depth = nt == 1 ? 1 : 0;
        s.leaf_count = nt;
        return 0;
    }

    float *lo = nullptr, *hi = nullptr;
    unsigned *cb = nullptr;
    uint64_t *keys = nullptr, *keys2 = nullptr;
    int32_t *ids = nullptr, *ids2 = nullptr, *par_i = nullptr, *par_l = nullptr;
    int *counters = nullptr, *depth = nullptr;
    void *tmp = nullptr;
    size_t tmp_bytes = 0;
    int rc = 0;
    Temps t;
    auto fail = [&](int code) {
        rc = code;
        return code;
    };
    do {
        if (cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, keys, keys2, ids, ids2, (int)nt, 0, 63, st) !=
            cudaSuccess) {
            err = "radix sort size query failed";
            fail(2);
            break;
        }
        t.want(&tmp, tmp_bytes);
        t.want(&lo, sizeof(float) * 3 * nt);
        t.want(&hi, sizeof(float) * 3 * nt);
        t.want(&cb, sizeof(unsigned) * 6);
        t.want(&keys, sizeof(uint64_t) * nt);
        t.want(&keys2, sizeof(uint64_t) * nt);
        t.want(&ids, sizeof(int32_t) * nt);
        t.want(&ids2, sizeof(int32_t) * nt);
        t.want(&par_i, sizeof(int32_t) * n_nodes);
        t.want(&par_l, sizeof(int32_t) * nt);
        t.want(&counters, sizeof(int) * n_nodes);
        t.want(&depth, sizeof(int) * 2);
        if (!t.get(err)) {
            fail(3);
            break;
        }
        unsigned init[6] = {0xffffffffu, 0xffffffffu, 0xffffffffu, 0u, 0u, 0u};
        cudaMemcpyAsync(cb, init, sizeof(init), cudaMemcpyHostToDevice, st);
        cudaMemsetAsync(counters, 0, sizeof(int) * n_nodes, st);
        cudaMemsetAsync(depth, 0, sizeof(int) * 2, st);
        cudaMemsetAsync(par_i, 0xff, sizeof(int32_t) * n_nodes, st);  // root keeps -1
        const int T = 256;
        k_bounds<<<blocks_for(nt, T), T, 0, st>>>(d_v, d_idx, nt, lo, hi, cb);
        k_morton<<<blocks_for(nt, T), T, 0, st>>>(lo, hi, nt, cb, keys, ids);
        note_launches(2);
        if (cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, keys, keys2, ids, ids2, (int)nt, 0, 63, st) !=
            cudaSuccess) {
            err = "radix sort failed";
            fail(2);
            break;
        }
        k_write_tris<<<blocks_for(nt, T), T, 0, st>>>(d_v, d_idx, ids2, nt, s.tris);
        if (g_bvh_builder == 0) {
            note_launches(1);
            const int prc = build_ploc(s, nt, ids2, lo, hi, par_i, par_l, depth, st, err);
            if (prc) {
                fail(prc);
                break;
            }
        } else {
            k_karras<<<blocks_for(nt - 1, T), T, 0, st>>>(keys2, nt, s.nodes, par_i, par_l);
            k_refit<<<blocks_for(nt, T), T, 0, st>>>(nt, ids2, lo, hi, s.nodes, par_i, par_l, counters, depth);
            k_leaf_depth<<<blocks_for(nt, T), T, 0, st>>>(nt, par_i, par_l, depth + 1);
            note_launches(4);
        }
        cudaError_t e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) {
            err = std::string("BVH build: ") + cudaGetErrorString(e);
            fail(2);
            break;
        }
        const int orc = optimize_tree(s, nt, par_i, par_l, st, err);
        if (orc) {
            fail(orc);
            break;
        }
        if (g_bvh_optimize > 0) {  // the depth of the tree as it now is
            cudaMemsetAsync(depth + 1, 0, sizeof(int), st);
            k_leaf_depth<<<blocks_for(nt, T), T, 0, st>>>(nt, par_i, par_l, depth + 1);
            note_launches(1);
        }
        const int lrc = collapse_leaves(s, nt, par_i, par_l, counters, st, err);
        if (lrc) {
            fail(lrc);
            break;
        }
        const int drc = renumber_depth_first(s, par_i, counters, st, err);
        if (drc) {
            fail(drc);
            break;
        }
        int hd[2];
        cudaMemcpy(hd, depth, sizeof(hd), cudaMemcpyDeviceToHost);
        s.max_depth = hd[1];
        s.leaf_count = nt;
        const int mrc = measure_density(s, st, err);
        if (mrc) {
            fail(mrc);
            break;
        }
    } while (false);
    return rc;
}

namespace {

// Triangle records of new vertex positions: slot s keeps its triangle (the original id in
// v0.w), as k_write_tris forms them.
__global__ void k_refit_tris(int64_t nt, const float *__restrict__ v, const int32_t *__restrict__ idx,
                             DTri *__restrict__ tris) {
    const int64_t s = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (s >= nt) return;
    const float idbits = tris[s].v0.w;
    const int64_t t = __float_as_int(idbits);
    const float *p0 = v + 3 * int64_t(idx[3 * t + 0]);
    const float *p1 = v + 3 * int64_t(idx[3 * t + 1]);
    const float *p2 = v + 3 * int64_t(idx[3 * t + 2]);
    DTri T;
    T.v0 = make_float4(p0[0], p0[1], p0[2], idbits);
    T.e1 = make_float4(p1[0] - p0[0], p1[1] - p0[1], p1[2] - p0[2], 0.f);
    T.e2 = make_float4(p2[0] - p0[0], p2[1] - p0[1], p2[2] - p0[2], 0.f);
    tris[s] = T;
}

// One level of the bottom-up refit: each node's two child boxes from its children (a
// leaf: the padded boxes of its triangles, as k_bounds pads them; a node: the union of
// its own two boxes, refitted one level deeper).
__global__ void k_refit_level(int64_t count, const int32_t *__restrict__ order, DNode *nodes,
                              const DTri *__restrict__ tris, const float *__restrict__ v,
                              const int32_t *__restrict__ idx) {
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= count) return;
    const int i = order[k];
    const int c[2] = {nodes[i].d.x, nodes[i].d.y};
    Box bx[2];
    for (int w = 0; w < 2; ++w) {
        for (int a = 0; a < 3; ++a) {
            bx[w].lo[a] = __int_as_float(0x7f800000);
            bx[w].hi[a] = -__int_as_float(0x7f800000);
        }
        if (c[w] < 0) {
            const int ref = ~c[w];
            for (int slot = ref >> 3; slot <= (ref >> 3) + (ref & 7); ++slot) {
                const int64_t t = __float_as_int(tris[slot].v0.w);
                for (int a = 0; a < 3; ++a) {
                    const float x0 = v[3 * int64_t(idx[3 * t + 0]) + a];
                    const float x1 = v[3 * int64_t(idx[3 * t + 1]) + a];
                    const float x2 = v[3 * int64_t(idx[3 * t + 2]) + a];
                    const float mn = fminf(x0, fminf(x1, x2)), mx = fmaxf(x0, fmaxf(x1, x2));
                    const float pad = fmaxf(fabsf(mn), fabsf(mx)) * 4e-6f + 1e-6f;
                    bx[w].lo[a] = fminf(bx[w].lo[a], mn - pad);
                    bx[w].hi[a] = fmaxf(bx[w].hi[a], mx + pad);
                }
            }
        } else {
            const DNode cn = nodes[c[w]];
            const Box b0 = child_box(cn, 0), b1 = child_box(cn, 1);
            for (int a = 0; a < 3; ++a) {
                bx[w].lo[a] = fminf(b0.lo[a], b1.lo[a]);
                bx[w].hi[a] = fmaxf(b0.hi[a], b1.hi[a]);
            }
        }
    }
    DNode &n = nodes[i];
    n.a = make_float4(bx[0].lo[0], bx[0].hi[0], bx[0].lo[1], bx[0].hi[1]);
    n.b = make_float4(bx[1].lo[0], bx[1].hi[0], bx[1].lo[1], bx[1].hi[1]);
    n.c = make_float4(bx[0].lo[2], bx[0].hi[2], bx[1].lo[2], bx[1].hi[2]);
}

}  // namespace

int bvh_refit(SceneDev &s, const float *d_v, cudaStream_t st, std::string &err) {
    const int64_t nt = s.tri_count;
    if (nt < 2) {  // the one-node tree of 0 or 1 triangle: built again
        cudaFree(s.tris);
        cudaFree(s.nodes);
        s.tris = nullptr;
        s.nodes = nullptr;
        return bvh_build(s, d_v, s.vertex_count, s.indices, nt, st, err);
    }
    if (!s.refit_order) {
        // the reachable internal nodes, level by level from the root (host breadth-first
        // walk over the child references)
        std::vector<DNode> h(size_t(s.node_count));
        if (cudaMemcpy(h.data(), s.nodes, sizeof(DNode) * h.size(), cudaMemcpyDeviceToHost) != cudaSuccess) {
            err = "refit: node download failed";
            return 2;
        }
        std::vector<int32_t> order{0}, next;
        std::vector<int64_t> levels{0};
        size_t begin = 0;
        while (begin < order.size()) {
            const size_t end = order.size();
            for (size_t k = begin; k < end; ++k)
                for (int c : {h[order[k]].d.x, h[order[k]].d.y})
                    if (c >= 0) order.push_back(c);
            levels.push_back(int64_t(end));
            begin = end;
        }
        if (!dev_alloc(&s.refit_order, sizeof(int32_t) * order.size(), err)) return 3;
        if (cudaMemcpy(s.refit_order, order.data(), sizeof(int32_t) * order.size(), cudaMemcpyHostToDevice) !=
            cudaSuccess) {
            err = "refit: order upload failed";
            return 2;
        }
        s.refit_levels = levels;
    }
    const int T = 256;
    k_refit_tris<<<blocks_for(nt, T), T, 0, st>>>(nt, d_v, s.indices, s.tris);
    note_launches(1);
    for (size_t l = s.refit_levels.size() - 1; l-- > 0;) {  // deepest level first
        const int64_t b = s.refit_levels[l], e = s.refit_levels[l + 1];
        k_refit_level<<<blocks_for(e - b, T), T, 0, st>>>(e - b, s.refit_order + b, s.nodes, s.tris, d_v, s.indices);
        note_launches(1);
    }
    const cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        err = std::string("BVH refit: ") + cudaGetErrorString(e);
        return 2;
    }
    return 0;
}

}  // namespace hsr
