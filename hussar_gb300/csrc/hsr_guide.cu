// GuidingWrapper::step (libhussar/include/hussar/integrators/path.h:119-126) on the
// device, one CTA per pose with the tree staged in shared memory (at most 2048 nodes):
//   build   leaf energy = sqrt(sum w d^2 * leaf area) (second moment, path.h:232),
//           internal energy = sum of its children, first-child probability = share;
//   copy    sampling tree := built training tree;
//   refine  new training topology: a subtree whose energy fraction is at most the split
//           threshold (0.005, path.h:230) collapses to a leaf; a leaf above it splits in
//           halves (recursively, each half taking half the fraction); statistics reset.
// Every pass runs level by level over the CTA: depths and fractions from the root down,
// energies and subtree sizes from the leaves up. New nodes are numbered as a depth-first
// walk would meet them (the k-th node to split, in preorder, has children 1 + 2k and
// 2 + 2k); with the subtrees' sizes known, each node's place in that order follows from its
// parent's. A thread walking the tree alone, as before, waited on every link: 49, 130 and
// 153 us for the three steps of a 2^18-sample guided run, now 9, 24 and 38 us (the run
// 650 -> 400 us, with a warp per halved leaf; one thread per leaf 68, 51 and 44 us). It
// still does the
// refinement where the new tree would not fit, since what fits then depends on the order,
// and every pass of a tree that no step could have made (one written from outside, with
// shared children or more levels).
#include "hsr_guide.cuh"
#include "hsr_internal.h"

namespace hsr {

namespace {

__global__ void k_guide_reset(int P, int *samp_child, float *samp_p, int *train_child, float *train_acc,
                              int *train_count) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P) return;
    samp_child[size_t(p) * kGuideMaxNodes] = -1;
    samp_p[size_t(p) * kGuideMaxNodes] = 0.5f;
    train_child[size_t(p) * kGuideMaxNodes] = -1;
    float *acc = train_acc + size_t(p) * kGuideMaxNodes * 3;
    acc[0] = acc[1] = acc[2] = 0.f;
    train_count[p] = 1;
}

// The refinement's depth-first walk on one thread: the new child links and node count.
__device__ int refine_serial(const int *tc, const float *e, int *fresh) {
    int ncount = 1;
    struct Item {
        int old;
        float f;
        int d;
        int ni;
    } stack[2 * kGuideMaxDepth + 4];
    int top = 0;
    stack[top++] = Item{0, 1.f, 0, 0};
    while (top > 0) {
        const Item it = stack[--top];
        const bool internal = it.old >= 0 && tc[it.old] >= 0;
        const bool split = it.f > kGuideSplitThreshold && it.d < kGuideMaxDepth && ncount + 2 <= kGuideMaxNodes &&
                           top + 2 <= 2 * kGuideMaxDepth + 4;
        if (!split) {
            fresh[it.ni] = -1;
            continue;
        }
        const int c = ncount;
        ncount += 2;
        fresh[it.ni] = c;
        if (internal) {
            const int oc = tc[it.old];
            const float eo = e[it.old];
            const float f0 = eo > 0.f ? it.f * (e[oc] / eo) : 0.5f * it.f;
            const float f1 = eo > 0.f ? it.f * (e[oc + 1] / eo) : 0.5f * it.f;
            stack[top++] = Item{oc + 1, f1, it.d + 1, c + 1};
            stack[top++] = Item{oc, f0, it.d + 1, c};
        } else {
            stack[top++] = Item{-1, 0.5f * it.f, it.d + 1, c + 1};
            stack[top++] = Item{-1, 0.5f * it.f, it.d + 1, c};
        }
    }
    return ncount;
}

// Depths (children always follow their parent), then energies bottom-up, on one thread.
__device__ void energies_serial(const int *tc, const float *m2, int count, int *depth, float *e) {
    depth[0] = 0;
    for (int i = 0; i < count; ++i) {
        const int c = tc[i];
        if (c >= 0 && c + 1 < count) depth[c] = depth[c + 1] = depth[i] + 1;
    }
    for (int i = count - 1; i >= 0; --i) {
        const int c = tc[i];
        if (c < 0) {
            const float area = ldexpf(1.f, -depth[i]);
            e[i] = sqrtf(fmaxf(m2[i], 0.f) * area);
        } else {
            e[i] = e[c] + e[c + 1];
        }
    }
}

// How many times a leaf of fraction f at depth d is halved.
__device__ __forceinline__ int halvings(float f, int d) {
    int m = 0;
    while (f > kGuideSplitThreshold && d + m < kGuideMaxDepth) {
        f *= 0.5f;
        ++m;
    }
    return m;
}

__global__ void __launch_bounds__(256) k_guide_step(const int *__restrict__ active, int *samp_child, float *samp_p,
                                                    int *train_child, float *train_acc, int *train_count) {
    const int p = blockIdx.x;
    if (!active[p]) return;  // uniform over the CTA
    __shared__ int tc_s[kGuideMaxNodes];       // training topology
    __shared__ float f_s[kGuideMaxNodes];      // second-moment statistic, then energy fraction
    __shared__ float e_s[kGuideMaxNodes];      // energies
    __shared__ int fresh_s[kGuideMaxNodes];    // the new topology
    __shared__ short split_s[kGuideMaxNodes];  // nodes that split in the new subtree
    __shared__ short pre_s[kGuideMaxNodes];    // splits before the node, in preorder
    __shared__ short ni_s[kGuideMaxNodes];     // the node's place in the new tree, -1: none
    __shared__ unsigned char depth_s[kGuideMaxNodes];
    __shared__ int s_ncount;
    const size_t base = size_t(p) * kGuideMaxNodes;
    int *tc = train_child + base;
    float *acc = train_acc + base * 3;
    int *sc = samp_child + base;
    float *sp = samp_p + base;
    const int tid = threadIdx.x, step = blockDim.x;
    const int count = min(max(train_count[p], 1), kGuideMaxNodes);
    constexpr unsigned char kUnreached = 255;
    for (int i = tid; i < count; i += step) {
        tc_s[i] = tc[i];
        f_s[i] = acc[3 * i + 2];
        depth_s[i] = i == 0 ? 0 : kUnreached;
    }
    __syncthreads();
    int levels = 0;     // the deepest level
    bool odd = false;   // a tree of another shape
    for (int d = 0; d <= kGuideMaxDepth; ++d) {
        bool more = false;
        for (int i = tid; i < count; i += step) {
            if (depth_s[i] != d) continue;
            const int c = tc_s[i];
            if (c < 0) continue;
            if (c + 1 < count && d < kGuideMaxDepth) {
                depth_s[c] = depth_s[c + 1] = (unsigned char)(d + 1);
                more = true;
            } else {
                odd = true;
            }
        }
        if (!__syncthreads_or(more)) break;
        levels = d + 1;
    }
    // every node but the root is one link's: nodes reached = 1 + 2 x nodes with a link
    int spare = 0;
    for (int i = tid; i < count; i += step)
        if (depth_s[i] != kUnreached) spare += tc_s[i] >= 0 ? -1 : 1;
    if (tid == 0) s_ncount = 0;
    __syncthreads();
    atomicAdd(&s_ncount, spare);
    odd = __syncthreads_or(odd) || s_ncount != 1;
    __syncthreads();
    if (odd) {
        if (tid == 0) energies_serial(tc_s, f_s, count, fresh_s, e_s);
        __syncthreads();
    } else {
        // energies from the leaves up
        for (int d = levels; d >= 0; --d) {
            for (int i = tid; i < count; i += step) {
                if (depth_s[i] != d) continue;
                const int c = tc_s[i];
                if (c < 0) {
                    const float area = ldexpf(1.f, -d);
                    e_s[i] = sqrtf(fmaxf(f_s[i], 0.f) * area);
                } else {
                    e_s[i] = e_s[c] + e_s[c + 1];
                }
            }
            __syncthreads();
        }
    }
    // copy to the sampling tree
    for (int i = tid; i < count; i += step) {
        const int c = tc_s[i];
        sc[i] = c;
        if (c >= 0 && (odd || depth_s[i] != kUnreached)) {
            const float s = e_s[c] + e_s[c + 1];
            sp[i] = s > 0.f ? e_s[c] / s : 0.5f;
        } else {
            sp[i] = 0.5f;
        }
    }
    const float total = e_s[0];
    int ncount = count;  // no information: keep the topology
    if (total > 0.f && !odd) {
        // the fractions of the nodes whose ancestors all split (ni_s 0 marks them), and how
        // many nodes split below each
        for (int i = tid; i < count; i += step) ni_s[i] = -1;
        __syncthreads();
        if (tid == 0) {
            f_s[0] = 1.f;
            ni_s[0] = 0;
        }
        __syncthreads();
        for (int d = 0; d < levels; ++d) {
            for (int i = tid; i < count; i += step) {
                if (depth_s[i] != d || ni_s[i] < 0) continue;
                const int c = tc_s[i];
                const float f = f_s[i], eo = e_s[i];
                if (c < 0 || !(f > kGuideSplitThreshold)) continue;
                f_s[c] = eo > 0.f ? f * (e_s[c] / eo) : 0.5f * f;
                f_s[c + 1] = eo > 0.f ? f * (e_s[c + 1] / eo) : 0.5f * f;
                ni_s[c] = ni_s[c + 1] = 0;
            }
            __syncthreads();
        }
        for (int d = levels; d >= 0; --d) {
            for (int i = tid; i < count; i += step) {
                if (depth_s[i] != d || ni_s[i] < 0) continue;
                const int c = tc_s[i];
                int n = 0;
                if (c < 0)
                    n = (1 << halvings(f_s[i], d)) - 1;
                else if (f_s[i] > kGuideSplitThreshold && d < kGuideMaxDepth)
                    n = 1 + split_s[c] + split_s[c + 1];
                split_s[i] = short(n);
            }
            __syncthreads();
        }
        ncount = 1 + 2 * int(split_s[0]);
        if (ncount <= kGuideMaxNodes) {
            if (tid == 0) pre_s[0] = 0;
            __syncthreads();
            for (int d = 0; d <= levels; ++d) {
                for (int i = tid; i < count; i += step) {
                    if (depth_s[i] != d || ni_s[i] < 0) continue;
                    const int c = tc_s[i], at = pre_s[i];
                    if (split_s[i] == 0) {
                        fresh_s[ni_s[i]] = -1;
                    } else if (c >= 0) {
                        fresh_s[ni_s[i]] = 1 + 2 * at;
                        ni_s[c] = short(1 + 2 * at);
                        ni_s[c + 1] = short(2 + 2 * at);
                        pre_s[c] = short(at + 1);
                        pre_s[c + 1] = short(at + 1 + split_s[c]);
                    }
                }
                __syncthreads();
            }
            // a leaf halved m times becomes a complete binary tree of m levels: node `path`
            // of level k has its place by the subtrees to its left. A warp takes one at a time.
            const int lane = tid & 31;
            for (int i0 = tid - lane; i0 < count; i0 += step) {
                const int i = i0 + lane;
                unsigned todo = __ballot_sync(
                    0xffffffffu, i < count && depth_s[i] != kUnreached && ni_s[i] >= 0 && tc_s[i] < 0 && split_s[i] > 0);
                for (; todo; todo &= todo - 1) {
                    const int leaf = i0 + __ffs(int(todo)) - 1;
                    const int m = 31 - __clz(int(split_s[leaf]) + 1), at = pre_s[leaf], root = ni_s[leaf];
                    for (int v = 1 + lane; v < 2 << m; v += 32) {
                        const int k = 31 - __clz(v);
                        int q = at, n = root;
                        for (int b = k - 1; b >= 0; --b) {
                            const int right = (v >> b) & 1;
                            n = 1 + 2 * q + right;
                            q += 1 + right * ((1 << (m - (k - b))) - 1);
                        }
                        fresh_s[n] = k < m ? 1 + 2 * q : -1;
                    }
                }
            }
            __syncthreads();
        }
    }
    if (total > 0.f && (odd || ncount > kGuideMaxNodes)) {
        __syncthreads();  // the copy above has read the energies' links
        if (tid == 0) s_ncount = refine_serial(tc_s, e_s, fresh_s);
        __syncthreads();
        ncount = s_ncount;
    }
    if (total > 0.f)
        for (int i = tid; i < ncount; i += step) tc[i] = fresh_s[i];
    for (int i = tid; i < 3 * ncount; i += step) acc[i] = 0.f;
    if (tid == 0) train_count[p] = ncount;
}

}  // namespace

size_t guide_bytes_per_pose() {
    // samp child + p, train child + 3 acc, count, and the guided schedule (kGuideMaxIters
    // iterations x 32 B) with the total weight
    return size_t(kGuideMaxNodes) * (4 + 4 + 4 + 12) + size_t(kGuideMaxIters) * 32 + 8 + 16;
}

int launch_guide_reset(int P, int *samp_child, float *samp_p, int *train_child, float *train_acc, int *train_count,
                       cudaStream_t st) {
    k_guide_reset<<<(P + 127) / 128, 128, 0, st>>>(P, samp_child, samp_p, train_child, train_acc, train_count);
    note_launches(1);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

int launch_guide_step(int P, const int *active, int *samp_child, float *samp_p, int *train_child, float *train_acc,
                      int *train_count, cudaStream_t st) {
    k_guide_step<<<P, 256, 0, st>>>(active, samp_child, samp_p, train_child, train_acc, train_count);
    note_launches(1);
    return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // namespace hsr
