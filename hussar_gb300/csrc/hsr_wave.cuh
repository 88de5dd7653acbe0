// Wavefront form of the radar path tracer (geometrical-optics mode, the reference's
// default, path.h:156): the same per-path arithmetic as the one-thread-per-sample
// kernel, reorganised so that warps stay converged.
//
// A persistent CTA of 256 threads keeps a stack of up to 512 live path states in
// shared memory (four CTAs per SM: 64 registers; 27 to 43 KB of shared memory each plus the
// range row; the rest of the SM's 256 KB is L1 for the BVH) and alternates two stages:
//   GENERATE  (at most 256 live paths, or the queue threshold of the launch): 256 new
//             samples, one per thread: Halton point,
//             antenna ray, closest hit; paths that hit something are pushed.
//   EXTEND    (otherwise): 256 paths popped, one per thread: specular reflection,
//             next-event estimate towards RX (shadow ray, PO re-radiation, filtering,
//             phase), and the next closest hit; survivors are pushed back.
// Every next-event contribution is splatted by its warp cooperatively: lane l owns
// window offset l-16 of Frame::splat<16>, so one contribution's 33 bins are 33 distinct
// shared-memory addresses updated in one pass. The CTA's range row lives in shared
// memory and is flushed to the pose's FP64 accumulators when the CTA changes pose.
// Work items are (pose, tile) pairs pulled from a device counter, one at a time or in
// runs that shrink as the counter nears its end (pull_items).
//
// The kernel is a template over the phase mode; hsr_wave.cu instantiates the FP32
// reference-phase forms without multiply-add contraction (so the float expressions round
// as the CPU restatement does) and hsr_wave_split.cu the split-phase forms with it.
//
// Mixed batches (kMixed, the serving loop): each pose names its own resident scene,
// chirp, range-bin count and accumulator row (PoseJob). A CTA works on one pose at a
// time, so these are CTA-uniform: thread 0 copies the pose's job into shared memory
// when the CTA switches pose, and the arithmetic is the uniform kernel's.
#pragma once
#include "hsr_path.cuh"

namespace hsr {

namespace {

constexpr int kThreads = 256;
// GENERATE hands its samples to threads grouped by the cell of their primary sample point
// (4 x 2 cells of the unit square): a warp's primary rays leave the antenna in one part
// of the sphere, and their hits, pushed together, come back as neighbouring stack entries
constexpr int kPrimaryCells = 8;

// A CTA's live path states: a stack of kThreads + kQueue entries, where kQueue bounds the
// paths left when GENERATE runs (the queue threshold). Three capacities are built: 384
// entries (thresholds up to 128), 320 (up to 64), whose 5 KB less shared
// memory per CTA leaves more of the SM's L1 to the BVH (4 % on the dense boxes scenes,
// before their neighbourhood lists), and 512 (up to 256), whose fuller
// EXTEND stages pay where the BVH stays in L1 anyway (7 % on the sphere bench).
template <int kCap> struct WaveShared {
    float ox[kCap], oy[kCap], oz[kCap];  // hit point (origin of the next segment)
    float dx[kCap], dy[kCap], dz[kCap];  // incoming direction
    float h[6][kCap];                    // incoming H field (re, im) x 3
    float nx[kCap], ny[kCap], nz[kCap];  // faceforwarded normal at the hit
    float r[kCap], cosT[kCap], freq[kCap];
    int depth[kCap];
    // the phase input: time of flight (FP32 reference phase, as float) or the FP64 path
    // length (split phase); each mode carries only its own
    double tlen[kCap];
    int count;      // paths stacked from entry 0 up
    int count_far;  // neighbourhood lists: paths stacked from the last entry down
    int pose, pending_pose, exhausted;
    long long gen, gen_end, pending_first, pending_last;
    long long item, item_end;   // work items pulled and not yet started
    int item_want;              // length of the last run of items pulled
    long long since_flush;      // samples generated since the row was last flushed
    PoseJob job;                // mixed batches: the current pose's scene, chirp and row
    int cell_count[kThreads / 32][kPrimaryCells];  // GENERATE: samples per warp and cell
    int cell_total[kPrimaryCells];
    short order[kThreads];      // GENERATE: stage sample offset of each thread
    FfAnt ff[2];                // far-field launches: the current pose's TX and RX
    float max_dist, bandwidth;  // mixed batches: derived from job.rf
};

struct Guided {  // the guiding part of a path's state
    float x0, x1, pdf;
    cf gw;
};

// Guided launches keep the guiding part of each stacked path (primary sample, pdf,
// weight) in five more [kCap] arrays after the training sums (`gst`, null otherwise).
constexpr int kGuideStackFields = 5;

// Neighbourhood lists: the mark on a stacked path's depth that its origin, direction and
// field are those of a ray the list did not settle; without it they are a hit's.
constexpr int kRayPending = 1 << 30;

// The slots of the lanes that push a path at the lower or (`far`) the upper end: one shared
// atomic per warp and end. The whole warp calls.
template <int kCap> __device__ __forceinline__ int claim_slot(WaveShared<kCap> &S, bool push, bool far) {
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const unsigned lower = __ballot_sync(0xffffffffu, push && !far);
    const unsigned upper = __ballot_sync(0xffffffffu, push && far);
    int base = 0;
    if (lane == 0 && lower) base = atomicAdd(&S.count, __popc(lower));
    if (lane == 1 && upper) base = atomicAdd(&S.count_far, __popc(upper));
    const int low = __shfl_sync(0xffffffffu, base, 0) + __popc(lower & below);  // < kCap by construction (see k_wave)
    const int up = __shfl_sync(0xffffffffu, base, 1) + __popc(upper & below);
    return far ? kCap - 1 - up : low;
}

template <int kPhase, int kCap>
__device__ __forceinline__ void store_path(WaveShared<kCap> &S, float *gst, int slot, f3 o, f3 d, const c3 &H, f3 n,
                                           float time, float r, float cosT, float freq, int depth, double plen,
                                           const Guided &g) {
    S.ox[slot] = o.x;
    S.oy[slot] = o.y;
    S.oz[slot] = o.z;
    S.dx[slot] = d.x;
    S.dy[slot] = d.y;
    S.dz[slot] = d.z;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        S.h[2 * i][slot] = H.v[i].re;
        S.h[2 * i + 1][slot] = H.v[i].im;
    }
    S.nx[slot] = n.x;
    S.ny[slot] = n.y;
    S.nz[slot] = n.z;
    S.r[slot] = r;
    S.cosT[slot] = cosT;
    S.freq[slot] = freq;
    S.depth[slot] = depth;
    if (kPhase == HSR_PHASE_REFERENCE_FP32)
        reinterpret_cast<float *>(S.tlen)[slot] = time;
    else
        S.tlen[slot] = plen;
    if (gst) {
        gst[slot] = g.x0;
        gst[kCap + slot] = g.x1;
        gst[2 * kCap + slot] = g.pdf;
        gst[3 * kCap + slot] = g.gw.re;
        gst[4 * kCap + slot] = g.gw.im;
    }
}

// The lanes that call push a path each.
template <int kPhase, int kCap>
__device__ __forceinline__ void push_path(WaveShared<kCap> &S, float *gst, f3 o, f3 d, const c3 &H, f3 n, float time,
                                          float r, float cosT, float freq, int depth, double plen, const Guided &g) {
    // one shared atomic per warp: the lanes pushing here take consecutive slots
    const unsigned active = __activemask();
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(active) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(&S.count, __popc(active));
    base = __shfl_sync(active, base, leader);
    const int slot = base + __popc(active & ((1u << lane) - 1u));  // < kCap by construction (see k_wave)
    store_path<kPhase>(S, gst, slot, o, d, H, n, time, r, cosT, freq, depth, plen, g);
}

// A stable counting sort of the stage's items by key (< kPrimaryCells; the items
// [0, n) of the stage, thread t holding item t's key, threads t >= n holding
// kPrimaryCells): afterwards S.order[j] is the item thread j works on, for j < n. The
// order is the same in every run. Called by the whole CTA.
template <int kCap> __device__ __forceinline__ void order_by_key(WaveShared<kCap> &S, int key) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int rank = __popc(peers & ((1u << lane) - 1u));
    if (lane < kPrimaryCells) S.cell_count[warp][lane] = 0;
    __syncwarp();
    if (rank == 0 && key < kPrimaryCells) S.cell_count[warp][key] = __popc(peers);
    __syncthreads();
    if (tid < kPrimaryCells) {
        int t = 0;
#pragma unroll
        for (int w = 0; w < kThreads / 32; ++w) t += S.cell_count[w][tid];
        S.cell_total[tid] = t;
    }
    __syncthreads();
    if (key < kPrimaryCells) {
        int base = rank;
        for (int k = 0; k < key; ++k) base += S.cell_total[k];
        for (int w = 0; w < warp; ++w) base += S.cell_count[w][key];
        S.order[base] = short(tid);  // < n: the keyed items are the stage's
    }
    __syncthreads();
}

// The bookkeeping of a hit of the segment (o, d) (path.h:407-442, GO mode): the triangle
// slot and its distance. Returns true (and the new state) when the path continues.
__device__ __forceinline__ bool arrive(const DTri *tris, int slot, float th, f3 o, f3 d, float &time, float &r,
                                       double &plen, f3 &hp, f3 &n, float &cosT) {
    DTri T = load_tri(tris, slot);
    n = hit_normal(T, d);
    hp = add3(o, scl3(th, d));
    cosT = fabsf(dot3(n, neg3(d)));
    if (cosT < 0.001f) return false;
    r += th;
    time += th / kSpeedOfLight;
    plen += double(th);
    return true;
}

// Closest hit of the segment (o, d) and its bookkeeping. Returns true (and the new state)
// when the path continues with a stored hit. The reference's zero-field test (path.h:413,
// 439) is the caller's: in GO mode the field does not change across the hit, so testing it
// before or after is the same.
__device__ __forceinline__ bool walk(const TraceParams &p, const DNode *nodes, const DTri *tris, f3 o, f3 d,
                                     float &time, float &r, double &plen, f3 &hp, f3 &n, float &cosT) {
    float th;
    int primh;
    const int slot = closest_hit<false>(nodes, tris, o, d, kEpsilon, CUDART_INF_F, th, primh, p.status, nullptr);
    return slot >= 0 && arrive(tris, slot, th, o, d, time, r, plen, hp, n, cosT);
}

// Dense scenes: the closest hit of each lane's segment (o, d), or -1, from the pose's list
// (`local`) or the BVH. The whole warp calls, lanes without a segment with active = false,
// and leaves together: run by the lanes that have one, what follows the query ran once for each
// group of lanes that left it together (14 of 32 lanes active on the boxes; sweep of 96
// poses 16.1 ms against 14.3).
__device__ __forceinline__ int warp_closest(bool active, bool local, const LocalList &L, const TraceParams &p,
                                            const DNode *nodes, const DTri *tris, f3 o, f3 d, float &th) {
    int slot = -1, prim;
    if (!local)
        slot = closest_hit_in_step(active, nodes, tris, o, d, kEpsilon, CUDART_INF_F, th, prim, p.status);
    else if (active)
        slot = closest_local(L, tris, o, d, th);
    __syncwarp();
    return slot;
}

// Whether each lane's segment from o along d meets anything up to `dist`, in the same manner.
__device__ __forceinline__ bool warp_occluded(bool active, bool local, const LocalList &L, const TraceParams &p,
                                              const DNode *nodes, const DTri *tris, f3 o, f3 d, float dist) {
    bool hit = false;
    if (!local)
        hit = any_hit_in_step(active, nodes, tris, o, d, kEpsilon, dist, p.status);
    else if (active)
        hit = any_local(L, tris, o, d, dist);
    __syncwarp();
    return hit;
}

// PathTracer::run's derived chirp quantities (path.h:240, radar.h:128-130).
__device__ __forceinline__ float max_distance(const hsr_rf_config &rf) {
    return rf.adcRate / rf.freqSlope * kSpeedOfLight;
}
__device__ __forceinline__ float chirp_bandwidth(const hsr_rf_config &rf) { return rf.freqSlope * rf.rampTime; }

// Pulls the run of work items a CTA takes next: [S.item, S.item_end), empty (false) once
// the counter has passed `total`. With p.item_run = 0 it is one item. With p.item_run = R
// it is a third of the CTA's share of what is left, between 1 and R items (guided
// self-scheduling, Polychronopoulos and Kuck 1987): long runs of one pose while there is
// plenty, which drain the path stack and flush the row rarely, and single 256-sample items
// at the end, so that the CTAs finish together. What is left is estimated from the CTA's
// last run, assuming that every other CTA has pulled as much since: a fresh look at the
// counter would cost a second trip to the L2 per pull.
// Fixed 4096-sample items left the chip idle wherever a launch had few of them. Whole calls,
// fixed items -> runs, on the tree-walking forms (dense scenes did not have lists yet): one
// dihedral pose of 2^14 samples (4 items for 608 CTAs) 137 -> 98 us; 33 poses on 100 k
// triangles of boxes (1.7 M samples) 21.9 -> 12.2 ms; 27 far-field poses x 2^14 747 -> 480
// us; urban, 12 x 2^19 samples, 8.3 -> 7.3 ms; 96 poses on 1 M triangles (14 M samples)
// 101 -> 91 ms.
// A CTA that changes pose drains its stack and reads the next pose's list, so runs are as
// long as the balance allows: half the share was too much for poses that differ in cost
// (with lists, 96 boxes poses of 2^13 .. 2^18 samples 14.4 ms with R = 64 items; a third
// 12.7, a quarter 12.8, a sixth 13.1), and R = 16 items too little for large batches (256
// boxes poses of 2^16 .. 2^22 samples 0.88e9 paths/s, R = 32 1.04e9, R = 64 1.20e9, R = 256
// 1.20e9).
template <class Shared>
__device__ __forceinline__ bool pull_items(const TraceParams &p, Shared &S, long long total) {
    long long want = 1;
    if (p.item_run > 0) {
        const long long left = total - S.item_end - S.item_want * (long long)gridDim.x;
        want = min((long long)p.item_run, max(1ll, left / (3ll * gridDim.x)));
        S.item_want = int(want);
    }
    S.item = (long long)atomicAdd((unsigned long long *)p.work_counter, (unsigned long long)want);
    S.item_end = min(S.item + want, total);
    return S.item < total;
}

// FP64 accumulator row of a pose: the pose's job row (mixed), its listed row, or
// pose-major rows of 2N.
template <bool kMixed, class Shared>
__device__ __forceinline__ double *pose_row(const TraceParams &p, const Shared &S, int pose) {
    if (kMixed) return p.acc + S.job.acc_offset;
    return p.acc + (p.acc_row ? __ldg(&p.acc_row[pose]) : 2 * int64_t(pose) * p.samples);
}

// Dynamic shared memory of a launch: the stack, the range row of N bins and, guided, the
// CTA's training sums and the guiding part of the stacked paths; then, on dense scenes, the
// pose's neighbourhood list (local_offset).
template <int kCap> __host__ __device__ constexpr size_t wave_smem_of(int samples, bool guided) {
    return sizeof(WaveShared<kCap>) + 2 * size_t(samples) * sizeof(float) +
           (guided ? (kGuideMaxNodes + kGuideStackFields * kCap) * sizeof(float) : 0);
}
template <int kCap> __host__ __device__ constexpr size_t local_offset(int samples, bool guided) {
    return (wave_smem_of<kCap>(samples, guided) + 15) & ~size_t(15);
}
template <int kQueue> size_t wave_smem_for(int samples, bool guided, bool local = false) {
    constexpr int kCap = kThreads + kQueue;
    return local ? local_offset<kCap>(samples, guided) + sizeof(LocalList) : wave_smem_of<kCap>(samples, guided);
}

// Four CTAs per SM (64 registers): the spills cost less than the latency the extra
// warps hide (measured: 1.2x on the sphere bench, 1.13x on the serving mix over two).
// kLazy (the field_on_hit launch shape): with indirect-only paths, a primary ray's
// antenna field is formed only once the ray has hit something.
// kLocal (dense scenes): each pose has a neighbourhood list (p.local, hsr_local.cuh). The
// stack (384 entries; 512 leave the L1 too little beside the list: 0-5 % slower) then has two
// ends. Paths whose hit point lies in the list's cube are at the lower end; their EXTEND
// asks the list alone: the occlusion query is settled by it, and a closest-hit query that is
// not becomes a pending ray at the upper end. The upper end holds those and the paths
// outside the cube; its EXTEND asks the BVH. A stage works on one end (the fuller one), so a
// warp never waits for one lane's tree traversal among 31 list lookups. The stages' parts
// run by the whole warp, which meets after each query; in this manner the other forms lose
// 4 % (urban) to 29 % (sphere, whose rays mostly miss at the root) and keep theirs.
// field_on_hit and coherent_order don't apply here (the coherent order costs 7 to 20 %).
template <int kPhase, bool kMixed, int kQueue, bool kFF = false, bool kLazy = false, bool kLocal = false>
__global__ void __launch_bounds__(kThreads, 4) k_wave(TraceParams p) {
    constexpr int kCap = kThreads + kQueue;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WaveShared<kCap> &S = *reinterpret_cast<WaveShared<kCap> *>(smem_raw);
    float *s_re = reinterpret_cast<float *>(smem_raw + sizeof(WaveShared<kCap>));
    float *s_im = s_re + p.samples;  // the row is sized for the largest N of the launch
    // guided launches: the CTA's training sums (second moment per training-tree node)
    float *s_g = s_re + 2 * p.samples;
    float *gst = p.do_guide ? s_g + kGuideMaxNodes : nullptr;
    // the pose's list, after the row (and the guiding part): 16-byte aligned
    LocalList &L = *reinterpret_cast<LocalList *>(
        smem_raw + (kLocal ? local_offset<kCap>(p.samples, p.do_guide != 0) : 0));
    const int tid = threadIdx.x;
    const hsr_tracer_flags &fl = p.flags;
    // the scene, chirp and row of the current pose: launch-uniform, or the pose's job
    const hsr_rf_config &rf = kMixed ? S.job.rf : p.rf;
    const float maxDist0 = max_distance(p.rf), bandwidth0 = chirp_bandwidth(p.rf);
#define HSR_NODES (kMixed ? S.job.nodes : p.nodes)
#define HSR_TRIS (kMixed ? S.job.tris : p.tris)
#define HSR_N (kMixed ? S.job.samples : p.samples)
#define HSR_MAXDIST (kMixed ? S.max_dist : maxDist0)
#define HSR_BANDWIDTH (kMixed ? S.bandwidth : bandwidth0)
    const long long total = __ldg(&p.tile_start[p.pose_count]);
    static_assert(kQueue <= kWaveMaxQueueThreshold, "queue threshold bound");
    const int queue_threshold = (p.queue_threshold > 0 && p.queue_threshold < kQueue) ? p.queue_threshold : kQueue;

    for (int k = tid; k < 2 * p.samples; k += kThreads) s_re[k] = 0.f;
    if (p.do_guide)
        for (int k = tid; k < kGuideMaxNodes; k += kThreads) s_g[k] = 0.f;
    if (tid == 0) {
        S.count = 0;
        S.count_far = 0;
        S.pose = -1;
        S.pending_pose = -1;
        S.exhausted = 0;
        S.gen = S.gen_end = 0;
        S.item = S.item_end = 0;
        S.item_want = 0;
        S.since_flush = 0;
    }
    __syncthreads();

    PoseCtx pc;
    int cur_pose = -1;

    while (true) {
        // thread 0 pulls work items while the generation range is used up
        if (tid == 0) {
            while (S.gen >= S.gen_end && !S.exhausted && S.pending_pose < 0) {
                if (S.item >= S.item_end && !pull_items(p, S, total)) {
                    S.exhausted = 1;
                    break;
                }
                // the pulled items of one pose are one sample range
                const int pose = find_pose(p.tile_start, p.pose_count, S.item);
                const long long pose_first = __ldg(&p.tile_start[pose]);
                const long long stop = min(S.item_end, (long long)__ldg(&p.tile_start[pose + 1]));
                const long long first = (S.item - pose_first) * p.tile;
                const long long last = min((stop - pose_first) * p.tile, (long long)__ldg(&p.budget[pose]));
                S.item = stop;
                if (pose == S.pose) {
                    S.gen = first;
                    S.gen_end = last;
                } else {
                    S.pending_pose = pose;
                    S.pending_first = first;
                    S.pending_last = last;
                }
            }
        }
        __syncthreads();
        const int count = S.count, count_far = kLocal ? S.count_far : 0;
        const long long gen = S.gen, gen_end = S.gen_end;
        const int pending = S.pending_pose;
        const int exhausted = S.exhausted;
        const long long since_flush = S.since_flush;
        __syncthreads();  // every thread has read the shared control words

        if (since_flush >= kFlushSamples && cur_pose >= 0) {
            // bound the FP32 partial sums: move the row to the FP64 accumulators
            flush_row(pose_row<kMixed>(p, S, cur_pose), s_re, s_im, HSR_N);
            if (p.do_guide) flush_guide(pc, s_g);
            if (tid == 0) S.since_flush = 0;
            __syncthreads();
            continue;
        }

        if (gen < gen_end && count + count_far <= queue_threshold) {
            // ---------------- GENERATE ----------------
            if (tid == 0) {
                S.gen = min(gen + (long long)kThreads, gen_end);
                S.since_flush += S.gen - gen;
            }
            // the stage's samples gen + [0, n), ordered by primary cell: thread t traces
            // sample gen + S.order[t]
            const int n_stage = int(min((long long)kThreads, gen_end - gen));
            const bool ordered = !kLocal && p.coherent_order;
            if (ordered) {
                int key = kPrimaryCells;
                if (tid < n_stage) {
                    const uint64_t h0 = uint64_t(pc.offset + gen + tid);
                    const float u0 = halton(h0, 1 + kGet2DFirst), u1 = halton(h0, 1 + kGet2DSecond);
                    key = min(int(u0 * 4.f), 3) * 2 + min(int(u1 * 2.f), 1);
                }
                order_by_key(S, key);
            }
            const long long s = gen + (ordered && tid < n_stage ? S.order[tid] : tid);
            const bool local = kLocal && L.planes > 0;  // the sensor lies in the cube
            bool has_item = false;
            float4 item = make_float4(0.f, 0.f, 0.f, 0.f);
            if constexpr (kLocal) {
                const bool mine = s < gen_end;
                float freq = 0.f;
                Guided g{0.f, 0.f, 1.f, cf{0.f, 0.f}};
                f3 o = mk3(0.f, 0.f, 0.f), d = mk3(0.f, 0.f, 1.f);
                c3 H;
                bool onward = false;
                if (mine) {
                    const uint64_t hindex = uint64_t(pc.offset + s);
                    freq = rf.startFreq + halton(hindex, 0) * HSR_BANDWIDTH;
                    g.x0 = halton(hindex, 1 + kGet2DFirst);
                    g.x1 = halton(hindex, 1 + kGet2DSecond);
                    if (fl.doGuiding) g.pdf = guide_sample(pc.samp_child, pc.samp_p, g.x0, g.x1);
                    o = pc.tx.pos;
                    antenna_sample<kPhase == HSR_PHASE_REFERENCE_FP32>(pc.tx, g.x0, g.x1, d, H);
                    H = c3_scl(H, 1.f / g.pdf);
                    if (!fl.onlyIndirect) {
                        NeeOut ne;
                        if (nee_eval<kPhase, false>(p, HSR_NODES, HSR_TRIS, rf, HSR_N, pc.tx, pc.rx, 0, o, d,
                                                         mk3(0.f, 0.f, 0.f), mk3(0.f, 0.f, 0.f), H, H, 0.f, 0.0, 0.f,
                                                         1.f, freq, pc.weight, ne, nullptr, nullptr, nullptr,
                                                         local ? &L : nullptr) &&
                            ne.splat) {
                            if (pc.fine_row) {
                                splat_fine(pc.fine_row, p.fine_bins, ne.sample, ne.value);
                            } else {
                                item = splat_item(ne.sample, ne.value);
                                has_item = true;
                            }
                        }
                    }
                    onward = !(0 >= fl.maxDepth || 0.f >= HSR_MAXDIST) && !c3_is_zero(H);
                }
                float time = 0.f, r = 0.f, cosT = 1.f;
                double plen = 0.0;
                f3 hp = o, n = d;
                const int tri = warp_closest(onward, local, L, p, HSR_NODES, HSR_TRIS, o, d, cosT);
                // what the list did not settle goes to the BVH in a stage of its own
                const bool pending = local && onward && tri < 0;
                const bool alive =
                    pending || (tri >= 0 && arrive(HSR_TRIS, tri, cosT, o, d, time, r, plen, hp, n, cosT));
                const int slot = claim_slot(S, alive, pending || !(local && local_holds(L, hp)));
                if (alive)
                    store_path<kPhase>(S, gst, slot, pending ? o : hp, d, H, n, time, r, cosT, freq,
                                       pending ? kRayPending : 1, plen, g);
                else if (mine)
                    guide_train(pc, pc.train_child, s_g, 1, g.gw, g.pdf, g.x0, g.x1);
            } else {
                if (s < gen_end) {
                    const uint64_t hindex = uint64_t(pc.offset + s);
                    const float freq = rf.startFreq + halton(hindex, 0) * HSR_BANDWIDTH;
                    Guided g{halton(hindex, 1 + kGet2DFirst), halton(hindex, 1 + kGet2DSecond), 1.f, cf{0.f, 0.f}};
                    if (fl.doGuiding) g.pdf = guide_sample(pc.samp_child, pc.samp_p, g.x0, g.x1);
                    f3 o, d;
                    c3 H;
                    f3 ldir = mk3(0.f, 0.f, 0.f);  // kLazy: the local direction the field is formed from
                    const bool deferred = kLazy && fl.onlyIndirect;
                    if (kFF) {
                        ff_sample(S.ff[0], g.x0, g.x1, o, d, H);
                        H = c3_scl(H, 1.f / g.pdf);
                    } else if (kLazy) {
                        o = pc.tx.pos;
                        ldir = uniform_sample_sphere<kPhase == HSR_PHASE_REFERENCE_FP32>(g.x0, g.x1);
                        d = mulv(pc.tx.rot, ldir);
                        if (!deferred) H = c3_scl(antenna_field(pc.tx, ldir), 1.f / g.pdf);
                    } else {
                        o = pc.tx.pos;
                        antenna_sample<kPhase == HSR_PHASE_REFERENCE_FP32>(pc.tx, g.x0, g.x1, d, H);
                        H = c3_scl(H, 1.f / g.pdf);
                    }
                    if (!fl.onlyIndirect) {
                        NeeOut ne;
                        if (nee_eval<kPhase, false, kFF>(p, HSR_NODES, HSR_TRIS, rf, HSR_N, pc.tx, pc.rx, 0, o, d,
                                                         mk3(0.f, 0.f, 0.f), mk3(0.f, 0.f, 0.f), H, H, 0.f, 0.0, 0.f,
                                                         1.f, freq, pc.weight, ne, nullptr, nullptr, &S.ff[1]) &&
                            ne.splat) {
                            if (pc.fine_row) {
                                splat_fine(pc.fine_row, p.fine_bins, ne.sample, ne.value);
                            } else {
                                item = splat_item(ne.sample, ne.value);
                                has_item = true;
                            }
                        }
                    }
                    bool alive = false;
                    if (!(0 >= fl.maxDepth || 0.f >= HSR_MAXDIST) && (deferred || !c3_is_zero(H))) {
                        float time = 0.f, r = 0.f, cosT;
                        double plen = 0.0;
                        f3 hp, n;
                        if (walk(p, HSR_NODES, HSR_TRIS, o, d, time, r, plen, hp, n, cosT)) {
                            // deferred: the field now (the same operations as antenna_sample); a
                            // zero field ends the path as the reference's test before tracing would
                            if (deferred) H = c3_scl(antenna_field(pc.tx, ldir), 1.f / g.pdf);
                            if (!deferred || !c3_is_zero(H)) {
                                push_path<kPhase>(S, gst, hp, d, H, n, time, r, cosT, freq, 1, plen, g);
                                alive = true;
                            }
                        }
                    }
                    if (!alive) guide_train(pc, pc.train_child, s_g, 1, g.gw, g.pdf, g.x0, g.x1);
                }
            }
            if (!fl.onlyIndirect) splat_warp(s_re, s_im, HSR_N, has_item, item);
            __syncthreads();
            continue;
        }

        if (count + count_far > 0) {
            // ---------------- EXTEND ----------------
            // kLocal: the fuller end of the stack; the lower one asks the pose's list
            const bool local = kLocal && count > count_far;
            const bool upper = kLocal && !local;
            const int n = min(upper ? count_far : count, kThreads);
            const bool mine = tid < n;
            f3 o, din, nrm;
            c3 Hin;
            float time = 0.f, r = 0.f, cosT = 1.f, freq = 0.f;
            int depth = 0;
            double plen = 0.0;
            Guided g{0.f, 0.f, 1.f, cf{0.f, 0.f}};
            // the popped paths, ordered by the octant of their reflected direction: thread t
            // continues stack entry count - 1 - S.order[t]
            const bool ordered = !kLocal && p.coherent_order;
            if (ordered) {
                int key = kPrimaryCells;
                if (mine) {
                    const int e = count - 1 - tid;
                    const f3 di = mk3(S.dx[e], S.dy[e], S.dz[e]), nn = mk3(S.nx[e], S.ny[e], S.nz[e]);
                    const float dn = 2.f * dot3(di, nn);
                    key = (di.x - dn * nn.x < 0.f ? 1 : 0) | (di.y - dn * nn.y < 0.f ? 2 : 0) |
                          (di.z - dn * nn.z < 0.f ? 4 : 0);
                }
                order_by_key(S, key);
            }
            if (mine) {
                const int slot = upper ? kCap - count_far + tid : count - 1 - (ordered ? S.order[tid] : tid);
                if (gst)
                    g = Guided{gst[slot], gst[kCap + slot], gst[2 * kCap + slot],
                               cf{gst[3 * kCap + slot], gst[4 * kCap + slot]}};
                o = mk3(S.ox[slot], S.oy[slot], S.oz[slot]);
                din = mk3(S.dx[slot], S.dy[slot], S.dz[slot]);
#pragma unroll
                for (int i = 0; i < 3; ++i) Hin.v[i] = cf{S.h[2 * i][slot], S.h[2 * i + 1][slot]};
                nrm = mk3(S.nx[slot], S.ny[slot], S.nz[slot]);
                if (kPhase == HSR_PHASE_REFERENCE_FP32)
                    time = reinterpret_cast<const float *>(S.tlen)[slot];
                else
                    plen = S.tlen[slot];
                r = S.r[slot];
                cosT = S.cosT[slot];
                freq = S.freq[slot];
                depth = S.depth[slot];
            }
            __syncthreads();  // all pops read before the stack shrinks
            if (tid == 0) {
                if (upper)
                    S.count_far = count_far - n;
                else
                    S.count = count - n;
            }
            __syncthreads();
            bool has_item = false;
            float4 item = make_float4(0.f, 0.f, 0.f, 0.f);
            if constexpr (kLocal) {
                f3 d = din;
                c3 H = Hin;
                NeeState ne{};
                bool estimate = false, onward = false;
                if (mine) {
                    const bool resumed = depth & kRayPending;  // its estimate is done
                    depth &= kRayPending - 1;
                    onward = resumed;
                    if (!resumed) {
                        reflect(nrm, d, H);
                        estimate = nee_begin<false, false>(p, pc.tx, pc.rx, depth, o, d, din, nrm, Hin, H, time, plen, r,
                                                         cosT, freq, pc.weight, nullptr, ne);
                        onward = !(depth >= fl.maxDepth || r >= HSR_MAXDIST) && !c3_is_zero(H);
                    }
                }
                const bool hidden = warp_occluded(estimate && ne.ask, local, L, p, HSR_NODES, HSR_TRIS, o, ne.nd,
                                                          ne.dist);
                if (estimate && !hidden) {
                    NeeOut out;
                    nee_end<kPhase>(rf, HSR_N, ne, pc.weight, out);
                    g.gw = cadd(g.gw, out.gw_add);
                    if (out.splat) {
                        if (pc.fine_row) {
                            splat_fine(pc.fine_row, p.fine_bins, out.sample, out.value);
                        } else {
                            item = splat_item(out.sample, out.value);
                            has_item = true;
                        }
                    }
                }
                f3 hp = o, n2 = d;
                float cosT2 = 1.f;
                const int tri = warp_closest(onward, local, L, p, HSR_NODES, HSR_TRIS, o, d, cosT2);
                const bool unsettled = local && onward && tri < 0;
                const bool alive =
                    unsettled || (tri >= 0 && arrive(HSR_TRIS, tri, cosT2, o, d, time, r, plen, hp, n2, cosT2));
                const int to = claim_slot(S, alive, unsettled || !(L.planes > 0 && local_holds(L, hp)));
                if (alive)
                    store_path<kPhase>(S, gst, to, unsettled ? o : hp, d, H, n2, time, r, cosT2, freq,
                                       unsettled ? depth | kRayPending : depth + 1, plen, g);
                else if (mine)
                    guide_train(pc, pc.train_child, s_g, 1, g.gw, g.pdf, g.x0, g.x1);
            } else {
                if (mine) {
                    f3 d = din;
                    c3 H = Hin;
                    reflect(nrm, d, H);
                    NeeOut ne;
                    if (nee_eval<kPhase, false, kFF>(p, HSR_NODES, HSR_TRIS, rf, HSR_N, pc.tx, pc.rx, depth, o, d, din,
                                                     nrm, Hin, H, time, plen, r, cosT, freq, pc.weight, ne, nullptr,
                                                     nullptr, &S.ff[1])) {
                        g.gw = cadd(g.gw, ne.gw_add);
                        if (ne.splat) {
                            if (pc.fine_row) {
                                splat_fine(pc.fine_row, p.fine_bins, ne.sample, ne.value);
                            } else {
                                item = splat_item(ne.sample, ne.value);
                                has_item = true;
                            }
                        }
                    }
                    bool alive = false;
                    if (!(depth >= fl.maxDepth || r >= HSR_MAXDIST) && !c3_is_zero(H)) {
                        f3 hp, n2;
                        float cosT2;
                        if (walk(p, HSR_NODES, HSR_TRIS, o, d, time, r, plen, hp, n2, cosT2)) {
                            push_path<kPhase>(S, gst, hp, d, H, n2, time, r, cosT2, freq, depth + 1, plen, g);
                            alive = true;
                        }
                    }
                    if (!alive) guide_train(pc, pc.train_child, s_g, 1, g.gw, g.pdf, g.x0, g.x1);
                }
            }
            splat_warp(s_re, s_im, HSR_N, has_item, item);
            __syncthreads();
            continue;
        }

        if (pending >= 0) {
            // stack drained: finish the old pose's row and switch to the new pose
            if (cur_pose >= 0) {
                flush_row(pose_row<kMixed>(p, S, cur_pose), s_re, s_im, HSR_N);
                if (p.do_guide) flush_guide(pc, s_g);
            }
            cur_pose = pending;
            pc = load_pose(p, cur_pose);
            __syncthreads();  // every thread is done with the old pose's job and list
            if (kLocal) {
                const int4 *src = reinterpret_cast<const int4 *>(p.local + pending);
                int4 *dst = reinterpret_cast<int4 *>(&L);
                for (int k = tid; k < int(sizeof(LocalList) / sizeof(int4)); k += kThreads) dst[k] = __ldg(src + k);
            }
            if (tid == 0) {
                if (kMixed) {
                    S.job = p.jobs[pending];
                    S.max_dist = max_distance(S.job.rf);
                    S.bandwidth = chirp_bandwidth(S.job.rf);
                }
                if (kFF) {
                    S.ff[0] = load_ff(p.ff_tx + pending);
                    S.ff[1] = load_ff(p.ff_rx + pending);
                }
                S.pose = pending;
                S.since_flush = 0;
                S.gen = S.pending_first;
                S.gen_end = S.pending_last;
                S.pending_pose = -1;
            }
            __syncthreads();
            continue;
        }
        if (exhausted) break;
    }
    if (cur_pose >= 0) {
        __syncthreads();
        flush_row(pose_row<kMixed>(p, S, cur_pose), s_re, s_im, HSR_N);
        if (p.do_guide) flush_guide(pc, s_g);
    }
#undef HSR_NODES
#undef HSR_TRIS
#undef HSR_N
#undef HSR_MAXDIST
#undef HSR_BANDWIDTH
}

// The stack capacity (as its GENERATE threshold) a launch with threshold q runs: 64 for
// 1..64, 128 for 65..128, 256 above; 0 takes wave_default_queue.
inline int wave_capacity(int32_t q, int32_t samples, bool guided) {
    if (q == 0) q = wave_default_queue(samples, guided);
    return q <= kWaveSmallQueue ? kWaveSmallQueue : q > kWaveDefaultQueue ? kWaveMaxQueueThreshold : kWaveDefaultQueue;
}

// The launch of one instantiation.
template <int kPhase, bool kMixed, int kQueue, bool kFF = false, bool kLazy = false, bool kLocal = false>
void wave_instance(const TraceParams &p, int grid, cudaStream_t st) {
    const size_t smem = wave_smem_for<kQueue>(p.samples, p.do_guide != 0, kLocal);
    auto *kernel = k_wave<kPhase, kMixed, kQueue, kFF, kLazy, kLocal>;
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    kernel<<<grid, kThreads, smem, st>>>(p);
}

// The uniform form at one capacity, with the primary field formed eagerly or on a hit.
template <int kPhase, int kQueue> void wave_uniform(const TraceParams &p, int grid, cudaStream_t st) {
    if (p.field_on_hit)
        wave_instance<kPhase, false, kQueue, false, true>(p, grid, st);
    else
        wave_instance<kPhase, false, kQueue>(p, grid, st);
}

// Every instantiation of one phase mode: the mixed form (serving ticks) and the uniform
// form, each at both stack capacities. The mixed form takes the small stack unless the
// tick asks for a threshold above 64 (its default: on the serving mix of dense boxes
// and urban scenes it gives 1.18x the capacity of the 384-entry stack).
template <int kPhase> void wave_dispatch(const TraceParams &p, int grid, cudaStream_t st) {
    const int cap = wave_capacity(p.queue_threshold, p.samples, p.do_guide != 0);
    if (p.ff_tx) {  // far-field runs: the uniform form at one capacity
        wave_instance<kPhase, false, kWaveDefaultQueue, true>(p, grid, st);
    } else if (p.local) {
        if (p.jobs)
            wave_instance<kPhase, true, kWaveLocalQueue, false, false, true>(p, grid, st);
        else
            wave_instance<kPhase, false, kWaveLocalQueue, false, false, true>(p, grid, st);
    } else if (p.jobs) {  // the mixed form is built at the two smaller capacities
        if (p.queue_threshold > kWaveSmallQueue)
            wave_instance<kPhase, true, kWaveDefaultQueue>(p, grid, st);
        else
            wave_instance<kPhase, true, kWaveSmallQueue>(p, grid, st);
    } else if (cap == kWaveSmallQueue) {
        wave_uniform<kPhase, kWaveSmallQueue>(p, grid, st);
    } else if (cap == kWaveMaxQueueThreshold) {
        wave_uniform<kPhase, kWaveMaxQueueThreshold>(p, grid, st);
    } else {
        wave_uniform<kPhase, kWaveDefaultQueue>(p, grid, st);
    }
}

}  // namespace

}  // namespace hsr
