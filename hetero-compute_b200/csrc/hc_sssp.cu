// Single-source shortest paths: one persistent launch for all sources of a call,
// teams of blocks running several of them at a time.
//
// Reference path: sssp_pull_gpu (src/kernels/gpu/sssp.cuh:42-100) sweeps every
// vertex each epoch with an in-place Bellman-Ford pull over float weights and
// round-trips a counter to the host per epoch.  Here the epoch loop stays on
// the device and each epoch picks its direction:
//   push  relax only the edges out of vertices whose distance dropped (int32
//         atomicMin), split near/far by a moving threshold (Davidson et al.,
//         "Work-efficient parallel GPU methods for single-source shortest
//         paths", IPDPS 2014);
//   pull  when the frontier's edges exceed M / pull_alpha, sweep every row
//         with the reference's own Bellman-Ford pull (min over neighbours of
//         dist[u] + w) over each row's (neighbour, weight) pairs in weight
//         order, stopping a row once no later pair can lower it, without
//         per-edge atomics, then turn the vertices it lowered back into the
//         near queue / far pile.
// Distances are exact integers; unreachable = INT32_MAX.
//
// Thin epochs (a few thousand edges) run on the team's first block alone, phase
// changes included, with the near queue in shared memory.
//
// Working set of a team (N vertices): dist int32[N]; near queues q[2] int32[N];
// far piles far[2] int32[N]; stamp / fstamp int32[N] (queue dedup without
// clearing: a vertex joins the epoch-E queue by raising stamp[v] to E);
// changed bitmap uint32[N/32] (pull sweeps); tasks int2[] for long rows.
// Per graph: the pull sweeps' pair array int2[M + 64] (weight_order_rows).
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstddef>
#include <cstdio>
#include <cstring>
#include <cstdlib>
#include <vector>

#include "hc_expand.cuh"
#include "hc_graph.cuh"

namespace hc {
namespace {

constexpr int kSsspThreads = 512;
constexpr int kTraceEpochs = 96;
constexpr int kDefaultPullAlpha = 10;
// After a pull epoch, far piles of at most this many entries end the near/far
// phases (one last phase takes every remaining vertex).
#ifndef HC_SSSP_TAIL_PILE
#define HC_SSSP_TAIL_PILE 16384
#endif
constexpr int kTailPile = HC_SSSP_TAIL_PILE;

// Thin epochs: at most kSoloCap queued vertices with at most kSoloEdges edges,
// none of more than kSoloDeg, and phase changes over at most kSoloFar far-pile
// entries, up to kSoloEpochs at a time.  One block keeps 2048 edges in flight;
// above one round of those the whole team is faster (grid graph 701 x 517: limit
// 1024 7.4 ms, 2048 6.9 ms, 4096 7.2 ms, 8192 8.3 ms, no thin epochs 10.9 ms).
constexpr int kSoloCap = 1920;
constexpr int kSoloEdges = 2048;
constexpr int kSoloDeg = 128;
constexpr int kSoloFar = 8192;
constexpr int kSoloEpochs = 1024;
// Sources of one launch.
constexpr int kSsspLaunchSources = 256;
// Bytes that the workspaces of sources run at the same time may take in all.
constexpr size_t kSsspTeamBytes = 2ull << 30;

struct EpochCnt {
    int nq;                 // vertices in this near queue
    int tasks;              // long-row tasks queued while expanding it
    unsigned long long mf;  // sum of their degrees
    int32_t low;            // at most the smallest distance in it
};

// Loop state of a run that one block hands to the others after thin epochs.
struct SoloState {
    int E, phase, fgen, nq;
    int32_t T, low;
    unsigned long long mf, vproc, erelax;
};

struct SsspCtl {
    GridSync gs;
    // By run parity: a run's counters are set while blocks may still read the
    // last run's.
    EpochCnt cnt[2][3];
    // Lengths of the two far piles, in two pairs of which one is current: a
    // turn of thin epochs reads that pair and writes the other (see far_len in
    // sssp_persistent).
    int far_len[2][2][2];
    int min_far[2];
    // Degree sum of the rows a pull sweep lowered below the near threshold
    // (three slots, by pull): the next epoch's push-or-pull test, without
    // building its queue.
    unsigned long long pull_mf[3];
    int32_t pull_low[3];  // the smallest distance it wrote
    SoloState solo;
    int epochs, phases, pulls, pad;
    unsigned long long vproc, erelax;
    struct {
        int nq, phase;
        unsigned long long t_ns;
    } trace[kTraceEpochs + 1];  // per-epoch record for HC_TRACE=1 (phase < 0: pull sweep)
};

// Results of the runs of one call: the first failure, the most epochs.
struct SsspFold {
    int err, err_src, epochs;
    int teams_done;  // of the running launch
    int range_src;   // a source whose distances come too close to INT32_MAX (-1: none)
};

struct SsspArgs {
    const int64_t *index;
    const int32_t *nbr;
    const int32_t *w;
    int32_t n, n_active;
    int64_t m;
    // Outputs: dist + i * dist_stride for source i (stride 0: not wanted, one
    // scratch row per team).
    int32_t *dist;
    int64_t dist_stride;
    // Team 0's workspace; team t's lies t * team_stride bytes further on.
    int32_t *q0, *q1, *far0, *far1, *stamp, *fstamp;
    uint32_t *changed;
    int2 *tasks;
    SsspCtl *ctl;
    SsspFold *fold, *fold_host;  // fold_host: mapped host copy, written by the launch's last team (null: none)
    int team;                    // blocks per team
    size_t team_stride;
    PrPlanDev plan;
    const int2 *adj;  // pull sweeps: (neighbour, weight) pairs of each row in weight-bucket order
    int ws;           // bucket shift: bucket(w) = w >> ws < 256
    int32_t delta;  // <= 0: no far pile (plain frontier Bellman-Ford)
    int pull_alpha;  // <= 0: push only
    int max_epochs;
    int nsrc;
    int32_t src[kSsspLaunchSources];
};

// What one run works on (in shared memory: as registers these pointers would
// spill the epochs' inner loops).
struct SsspRun {
    int32_t src;
    int32_t *dist, *q0, *q1, *far0, *far1, *stamp, *fstamp;
    uint32_t *changed;
    int2 *tasks;
};

// dist + w for a distance and a weight in [0, INT32_MAX], clamped at
// INT32_MAX (unreachable): the sum never wraps, and a candidate that reaches
// the clamp lowers nothing.  Callers check afterwards that no distance came
// within the largest weight of the clamp.
__device__ __forceinline__ int32_t sat_add(int32_t d, int32_t w) {
    const uint32_t s = (uint32_t)d + (uint32_t)w;
    return s < (uint32_t)kInfDist ? (int32_t)s : kInfDist;
}

// Push relaxation visitor: nd = dist[u] + w; lower dist[v] with atomicMin and
// queue v once per epoch (near) or once per phase (far), by raising a stamp.
struct RelaxVisit {
    const int64_t *index;
    const int32_t *nbr, *w;
    int32_t *dist, *stamp, *fstamp;
    int32_t *qnext;
    int *qlen;
    int32_t *fpile;
    int *fpile_len;
    int32_t T;
    int next_e, far_claim;
    bool use_far;
    unsigned long long relaxed;
    unsigned long long mf;  // degree sum of this thread's near appends
    int32_t low;            // smallest near candidate below its target's distance (this thread)
    struct Item {
        int32_t v, nd, dv;
    };
    __device__ __forceinline__ void load(Item &it, int32_t u, int64_t e) {
        it.v = __ldg(nbr + e);
        it.nd = sat_add(__ldcg(dist + u), __ldg(w + e));
    }
    __device__ __forceinline__ void probe(Item &it) { it.dv = __ldcg(dist + it.v); }
    // All atomics of the round in flight together, then one append per queue
    // for the whole warp.  A vertex is claimed whenever the probed distance was
    // above the candidate: then it fell in this epoch, by this edge or by one
    // that overtook it, and whoever wins the claim queues it once.
    __device__ __forceinline__ void commit(Item (&it)[kUnroll], const bool (&act)[kUnroll]) {
        bool imp[kUnroll], near[kUnroll], far[kUnroll];
        int32_t old[kUnroll], v[kUnroll];
#pragma unroll
        for (int j = 0; j < kUnroll; j++) {
            relaxed += act[j];
            imp[j] = act[j] && it[j].nd < it[j].dv;
            if (imp[j]) {
                atomicMin(dist + it[j].v, it[j].nd);
                low = min(low, it[j].nd);
            }
            old[j] = imp[j] ? (it[j].nd < T ? atomicMax(stamp + it[j].v, next_e) : atomicMax(fstamp + it[j].v, far_claim))
                            : 0;
        }
#pragma unroll
        for (int j = 0; j < kUnroll; j++) {
            const bool is_near = it[j].nd < T;
            near[j] = imp[j] && is_near && old[j] < next_e;
            far[j] = imp[j] && !is_near && old[j] < far_claim;
            v[j] = imp[j] ? it[j].v : 0;
        }
#pragma unroll
        for (int j = 0; j < kUnroll; j++)
            if (near[j]) mf += (unsigned long long)(__ldg(index + v[j] + 1) - __ldg(index + v[j]));
        warp_append_n(near, v, qnext, qlen);
        if (use_far) warp_append_n(far, v, fpile, fpile_len);
    }
};

// Weight buckets of the pull sweeps' pair array: bucket(w) = w >> ws, ws the
// shift that brings the largest weight below 256, non-decreasing along each
// row.  Every pair at or after one of bucket b has weight >= b << ws.
__device__ __forceinline__ int wbucket(int32_t w, int ws) { return w >> ws; }
__device__ __forceinline__ int32_t wbucket_floor(int bk, int ws) { return bk << ws; }

// dist[u] + w for a pair whose weight is below `gap`, else INT32_MAX without
// touching dist.  The gap of a row is the best distance it has so far, less
// `low`: a distance that has not been relaxed along its edges yet is at least
// `low` (the smallest one in the queue, and candidates only add to it), and the
// smaller ones were relaxed when they were set, so a pair with w >= gap cannot
// lower the row.
// The gather goes through L1 (.ca): most edges point at a few thousand hub
// rows, whose distances then stay on the SM.  A value cached earlier in the
// same sweep can be stale, but distances only fall, so it is an upper bound,
// and the row that lowered it is marked changed and relaxed again next epoch;
// kernel boundaries and the grid barrier's fence invalidate L1 between epochs.
__device__ __forceinline__ int32_t pull_cand(const int32_t *dist, int2 p, int32_t gap) {
    return p.y < gap ? sat_add(__ldca(dist + p.x), p.y) : kInfDist;
}

// The warp walks the pairs [b, e) of one row, 128 at a time, with a running
// bound (the row's distance d0, then the best candidate): pairs at or above its
// gap to `low` gather nothing, and the walk stops at the first window whose
// leading bucket floor reaches it.  The leading weight of the next window is read one window
// ahead, so that the stop test comes before the window's loads; `test_first`
// tests the first window too (a range that starts among the row's heavier
// pairs).  Returns the bound; *next receives the slot it stopped at.
__device__ __forceinline__ int32_t pull_walk(const SsspArgs &a, const int32_t *dist, int64_t b, int64_t e, int32_t d0,
                                             int32_t low, bool test_first, int64_t *next) {
    const int lane = threadIdx.x & 31;
    const int32_t *wcol = reinterpret_cast<const int32_t *>(a.adj) + 1;
    int32_t wnext = test_first ? __ldg(wcol + 2 * b) : 0;
    int32_t bound = d0;
    int64_t i0 = b;
    for (; i0 < e; i0 += 128) {
        // Pair i0 carries the smallest bucket of the rest of the range.
        if ((i0 > b || test_first) && wbucket_floor(wbucket(wnext, a.ws), a.ws) >= bound - low) break;
        int2 q[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int64_t i = i0 + 32 * j + lane;
            q[j] = i < e ? __ldg(a.adj + i) : make_int2(0, kInfDist);
        }
        if (i0 + 128 < e) wnext = __ldg(wcol + 2 * (i0 + 128));
        int32_t m = kInfDist;
#pragma unroll
        for (int j = 0; j < 4; j++) m = min(m, pull_cand(dist, q[j], bound - low));
        bound = min(bound, __reduce_min_sync(kFull, m));
    }
    *next = min(i0, e);
    return bound;
}

// One Bellman-Ford pull over every row with edges (the reference's epoch,
// src/kernels/gpu/sssp.cuh:120-281), on the shared row plan, over the rows'
// pairs in weight-bucket order.  Hub chunks and long rows are walked by a warp
// each and lower dist by atomicMin.  In a stream group (32 rows, one warp, the
// only writer of its rows and of their word of the bitmap) a lane walks its own
// row, four pairs at a time, and stops where the bucket floor reaches its
// gap: on weights uniform in [1, 255] that is a small part of the row, so the
// sweep reads and searches that much less than a warp that streams the whole
// group.  Rows longer than kLaneRow would hold their warp up and are walked by
// the whole of it.  Lowered vertices are marked in `changed`.
constexpr int kLaneRow = 128;
template <bool kStats>
__device__ __forceinline__ void pull_sweep(const SsspArgs &a, int32_t *dist, uint32_t *changed, int gwarp, int nwarps,
                                           unsigned long long &my_e, int32_t T, int32_t low,
                                           unsigned long long &my_mf, int32_t &my_low) {
    const int lane = threadIdx.x & 31;
    const PrPlanDev &p = a.plan;
    const int total = p.n_tasks + p.n_long + p.n_stream;
    for (int item = gwarp; item < total; item += nwarps) {
        if (item < p.n_tasks + p.n_long) {
            int32_t r;
            int64_t b, e;
            bool test_first = false;
            if (item < p.n_tasks) {
                const int2 tk = p.tasks[item];
                r = p.hubs[tk.x].row;
                const int64_t rb = __ldg(a.index + r), re = __ldg(a.index + r + 1);
                b = rb + (int64_t)tk.y * p.chunk;
                e = min(re, b + (int64_t)p.chunk);
                test_first = tk.y > 0;
            } else {
                r = p.longrows[item - p.n_tasks];
                b = __ldg(a.index + r);
                e = __ldg(a.index + r + 1);
            }
            const int32_t d0 = __shfl_sync(kFull, __ldcg(dist + r), 0);
            int64_t next;
            if (d0 <= low) continue;  // final
            const int32_t bound = pull_walk(a, dist, b, e, d0, low, test_first, &next);
            if (lane == 0) {
                if (bound < d0 && bound < __ldcg(dist + r) && bound < atomicMin(dist + r, bound)) {
                    my_low = min(my_low, bound);
                    const uint32_t bit = 1u << (r & 31);
                    if (!(atomicOr(changed + (r >> 5), bit) & bit) && bound < T)
                        my_mf += (unsigned long long)(__ldg(a.index + r + 1) - __ldg(a.index + r));
                }
                if (kStats) my_e += (unsigned long long)(next - b);
            }
        } else {
            const int32_t r0 = p.stream[item - p.n_tasks - p.n_long] * 32;
            const int32_t r = r0 + lane;
            int64_t b = 0, e = 0;
            int32_t d0 = kInfDist;
            if (r < a.n_active) {
                b = __ldg(a.index + r);
                e = __ldg(a.index + r + 1);
                d0 = __ldcg(dist + r);
            }
            int32_t bound = d0;
            const bool whole = e - b > kLaneRow && d0 > low;
            int64_t i = whole || d0 <= low ? e : b;
            while (i < e) {
                int2 q[4];
#pragma unroll
                for (int j = 0; j < 4; j++) q[j] = i + j < e ? __ldg(a.adj + i + j) : make_int2(0, kInfDist);
                if (wbucket_floor(wbucket(q[0].y, a.ws), a.ws) >= bound - low) break;
                int32_t m[4];
#pragma unroll
                for (int j = 0; j < 4; j++) m[j] = pull_cand(dist, q[j], bound - low);
                bound = min(bound, min(min(m[0], m[1]), min(m[2], m[3])));
                i += 4;
            }
            if (kStats && !whole && d0 > low) my_e += (unsigned long long)(min(i, e) - b);
            for (unsigned left = __ballot_sync(kFull, whole); left; left &= left - 1u) {
                const int src = __ffs(left) - 1;
                const int64_t wb = __shfl_sync(kFull, b, src), we = __shfl_sync(kFull, e, src);
                int64_t next;
                const int32_t got = pull_walk(a, dist, wb, we, __shfl_sync(kFull, d0, src), low, false, &next);
                if (lane == src) bound = got;
                if (kStats && lane == 0) my_e += (unsigned long long)(next - wb);
            }
            const bool ch = bound < d0;
            if (ch) {
                dist[r] = bound;
                my_low = min(my_low, bound);
                if (bound < T) my_mf += (unsigned long long)(e - b);
            }
            const unsigned bal = __ballot_sync(kFull, ch);
            if (lane == 0 && bal) changed[r0 >> 5] = bal;
        }
    }
}

// Shared-memory queue of the thin epochs: vertex, and its row's first slot and
// degree packed (44 + 20 bits, the degree clamped).
struct SoloQueue {
    int32_t u[kSoloCap];
    unsigned long long row[kSoloCap];
};
constexpr unsigned long long kSoloDegMask = (1ull << 20) - 1ull;
__device__ __forceinline__ unsigned long long solo_row(int64_t b, int64_t d) {
    return ((unsigned long long)b << 20) | min((unsigned long long)d, kSoloDegMask);
}

struct SoloArgs {
    const int64_t *index;
    const int32_t *nbr, *w;
    int64_t m;
    int32_t delta;
    int pull_alpha, max_epochs;
    bool pulled;  // a pull sweep has run: a small pile is finished in one phase
};

// Thin epochs and phase changes from st on, by one block (every thread calls
// it): the same relaxations, claims and buckets as the grid's, with the near
// queue in shared memory and mirrored in the global queue, so that the grid can
// take any epoch over.  Stops before an epoch that is too wide or a pull, before
// a phase change over too long a pile, after kSoloEpochs, or at the end.  The far
// piles' lengths are read from far_len and left in far_next: the other blocks may
// still be reading far_len while this one runs.
// Not inlined: its registers would spill the grid's epochs.
template <bool kStats>
__device__ __noinline__ SoloState solo_epochs(SoloArgs a, const SsspRun &r, SsspCtl *ctl, const int *far_len,
                                              int *far_next, SoloQueue *sq, SoloState st) {
    __shared__ int s_n[3], s_wide[3], s_far[2], s_min;
    __shared__ unsigned s_mf[3];  // exact while no row is long (see the end)
    __shared__ unsigned long long s_sum;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    int32_t *const dist = r.dist;
    const bool use_far = a.delta > 0;
    __syncthreads();  // far_len as this block's thread 0 left it
    if (threadIdx.x < 3) {
        s_n[threadIdx.x] = 0;
        s_mf[threadIdx.x] = 0u;
        s_wide[threadIdx.x] = 0;
    }
    if (threadIdx.x < 2) s_far[threadIdx.x] = __ldcg(far_len + threadIdx.x);
    __syncthreads();
    // Adds vertex v to queue slot p of set k (shared, mirrored in `q`).
    auto put = [&](SoloQueue &nq, int32_t *q, int k, int p, int32_t v, int64_t b, int64_t d) {
        q[p] = v;
        if (p < kSoloCap) {
            nq.u[p] = v;
            nq.row[p] = solo_row(b, d);
        }
        if (d > kSoloDeg) s_wide[k] = 1;
    };
    {
        const int32_t *qin = (st.E & 1) ? r.q1 : r.q0;
        unsigned edges = 0;
        for (int i = threadIdx.x; i < st.nq; i += blockDim.x) {
            const int32_t u = __ldcg(qin + i);
            const int64_t b = __ldg(a.index + u), d = __ldg(a.index + u + 1) - b;
            sq[0].u[i] = u;
            sq[0].row[i] = solo_row(b, d);
            edges += (unsigned)min(d, (int64_t)kSoloEdges);
            if (d > kSoloDeg) s_wide[0] = 1;
        }
        edges = __reduce_add_sync(kFull, edges);
        if (lane == 0 && edges) atomicAdd(&s_mf[0], edges);
    }
    __syncthreads();
    int k = 0;  // queue set of the current epoch: counters k % 3, queue k & 1
    bool wide = s_wide[0] || s_mf[0] > (unsigned)kSoloEdges;
    for (int step = 0; step < kSoloEpochs; step++) {
        if (st.nq == 0) {
            const int fl = s_far[st.phase & 1];
            if (!use_far || fl == 0 || fl > kSoloFar) break;
            // Next phase: the smallest live distance of the pile picks the
            // bucket, [T_old, T) joins the queue, >= T stays far.
            const int32_t *fcur = (st.phase & 1) ? r.far1 : r.far0;
            int32_t *fnew = (st.phase & 1) ? r.far0 : r.far1;
            int32_t *q = (st.E & 1) ? r.q1 : r.q0;
            if (threadIdx.x == 0) s_min = kInfDist;
            __syncthreads();
            int mn = kInfDist;
            for (int i = threadIdx.x; i < fl; i += blockDim.x) {
                const int32_t d = __ldcg(dist + __ldcg(fcur + i));
                if (d >= st.T) mn = min(mn, d);
            }
            mn = __reduce_min_sync(kFull, mn);
            if (lane == 0 && mn < kInfDist) atomicMin(&s_min, mn);
            __syncthreads();
            const int32_t mfar = s_min;
            if (mfar == kInfDist) {  // only settled entries are left: the run is over
                __syncthreads();
                if (threadIdx.x == 0) s_far[st.phase & 1] = 0;
                break;
            }
            const int32_t T_old = st.T;
            const long long tn = a.pulled && fl <= kTailPile
                                     ? (long long)kInfDist
                                     : ((long long)mfar / a.delta + 1) * (long long)a.delta;
            st.T = (int32_t)(tn < (long long)kInfDist ? tn : (long long)kInfDist);
            const int cs = k % 3;  // empty queue: its counters are all zero but s_mf / s_wide of the last epoch
            if (threadIdx.x == 0) {
                s_n[cs] = 0;
                s_mf[cs] = 0u;
                s_wide[cs] = 0;
                s_far[(st.phase + 1) & 1] = 0;
            }
            __syncthreads();
            unsigned dsum = 0;
            for (int i0 = 0; i0 < fl; i0 += blockDim.x) {
                const int i = i0 + threadIdx.x;
                const int32_t v = i < fl ? __ldcg(fcur + i) : 0;
                const int32_t d = i < fl ? __ldcg(dist + v) : -1;
                const bool near = d >= T_old && d < st.T, far = d >= st.T;
                if (near && atomicMax(r.stamp + v, st.E) < st.E) {
                    const int64_t b = __ldg(a.index + v), dg = __ldg(a.index + v + 1) - b;
                    put(sq[k & 1], q, cs, atomicAdd(&s_n[cs], 1), v, b, dg);
                    dsum += (unsigned)min(dg, (int64_t)kSoloEdges);
                }
                if (far && atomicMax(r.fstamp + v, st.fgen + 1) < st.fgen + 1)
                    fnew[atomicAdd(&s_far[(st.phase + 1) & 1], 1)] = v;
            }
            dsum = __reduce_add_sync(kFull, dsum);
            if (lane == 0 && dsum) atomicAdd(&s_mf[cs], dsum);
            __syncthreads();
            if (threadIdx.x == 0) s_far[st.phase & 1] = 0;
            st.phase++;
            st.fgen++;
            st.nq = s_n[cs];
            st.mf = s_mf[cs];
            wide = s_wide[cs] || st.mf > (unsigned long long)kSoloEdges;
            __syncthreads();
            continue;
        }
        const int ns = (k + 1) % 3;
        if (st.nq > kSoloCap || wide || st.E >= a.max_epochs ||
            (a.pull_alpha > 0 && (double)st.mf * (double)a.pull_alpha > (double)a.m))
            break;
        const SoloQueue &cq = sq[k & 1];
        SoloQueue &nq = sq[(k + 1) & 1];
        int32_t *qnext = (st.E & 1) ? r.q0 : r.q1;
        int32_t *fpile = (st.phase & 1) ? r.far1 : r.far0;
        if (threadIdx.x == 0) {
            s_n[(k + 2) % 3] = 0;
            s_mf[(k + 2) % 3] = 0u;
            s_wide[(k + 2) % 3] = 0;
            if (st.E < kTraceEpochs) {
                ctl->trace[st.E].nq = st.nq;
                ctl->trace[st.E].phase = st.phase;
                ctl->trace[st.E].t_ns = globaltimer_ns();
            }
        }
        if (kStats) {
            st.vproc += st.nq;
            st.erelax += st.mf;
        }
        const int next_e = st.E + 1;
        const int per = min(32, max(1, (st.nq + nwarps - 1) / nwarps));
        for (int base = wib * per; base < st.nq; base += nwarps * per) {
            const int i = base + lane;
            const bool mine = lane < per && i < st.nq;
            const int32_t u = mine ? cq.u[i] : -1;
            const unsigned long long row = mine ? cq.row[i] : 0ull;
            const int32_t du = mine ? __ldcg(dist + u) : 0;
            const long long beg = (long long)(row >> 20);
            int total;
            const int excl = warp_exclusive_scan((int)(row & kSoloDegMask), &total);
            for (int k0 = 0; k0 < total; k0 += 32 * kUnroll) {
                int32_t v[kUnroll], nd[kUnroll], dv[kUnroll], old[kUnroll];
                bool near[kUnroll], far[kUnroll];
#pragma unroll
                for (int j = 0; j < kUnroll; j++) {
                    const int kk = k0 + 32 * j + lane;
                    int lo = 0;
#pragma unroll
                    for (int s = 16; s > 0; s >>= 1) {
                        const int c = __shfl_sync(kFull, excl, lo + s);
                        if (c <= kk) lo += s;
                    }
                    const long long e = __shfl_sync(kFull, beg, lo) + (kk - __shfl_sync(kFull, excl, lo));
                    const int32_t duo = __shfl_sync(kFull, du, lo);
                    v[j] = kk < total ? __ldg(a.nbr + e) : -1;
                    nd[j] = kk < total ? sat_add(duo, __ldg(a.w + e)) : kInfDist;
                }
#pragma unroll
                for (int j = 0; j < kUnroll; j++) dv[j] = v[j] >= 0 ? __ldcg(dist + v[j]) : 0;
#pragma unroll
                for (int j = 0; j < kUnroll; j++) {
                    const bool imp = v[j] >= 0 && nd[j] < dv[j];
                    near[j] = imp && nd[j] < st.T;
                    far[j] = imp && nd[j] >= st.T && use_far;
                    if (imp) atomicMin(dist + v[j], nd[j]);
                    old[j] = near[j] ? atomicMax(r.stamp + v[j], next_e)
                             : far[j] ? atomicMax(r.fstamp + v[j], st.fgen) : 0;
                }
                int count = 0;
                unsigned bal[kUnroll];
#pragma unroll
                for (int j = 0; j < kUnroll; j++) {
                    near[j] = near[j] && old[j] < next_e;
                    far[j] = far[j] && old[j] < st.fgen;
                    bal[j] = __ballot_sync(kFull, near[j]);
                    count += __popc(bal[j]);
                }
#pragma unroll
                for (int j = 0; j < kUnroll; j++)
                    if (far[j]) fpile[atomicAdd(&s_far[st.phase & 1], 1)] = v[j];
                if (count == 0) continue;
                int64_t nb[kUnroll], nx[kUnroll];
#pragma unroll
                for (int j = 0; j < kUnroll; j++) {
                    nb[j] = near[j] ? __ldg(a.index + v[j]) : 0;
                    nx[j] = near[j] ? __ldg(a.index + v[j] + 1) : 0;
                }
                int pos = 0;
                if (lane == 0) pos = atomicAdd(&s_n[ns], count);
                pos = __shfl_sync(kFull, pos, 0);
                unsigned dsum = 0;
#pragma unroll
                for (int j = 0; j < kUnroll; j++) {
                    if (near[j]) {
                        put(nq, qnext, ns, pos + __popc(bal[j] & lt), v[j], nb[j], nx[j] - nb[j]);
                        dsum += (unsigned)min(nx[j] - nb[j], (int64_t)kSoloEdges);
                    }
                    pos += __popc(bal[j]);
                }
                dsum = __reduce_add_sync(kFull, dsum);
                if (lane == 0) atomicAdd(&s_mf[ns], dsum);
            }
        }
        __syncthreads();
        st.nq = s_n[ns];
        st.mf = s_mf[ns];
        wide = s_wide[ns] || st.mf > (unsigned long long)kSoloEdges;
        st.E++;
        k++;
    }
    __syncthreads();
    if (st.nq > 0) {
        // The queue's degree sum (exact with long rows too) and its smallest
        // distance: a pull reads them.
        if (threadIdx.x == 0) {
            s_sum = 0ull;
            s_min = kInfDist;
        }
        __syncthreads();
        int32_t low = kInfDist;
        const int32_t *q = (st.E & 1) ? r.q1 : r.q0;
        unsigned long long sum = 0;
        for (int i = threadIdx.x; i < st.nq; i += blockDim.x) {
            const int32_t u = __ldcg(q + i);
            sum += (unsigned long long)(__ldg(a.index + u + 1) - __ldg(a.index + u));
            low = min(low, __ldcg(dist + u));
        }
        sum = warp_sum(sum);
        low = __reduce_min_sync(kFull, low);
        if (lane == 0) {
            if (sum) atomicAdd(&s_sum, sum);
            atomicMin(&s_min, low);
        }
        __syncthreads();
        st.mf = s_sum;
        st.low = s_min;
    }
    if (threadIdx.x < 2) far_next[threadIdx.x] = s_far[threadIdx.x];
    return st;
}

// Shared memory of one block.
union SsspShared {
    SoloQueue solo[2];                          // thin epochs
    uint32_t fold[kSsspThreads / 32][2][32];    // per warp: near / far masks of its 32 words
};

// Lowers *p to the smallest x of the warp (every lane calls it).
__device__ __forceinline__ void note_low(int32_t *p, int32_t x) {
    x = __reduce_min_sync(kFull, x);
    if ((threadIdx.x & 31) == 0 && x < kInfDist && x < __ldcg(p)) atomicMin(p, x);
}

// kBlocks resident blocks per SM: two, or three for many sources at a time on a
// large graph with hub rows, whose pulls wait on gathers (issue slots 32 % used,
// DRAM 20 %) and gain more from a third block's warps than its spills cost: from
// kSsspWideEdges edges and kSsspWideWork edges times sources on.  Two / three blocks
// in ms: Kronecker scale 22, 2 sources 1.26 / 1.26, 8 4.98 / 4.54, 16 10.5 / 9.0; scale
// 20, 4 0.90 / 0.93, 8 1.35 / 1.37, 16 2.73 / 2.66, 64 10.2 / 9.2; scale 19, 8 0.78 / 0.86,
// 16 1.58 / 1.49; scale 18 (7.6M edges), 16 0.90 / 0.87, 64 2.62 / 2.75; scale 16, 16
// 0.42 / 0.46; without hubs, where the pushes' atomics are the work, uniform 2^18, 16
// sources 2.66 / 3.28.
constexpr int64_t kSsspWideEdges = 1ll << 23;
constexpr int64_t kSsspWideWork = 3ll << 26;
template <bool kStats, int kBlocks>
__global__ void __launch_bounds__(kSsspThreads, kBlocks) sssp_persistent(SsspArgs a) {
    __shared__ unsigned long long s_red[32];
    __shared__ int s_min[32];
    __shared__ SsspShared sh;
    __shared__ SsspRun r;
    __shared__ int s_stop;
    const int team = blockIdx.x / a.team, team_block = blockIdx.x - team * a.team;
    const int nteams = gridDim.x / a.team;
    SsspCtl *ctl = a.ctl + team;
    const int gtid = team_block * blockDim.x + threadIdx.x;
    const int nthreads = a.team * blockDim.x;
    const int gwarp = gtid >> 5, nwarps = nthreads >> 5;
    const int lane = threadIdx.x & 31;
    const int W_act = (a.n_active + 31) >> 5;
    const bool use_far = a.delta > 0;

    // A team of one block needs no more than its own block barrier; the acquire
    // drops what its L1 holds of distances that its atomics have lowered since.
    bool stop = false;  // thread 0 of a one-block team: it recorded a failure
    auto team_sync = [&]() -> bool {
        if (a.team > 1) return grid_barrier(&ctl->gs, (unsigned)a.team);
        __syncthreads();
        if (threadIdx.x == 0) {
            if (a.pull_alpha > 0) (void)ld_acquire_u64(&ctl->gs.count);
            s_stop = stop;
        }
        __syncthreads();
        return !s_stop;
    };
    if (threadIdx.x == 0) {
        auto at = [&](auto *p) { return reinterpret_cast<decltype(p)>(reinterpret_cast<char *>(p) + (size_t)team * a.team_stride); };
        r.q0 = at(a.q0);
        r.q1 = at(a.q1);
        r.far0 = at(a.far0);
        r.far1 = at(a.far1);
        r.stamp = at(a.stamp);
        r.fstamp = at(a.fstamp);
        r.changed = at(a.changed);
        r.tasks = at(a.tasks);
    }
    unsigned long long my_v = 0, my_e = 0;
    bool failed = false;
    int run = 0;

    for (int si = team; si < a.nsrc && !failed; si += nteams, run++) {
        __syncthreads();  // the last run's reads of r
        if (threadIdx.x == 0) {
            r.src = a.src[si];
            r.dist = a.dist + (a.dist_stride ? (size_t)si * a.dist_stride : (size_t)team * a.n);
        }
        __syncthreads();
        const int par = run & 1;
        EpochCnt *const cnt = ctl->cnt[par];
        // The current pair of pile lengths.  At the top of an epoch with an empty
        // near queue every thread reads far_len, and the first block may enter the
        // thin epochs before the last thread has: nothing orders that read before
        // what the thin epochs store.  So they store the new lengths into the other
        // pair, which nobody reads before the team barrier after the turn, where
        // every block changes over, whether the turn did anything or not.  The next
        // turn, which writes this pair, comes after a whole-team epoch (solo_ok) and
        // so after a barrier that every reader of this pair has reached.
        int pair = 0;
        int *far_len = ctl->far_len[par][0];
        int *const min_far = &ctl->min_far[par];
        {
            int32_t *const dist = r.dist, *const stamp = r.stamp, *const fstamp = r.fstamp;
            const int32_t src = r.src;
            for (int i = gtid; i < a.n; i += nthreads) {
                dist[i] = i == src ? 0 : kInfDist;
                stamp[i] = i == src ? 0 : -1;
                fstamp[i] = -1;
            }
            uint32_t *const changed = r.changed;
            for (int i = gtid; i < W_act; i += nthreads) changed[i] = 0;
        }
        const unsigned long long t_start = globaltimer_ns();
        if (gtid == 0) {
            r.q0[0] = r.src;
            cnt[0] = EpochCnt{1, 0, (unsigned long long)(a.index[r.src + 1] - a.index[r.src]), 0};
            cnt[1] = EpochCnt{0, 0, 0ull, kInfDist};
            cnt[2] = EpochCnt{0, 0, 0ull, kInfDist};
            far_len[0] = far_len[1] = 0;
            *min_far = kInfDist;
            ctl->pull_mf[0] = ctl->pull_mf[1] = ctl->pull_mf[2] = 0ull;
            ctl->pull_low[0] = ctl->pull_low[1] = ctl->pull_low[2] = kInfDist;
        }
        failed = !team_sync();

        int32_t T = use_far ? a.delta : kInfDist;
        int E = 0, phase = 0, pulls = 0;
        int C = 0;  // rotation of cnt: advances with the epochs the whole team runs
        // Far-pile claim: a vertex is in the current pile when fstamp[v] == fgen.
        int fgen = 1;
        bool solo_ok = true;      // one block may take thin epochs (not twice in a row: see the BFS)
        bool from_solo = false;   // nq and mf of this epoch come from there
        while (!failed) {
            EpochCnt *const ccur = &cnt[C % 3], *const cnxt = &cnt[(C + 1) % 3];
            if (gtid == 0) {
                if (globaltimer_ns() - t_start > c_limits.run_ns) {
                    atomicExch(&ctl->gs.err, (int)HC_ERR_TIMEOUT);
                    stop = true;
                }
                EpochCnt *const cold = &cnt[(C + 2) % 3];
                cold->nq = 0;
                cold->tasks = 0;
                cold->mf = 0;
                cold->low = kInfDist;
            }
            int nq = from_solo ? __ldcg(&ctl->solo.nq) : __ldcg(&ccur->nq);
            unsigned long long mfc = from_solo ? __ldcg(&ctl->solo.mf) : __ldcg(&ccur->mf);
            int32_t low = from_solo ? __ldcg(&ctl->solo.low) : __ldcg(&ccur->low);
            from_solo = false;
            int fl = 0;
            if (nq == 0) {
                if (!use_far) break;
                fl = __ldcg(far_len + (phase & 1));
                if (fl == 0) break;
            }
            if (solo_ok && nq <= kSoloCap && (nq > 0 ? mfc <= (unsigned long long)kSoloEdges : fl <= kSoloFar) &&
                !(a.pull_alpha > 0 && (double)mfc * (double)a.pull_alpha > (double)a.m)) {
                solo_ok = false;
                if (team_block == 0) {
                    const SoloState st = solo_epochs<kStats>(
                        SoloArgs{a.index, a.nbr, a.w, a.m, a.delta, a.pull_alpha, a.max_epochs, pulls > 0}, r, ctl,
                        far_len, ctl->far_len[par][pair ^ 1], sh.solo, SoloState{E, phase, fgen, nq, T, low, mfc, 0ull, 0ull});
                    if (threadIdx.x == 0) {
                        ctl->solo = st;
                        if (kStats) {
                            my_v += st.vproc;
                            my_e += st.erelax;
                        }
                    }
                }
                if ((failed = !team_sync())) break;
                pair ^= 1;
                far_len = ctl->far_len[par][pair];
                const int E1 = __ldcg(&ctl->solo.E), phase1 = __ldcg(&ctl->solo.phase);
                const bool moved = E1 != E || phase1 != phase || (nq == 0 && __ldcg(far_len + (phase & 1)) == 0);
                if (moved) {
                    E = E1;
                    phase = phase1;
                    fgen = __ldcg(&ctl->solo.fgen);
                    T = __ldcg(&ctl->solo.T);
                    from_solo = true;
                    C++;  // this epoch's counters were the ones before the thin epochs
                    continue;
                }
            }
            int32_t *qcur = (E & 1) ? r.q1 : r.q0;
            int32_t *qnext = (E & 1) ? r.q0 : r.q1;
            if (nq == 0) {
                const int32_t *fcur = (phase & 1) ? r.far1 : r.far0;
                int32_t *fnew = (phase & 1) ? r.far0 : r.far1;
                // Smallest live distance in the far pile picks the next bucket.
                int mn = kInfDist;
                for (int i = gtid; i < fl; i += nthreads) {
                    const int32_t d = __ldcg(r.dist + __ldcg(fcur + i));
                    if (d >= T) mn = min(mn, d);
                }
                mn = warp_min(mn);
                if (lane == 0) s_min[threadIdx.x >> 5] = mn;
                __syncthreads();
                if (threadIdx.x < 32) {
                    int x = threadIdx.x < (blockDim.x >> 5) ? s_min[threadIdx.x] : kInfDist;
                    x = warp_min(x);
                    if (threadIdx.x == 0 && x < kInfDist) atomicMin(min_far, x);
                }
                if ((failed = !team_sync())) break;
                const int32_t mfar = __ldcg(min_far);
                if (mfar == kInfDist) break;
                const int32_t T_old = T;
                // After a pull sweep (the dense part of a small-diameter graph is
                // done) a small pile is finished in one last near phase: a phase
                // costs a few grid barriers however few vertices it holds, and
                // relaxing those few out of distance order costs little.  On a
                // high-diameter graph (no pulls) the pile is the thin wavefront
                // and keeps its distance order.
                const long long tn = pulls > 0 && fl <= kTailPile
                                         ? (long long)kInfDist
                                         : ((long long)mfar / a.delta + 1) * (long long)a.delta;
                T = (int32_t)(tn < (long long)kInfDist ? tn : (long long)kInfDist);
                // Split: [T_old, T) joins the epoch-E queue, >= T stays far.  A
                // warp takes 1024 consecutive pile entries: pass 1 classifies them
                // 32 at a time and keeps the ballots in shared memory, pass 2
                // writes them at offsets taken with one atomicAdd per warp.
                unsigned long long mf_split = 0;
                const int wib = threadIdx.x >> 5;
                const uint32_t below = (1u << lane) - 1u;
                // Rounds of 32 entries per warp chunk: enough for every warp to
                // get one chunk, at most 32 (the shared ballot slots).
                const int per = min(32, max(1, (fl + 32 * nwarps - 1) / (32 * nwarps)));
                for (int c0 = gwarp * 32 * per; c0 < fl; c0 += nwarps * 32 * per) {
                    const int rounds = min(per, (fl - c0 + 31) / 32);
                    int n_near = 0, n_far = 0;
                    for (int j0 = 0; j0 < rounds; j0 += 4) {
                        int32_t v[4], d[4];
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const int i = c0 + 32 * (j0 + k) + lane;
                            v[k] = (j0 + k < rounds && i < fl) ? __ldcg(fcur + i) : -1;
                        }
#pragma unroll
                        for (int k = 0; k < 4; k++) d[k] = v[k] >= 0 ? __ldcg(r.dist + v[k]) : 0;
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            bool to_near = false, to_far = false;
                            if (v[k] >= 0) {
                                if (d[k] >= T_old && d[k] < T) to_near = atomicMax(r.stamp + v[k], E) < E;
                                else if (d[k] >= T) to_far = atomicMax(r.fstamp + v[k], fgen + 1) < fgen + 1;
                                if (to_near) mf_split += (unsigned long long)(a.index[v[k] + 1] - a.index[v[k]]);
                            }
                            const uint32_t nm = __ballot_sync(kFull, to_near), fm = __ballot_sync(kFull, to_far);
                            if (lane == 0 && j0 + k < rounds) {
                                sh.fold[wib][0][j0 + k] = nm;
                                sh.fold[wib][1][j0 + k] = fm;
                            }
                            n_near += __popc(nm);
                            n_far += __popc(fm);
                        }
                    }
                    int nbase = 0, fbase = 0;
                    if (lane == 0) {
                        if (n_near) nbase = atomicAdd(&ccur->nq, n_near);
                        if (n_far) fbase = atomicAdd(&far_len[(phase + 1) & 1], n_far);
                    }
                    nbase = __shfl_sync(kFull, nbase, 0);
                    fbase = __shfl_sync(kFull, fbase, 0);
                    __syncwarp();
                    for (int j = 0; j < rounds; j++) {
                        const uint32_t nm = sh.fold[wib][0][j], fm = sh.fold[wib][1][j];
                        if ((nm | fm) >> lane & 1u) {
                            const int32_t v = __ldcg(fcur + c0 + 32 * j + lane);
                            if ((nm >> lane) & 1u) qcur[nbase + __popc(nm & below)] = v;
                            else fnew[fbase + __popc(fm & below)] = v;
                        }
                        nbase += __popc(nm);
                        fbase += __popc(fm);
                    }
                    __syncwarp();
                }
                mf_split = block_sum(mf_split, s_red);
                if (threadIdx.x == 0 && mf_split) atomicAdd(&ccur->mf, mf_split);
                if ((failed = !team_sync())) break;
                if (gtid == 0) {
                    far_len[phase & 1] = 0;
                    *min_far = kInfDist;
                }
                phase++;
                fgen++;
                nq = __ldcg(&ccur->nq);
                mfc = __ldcg(&ccur->mf);
                low = mfar;
                if (nq == 0) continue;
            }
            if (E >= a.max_epochs) {
                if (gtid == 0) {
                    atomicExch(&ctl->gs.err, (int)HC_ERR_NOT_CONVERGED);
                    stop = true;
                }
                break;
            }
            // After the far split above: `phase` may have advanced.
            int32_t *fpile = (phase & 1) ? r.far1 : r.far0;
            int *fpile_len = far_len + (phase & 1);
            const int next_e = E + 1;
            bool pull = a.pull_alpha > 0 && (double)mfc * (double)a.pull_alpha > (double)a.m;
            if (gtid == 0 && E < kTraceEpochs) {
                ctl->trace[E].nq = nq;
                ctl->trace[E].phase = pull ? -1 - phase : phase;
                ctl->trace[E].t_ns = globaltimer_ns();
            }
            if (kStats && gtid == 0) my_v += nq;
            if (!pull) {
                RelaxVisit relax{a.index, a.nbr, a.w, r.dist, r.stamp, r.fstamp, qnext, &cnxt->nq, fpile,
                                 fpile_len, T, next_e, fgen, use_far, 0ull, 0ull, kInfDist};
                expand_small(a.index, qcur, nq, r.tasks, &ccur->tasks, gwarp, nwarps, relax);
                unsigned long long mfb = block_sum(relax.mf, s_red);
                if (threadIdx.x == 0 && mfb) atomicAdd(&cnxt->mf, mfb);
                relax.mf = 0;
                note_low(&cnxt->low, relax.low);
                if ((failed = !team_sync())) break;
                const int nt = __ldcg(&ccur->tasks);
                if (nt > 0) {
                    expand_tasks(a.index, r.tasks, nt, gwarp, nwarps, relax);
                    mfb = block_sum(relax.mf, s_red);
                    if (threadIdx.x == 0 && mfb) atomicAdd(&cnxt->mf, mfb);
                    note_low(&cnxt->low, relax.low);
                    if ((failed = !team_sync())) break;
                }
                if (kStats) my_e += relax.relaxed;
                E++;
                C++;
                solo_ok = true;
                continue;
            }
            // Pull sweeps, until the rows that one lowered no longer call for
            // another: a sweep propagates every distance it starts from, so
            // those rows need no queue, and the far pile's entries need no
            // later relaxation either (a value that falls during the sweep
            // marks its row changed): drop the pile.
            for (;;) {
                if (gtid == 0) {
                    *fpile_len = 0;
                    ctl->pull_mf[(pulls + 1) % 3] = 0ull;  // last read two sweeps ago
                    ctl->pull_low[(pulls + 1) % 3] = kInfDist;
                }
                unsigned long long my_mf = 0;
                int32_t my_low = kInfDist;
                pull_sweep<kStats>(a, r.dist, r.changed, gwarp, nwarps, my_e, T, low, my_mf, my_low);
                note_low(&ctl->pull_low[pulls % 3], my_low);
                const unsigned long long mfb = block_sum(my_mf, s_red);
                if (threadIdx.x == 0 && mfb) atomicAdd(&ctl->pull_mf[pulls % 3], mfb);
                if ((failed = !team_sync())) break;
                const unsigned long long pull_mf = __ldcg(&ctl->pull_mf[pulls % 3]);
                low = __ldcg(&ctl->pull_low[pulls % 3]);
                pulls++;
                fgen++;  // the rows it lowered rejoin the pile under a new claim
                if (!((double)pull_mf * (double)a.pull_alpha > (double)a.m) || E + 1 >= a.max_epochs) break;
                for (int w = gtid; w < W_act; w += nthreads) r.changed[w] = 0;
                E++;
                if (gtid == 0) {
                    if (globaltimer_ns() - t_start > c_limits.run_ns) {
                        atomicExch(&ctl->gs.err, (int)HC_ERR_TIMEOUT);
                        stop = true;
                    }
                    if (E < kTraceEpochs) {
                        ctl->trace[E].nq = 0;
                        ctl->trace[E].phase = -1 - phase;
                        ctl->trace[E].t_ns = globaltimer_ns();
                    }
                }
                if ((failed = !team_sync())) break;  // the bitmap is clear
            }
            if (failed) break;
            qnext = (E & 1) ? r.q0 : r.q1;
            // Lowered vertices back into the near queue / far pile.  A warp
            // takes up to 32 words of the changed bitmap; pass 1 classifies their
            // vertices a word at a time (lane l takes vertex 32j + l of word j:
            // coalesced reads; each vertex is in one bit, so its stamps need
            // no atomics) and keeps the ballots in shared memory; pass 2
            // writes the queue and pile entries at offsets taken with one
            // atomicAdd per warp.
            {
                const int next_f = E + 1;
                int32_t *const dist = r.dist, *const stamp = r.stamp, *const fstamp = r.fstamp;
                unsigned long long mf_next = 0;
                const int wib = threadIdx.x >> 5;
                const uint32_t below = (1u << lane) - 1u;
                // Up to 32 words per warp, fewer when there are not 32 for each.
                const int per = min(32, max(1, (W_act + nwarps - 1) / nwarps));
                for (int w0 = gwarp * per; w0 < W_act; w0 += nwarps * per) {
                    const int w = w0 + lane;
                    uint32_t bits = 0;
                    if (lane < per && w < W_act) {
                        bits = __ldcg(r.changed + w);
                        if (bits) r.changed[w] = 0;
                    }
                    const unsigned words = __ballot_sync(kFull, bits != 0u);
                    int n_near = 0, n_far = 0;
                    // Four words per round, their loads issued together.
                    for (unsigned left = words; left;) {
                        int j[4];
                        bool mine[4];
                        int32_t d[4], sp[4];
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            j[k] = left ? __ffs(left) - 1 : -1;
                            if (left) left &= left - 1u;
                            const uint32_t word = __shfl_sync(kFull, bits, j[k] < 0 ? 0 : j[k]);
                            mine[k] = j[k] >= 0 && ((word >> lane) & 1u);
                            d[k] = mine[k] ? __ldcg(dist + (w0 + j[k]) * 32 + lane) : 0;
                        }
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const int32_t v = (w0 + j[k]) * 32 + lane;
                            sp[k] = !mine[k] ? 0 : d[k] < T ? __ldcg(stamp + v) : __ldcg(fstamp + v);
                        }
#pragma unroll
                        for (int k = 0; k < 4; k++) {
                            const int32_t v = (w0 + j[k]) * 32 + lane;
                            bool near = false, far = false;
                            if (mine[k]) {
                                if (d[k] < T) {
                                    near = sp[k] < next_f;
                                    if (near) stamp[v] = next_f;
                                } else {
                                    far = sp[k] < fgen;
                                    if (far) fstamp[v] = fgen;
                                }
                                if (near) mf_next += (unsigned long long)(a.index[v + 1] - a.index[v]);
                            }
                            const uint32_t nm = __ballot_sync(kFull, near), fm = __ballot_sync(kFull, far);
                            if (lane == 0 && j[k] >= 0) {
                                sh.fold[wib][0][j[k]] = nm;
                                sh.fold[wib][1][j[k]] = fm;
                            }
                            n_near += __popc(nm);
                            n_far += __popc(fm);
                        }
                    }
                    if (!use_far) n_far = 0;
                    int nbase = 0, fbase = 0;
                    if (lane == 0) {
                        if (n_near) nbase = atomicAdd(&cnxt->nq, n_near);
                        if (n_far) fbase = atomicAdd(fpile_len, n_far);
                    }
                    nbase = __shfl_sync(kFull, nbase, 0);
                    fbase = __shfl_sync(kFull, fbase, 0);
                    __syncwarp();
                    for (unsigned left = words; left;) {
                        const int j = __ffs(left) - 1;
                        left &= left - 1u;
                        const uint32_t nm = sh.fold[wib][0][j], fm = use_far ? sh.fold[wib][1][j] : 0u;
                        const int32_t v = (w0 + j) * 32 + lane;
                        if ((nm >> lane) & 1u) qnext[nbase + __popc(nm & below)] = v;
                        if ((fm >> lane) & 1u) fpile[fbase + __popc(fm & below)] = v;
                        nbase += __popc(nm);
                        fbase += __popc(fm);
                    }
                    __syncwarp();
                }
                mf_next = block_sum(mf_next, s_red);
                if (threadIdx.x == 0 && mf_next) atomicAdd(&cnxt->mf, mf_next);
                if (gtid == 0) atomicMin(&cnxt->low, low);  // every queued row is one that the sweep lowered
            }
            if ((failed = !team_sync())) break;
            E++;
            C++;
            solo_ok = true;
        }
        if (gtid == 0) {
            ctl->epochs = E;
            ctl->phases = phase;
            ctl->pulls = pulls;
            ctl->trace[E < kTraceEpochs ? E : kTraceEpochs].t_ns = globaltimer_ns();
            const int err = *(volatile int *)&ctl->gs.err;
            if (err && atomicCAS(&a.fold->err, 0, err) == 0) a.fold->err_src = r.src;
            atomicMax(&a.fold->epochs, E);
        }
    }  // next source

    if (kStats) {
        unsigned long long v = block_sum(my_v, s_red);
        if (threadIdx.x == 0 && v) atomicAdd(&ctl->vproc, v);
        unsigned long long e = block_sum(my_e, s_red);
        if (threadIdx.x == 0 && e) atomicAdd(&ctl->erelax, e);
    }
    if (gtid == 0) {
        __threadfence();
        if (atomicAdd(&a.fold->teams_done, 1) == nteams - 1) {
            __threadfence();
            a.fold->teams_done = 0;
            if (a.fold_host) {
                a.fold_host->err = __ldcg(&a.fold->err);
                a.fold_host->err_src = __ldcg(&a.fold->err_src);
                a.fold_host->epochs = __ldcg(&a.fold->epochs);
                __threadfence_system();
            }
        }
    }
}

// Shortest-path tree: any u with dist[u] + w(u->v) == dist[v] is a valid
// parent (weights are non-negative integers).  Warp per source row, push
// direction, so directed weights are read from the row that owns them.
__global__ void sssp_parent_init(int32_t *parent, int32_t n, int32_t src) {
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        parent[v] = v == src ? src : -1;
}

__global__ void sssp_parents_fill(const int64_t *index, const int32_t *nbr, const int32_t *w, const int32_t *dist,
                                  int32_t n, int32_t src, int32_t *parent) {
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n; u += nw) {
        const int32_t du = dist[u];
        if (du == kInfDist) continue;
        const int64_t b = index[u], e = index[u + 1];
        for (int64_t i = b + lane; i < e; i += 32) {
            const int32_t v = nbr[i];
            if (v != src && sat_add(du, w[i]) == dist[v]) parent[v] = u;
        }
    }
}

__global__ void count_finite(const int32_t *dist, int32_t n, unsigned long long *out) {
    __shared__ unsigned long long s_red[32];
    unsigned long long c = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        c += dist[i] != kInfDist;
    c = block_sum(c, s_red);
    if (threadIdx.x == 0 && c) atomicAdd(out, c);
}

// Candidates are clamped at INT32_MAX (sat_add).  When every finite
// distance plus the largest weight stays below the clamp, no candidate
// reached it, so the clamp changed nothing; otherwise some distance may lie
// beyond int32 and the run is refused.  Puts src in *flag when a finite
// distance exceeds `limit` (INT32_MAX - 1 - largest weight).
__global__ void any_above(const int32_t *dist, int32_t n, int32_t limit, int32_t src, int *flag) {
    bool hi = false;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int32_t d = dist[i];
        hi |= d != kInfDist && d > limit;
    }
    if (__any_sync(kFull, hi) && (threadIdx.x & 31) == 0) *flag = src;
}

// Whether any weight is negative (flags[0]), the largest weight (flags[1])
// and the weights' sum.
__global__ void weight_stats(const int64_t *index, const int32_t *w, int32_t n, int *flags, unsigned long long *sum) {
    __shared__ unsigned long long s_red[32];
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    unsigned long long s = 0;
    int32_t mx = 0;
    for (int v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += nw) {
        const int64_t b = index[v], e = index[v + 1];
        for (int64_t i = b + lane; i < e; i += 32) {
            const int32_t x = w[i];
            if (x < 0) flags[0] = 1;
            s += (unsigned long long)max(x, 0);
            mx = max(mx, x);
        }
    }
    mx = __reduce_max_sync(kFull, mx);
    if (lane == 0 && mx > 0) atomicMax(flags + 1, mx);
    s = block_sum(s, s_red);
    if (threadIdx.x == 0 && s) atomicAdd(sum, s);
}

// The pull sweeps' pair array: each row's (neighbour, weight) pairs ordered
// by weight bucket, stable within a bucket (CSR order), so the result is the
// same on every run.  One warp per row: a bucket histogram in shared memory,
// its exclusive scan, then a stable scatter 32 pairs at a time (lanes of one
// bucket take consecutive slots in lane order).
constexpr int kOrderThreads = 256;
__global__ void __launch_bounds__(kOrderThreads) weight_order_rows(const int64_t *index, const int32_t *nbr,
                                                                   const int32_t *w, int32_t n, int ws,
                                                                   int2 *adj) {
    __shared__ int s_cnt[kOrderThreads / 32][256];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    int *cnt = s_cnt[wib];
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += nw) {
        const int64_t b = index[v], e = index[v + 1];
        if (e - b <= 1) {
            if (e > b && lane == 0) adj[b] = make_int2(nbr[b], w[b]);
            continue;
        }
#pragma unroll
        for (int k = 0; k < 8; k++) cnt[lane * 8 + k] = 0;
        __syncwarp();
        for (int64_t i = b + lane; i < e; i += 32) atomicAdd(&cnt[wbucket(w[i], ws)], 1);
        __syncwarp();
        int loc[8], tot = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            loc[k] = tot;
            tot += cnt[lane * 8 + k];
        }
        int incl = tot;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += y;
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 8; k++) cnt[lane * 8 + k] = incl - tot + loc[k];
        __syncwarp();
        for (int64_t i0 = b; i0 < e; i0 += 32) {
            const int64_t i = i0 + lane;
            const bool act = i < e;
            int2 q = make_int2(0, 0);
            int bk = -1;
            if (act) {
                q = make_int2(nbr[i], w[i]);
                bk = wbucket(q.y, ws);
            }
            const unsigned peers = __match_any_sync(kFull, bk);
            if (act) adj[b + cnt[bk] + __popc(peers & ((1u << lane) - 1u))] = q;
            __syncwarp();
            if (act && (peers >> lane) == 1u) cnt[bk] += __popc(peers);  // the bucket's highest lane
            __syncwarp();
        }
        __syncwarp();
    }
}

// Clears the fold record and what the teams' control blocks must start from.
__global__ void sssp_clear(SsspCtl *ctl, int teams, SsspFold *f) {
    if (threadIdx.x == 0) *f = SsspFold{0, 0, 0, 0, -1};
    for (int t = threadIdx.x; t < teams; t += blockDim.x) {
        ctl[t].gs = GridSync{0ull, 0, 0};
        ctl[t].vproc = ctl[t].erelax = 0ull;
    }
}

// Blocks of sssp_persistent that are resident at a time (fewer when the handle's tuning says so).
template <bool kStats, int kBlocks>
hc_status sssp_resident(hc_graph *g, int *blocks) {
    static int blocks_per_sm = 0;
    if (blocks_per_sm == 0) {
        HC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, sssp_persistent<kStats, kBlocks>,
                                                                  kSsspThreads, 0));
        if (blocks_per_sm < 1) return fail(HC_ERR_CUDA, "SSSP kernel cannot be resident");
    }
    const int use = g->tune.sssp_blocks_per_sm > 0 ? std::min(blocks_per_sm, g->tune.sssp_blocks_per_sm)
                                                   : blocks_per_sm;
    *blocks = use * g->sm_count;
    return HC_OK;
}

template <bool kStats, int kBlocks>
hc_status launch_sssp(hc_graph *g, SsspArgs &a, int teams) {
    dim3 grid(a.team * teams), block(kSsspThreads);
    ::hc::count_launch();
    if (a.team == 1) {  // no block waits for another
        sssp_persistent<kStats, kBlocks><<<grid, block, 0, g->stream>>>(a);
        HC_CUDA_TRY(cudaGetLastError());
        return HC_OK;
    }
    void *params[] = {&a};
    HC_CUDA_TRY(cudaLaunchCooperativeKernel((void *)sssp_persistent<kStats, kBlocks>, grid, block, params, 0, g->stream));
    return HC_OK;
}

// Blocks per team and teams for k sources on a graph of m edges (at most `room`
// teams), from sweeps of team sizes on Kronecker and uniform graphs of 20k to
// 128M edges.  No smaller than sqrt(m) / 300 blocks, where more sources at a time
// outgrow the L2 (16 sources, 128M edges: 8 teams 13.3 ms, 12 teams 18.4 ms, 1
// team 17.4 ms; 16 sources, 16M edges: 16 teams 1.5 ms, 1 team 5.5 ms), and no
// larger than sqrt(m) / 9, where a barrier costs more than the blocks bring
// (one source, 0.1M edges: 37 blocks 153 us, 16 blocks 166 us, 296 blocks 190
// us; 8M edges without hubs: 296 blocks 578 us, 148 blocks 595 us).
void sssp_teams(const hc_graph *g, int resident, int k, int room, int *team, int *teams) {
    const double root = std::sqrt((double)std::max<int64_t>(g->M, 1));
    const int least = std::max(1, std::min(resident, (int)std::lround(root / 300.0)));
    const int most = std::max(1, std::min(resident, (int)std::lround(root / 9.0)));
    const int at_a_time = std::max(1, std::min({k, room, resident / least, kSsspLaunchSources}));
    const int rounds = (std::max(k, 1) + at_a_time - 1) / at_a_time;
    *teams = (std::max(k, 1) + rounds - 1) / rounds;
    *team = std::max(least, std::min(most, resident / *teams));
}

}  // namespace

// The bucket shift for weights in [0, w_max]: the smallest ws with w_max >> ws < 256.
int weight_shift(int32_t w_max) {
    int ws = 0;
    while ((w_max >> ws) > 255) ws++;
    return ws;
}

// Builds the pull sweeps' weight-ordered pair array once per graph (after the
// weight statistics, which give the bucket shift).
hc_status ensure_weight_order(hc_graph *g) {
    if (g->sssp_adj_ready) return HC_OK;
    HC_TRY(g->sssp_adj.ensure(sizeof(int2) * ((size_t)g->M + 64)));
    {
        weight_order_rows<<<g->sm_count * 8, kOrderThreads, 0, g->stream>>>(
            g->index.as<int64_t>(), g->nbr.as<int32_t>(), g->wgt.as<int32_t>(), g->N, weight_shift(g->w_max),
            g->sssp_adj.as<int2>());
        ::hc::count_launch();
    }
    HC_CUDA_TRY(cudaGetLastError());
    g->sssp_adj_ready = 1;
    return HC_OK;
}

hc_status ensure_weight_stats(hc_graph *g) {
    if (g->wstats_done) return HC_OK;
    DevBuf buf;
    HC_TRY(buf.ensure(64));
    HC_CUDA_TRY(cudaMemsetAsync(buf.ptr, 0, 64, g->stream));
    int *flags = buf.as<int>();
    unsigned long long *sum = reinterpret_cast<unsigned long long *>(buf.as<char>() + 16);
    {
        weight_stats<<<g->sm_count * 8, 256, 0, g->stream>>>(g->index.as<int64_t>(), g->wgt.as<int32_t>(), g->N,
                                                             flags, sum);
        ::hc::count_launch();
    }
    HC_CUDA_TRY(cudaGetLastError());
    int hf[2] = {0, 0};
    unsigned long long hsum = 0;
    HC_CUDA_TRY(cudaMemcpyAsync(hf, flags, 8, cudaMemcpyDeviceToHost, g->stream));
    HC_CUDA_TRY(cudaMemcpyAsync(&hsum, sum, 8, cudaMemcpyDeviceToHost, g->stream));
    HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
    g->w_negative = hf[0];
    g->w_max = hf[1];
    // Symmetric weights (w(u->v) == w(v->u) for every edge): one hashing pass.
    bool st = false, ws = false;
    HC_TRY(edge_symmetry(g, reinterpret_cast<const uint32_t *>(g->wgt.ptr), &st, &ws));
    g->w_symmetric = ws;
    g->w_mean = g->M ? (double)hsum / (double)g->M : 1.0;
    g->wstats_done = 1;
    return HC_OK;
}

}  // namespace hc

using namespace hc;

extern "C" hc_status hc_sssp(hc_graph *g, const int32_t *sources, int32_t num_sources, int32_t *dist_out,
                             int32_t *parent_out, const hc_sssp_opts *opts, hc_sssp_stats *stats) {
    clear_error();
    HC_TRY(activate(g));
    ReclaimScope reclaim_scope(g, kKeepAdj);
    if (!sources || num_sources < 0) return fail(HC_ERR_INVALID_ARG, "hc_sssp: bad source list");
    if (g->wtype != HC_W_I32) return fail(HC_ERR_UNSUPPORTED, "hc_sssp: graph needs int32 edge weights");
    hc_sssp_opts o{};
    if (opts) o = *opts;
    if (stats) std::memset(stats, 0, sizeof(*stats));
    std::vector<int32_t> src(num_sources);
    if (is_device_pointer(sources))
        HC_CUDA_TRY(cudaMemcpy(src.data(), sources, sizeof(int32_t) * num_sources, cudaMemcpyDefault));
    else
        std::copy(sources, sources + num_sources, src.begin());
    for (int32_t s : src)
        if (s < 0 || s >= g->N) return fail(HC_ERR_INVALID_ARG, "hc_sssp: source %d outside [0, %d)", s, g->N);
    HC_TRY(after_default_stream(g));

    // Weights must be non-negative; the mean weight sets the default delta.
    HC_TRY(ensure_weight_stats(g));
    if (g->w_negative) return fail(HC_ERR_INVALID_ARG, "hc_sssp: negative edge weight");
    HC_TRY(ensure_plans(g, kPlanBase));
    // Zero fields: the handle's tuned values, else the defaults.
    // The pull sweep reads w(u->v) from v's row: only valid when weights are symmetric.
    if (o.pull_alpha == 0) o.pull_alpha = g->tune.sssp_pull_alpha;
    if (o.delta == 0) o.delta = g->tune.sssp_delta;
    const int pull_alpha =
        !g->w_symmetric ? 0 : (o.pull_alpha == 0 ? kDefaultPullAlpha : std::max(o.pull_alpha, 0));
    // Before the workspaces, which can do with one source's where the pair array
    // cannot be had smaller.
    if (pull_alpha > 0) HC_TRY(ensure_weight_order(g));

    const int64_t n = g->N;
    const int64_t W = (n + 31) / 32;
    const int64_t ntasks = max_expand_tasks(g->M, n);
    auto up = [](size_t b) { return (b + 255) / 256 * 256; };
    const size_t bytes = 6 * up(4 * (size_t)n) + up(4 * (size_t)W) + up(sizeof(int2) * (size_t)ntasks);
    const bool per_run = (o.collect_stats && stats) || std::getenv("HC_TRACE");
    const bool dev_dist = is_device_pointer(dist_out);
    const bool dev_parent = is_device_pointer(parent_out);
    // Host outputs: staged on the device and copied while the next sources run.
    const bool host_dist = dist_out && !dev_dist, host_parent = parent_out && !dev_parent;
    const bool staged = host_dist || host_parent;
    // Parents and the range check read the distances after a launch: without
    // an output for them, one scratch row per source of a launch is kept.
    int resident = 0;
    const bool wide = !per_run && num_sources >= 2 && g->M >= kSsspWideEdges &&
                      g->M * num_sources >= kSsspWideWork && g->base_view.n_tasks > 0;
    HC_TRY((o.collect_stats ? sssp_resident<true, 2>(g, &resident)
            : wide          ? sssp_resident<false, 3>(g, &resident)
                            : sssp_resident<false, 2>(g, &resident)));
    OutPipe pipe;
    int team = resident, teams = 1;
    const size_t fold_bytes = 256;
    auto reserve = [&]() -> hc_status {
        HC_TRY(g->ws_sssp.ensure(bytes * teams));
        HC_TRY(g->ws_ctl.ensure(std::max<size_t>(4096, fold_bytes + sizeof(SsspCtl) * (size_t)teams)));
        if (!dist_out) HC_TRY(g->ws_out0.ensure(4 * n * (size_t)teams));
        if (staged) HC_TRY(pipe.init(g, 2, 4 * n, teams));
        return HC_OK;
    };
    if (!per_run) {
        const size_t each = bytes + 4 * (size_t)n * ((staged ? 4 : 0) + !dist_out);
        sssp_teams(g, resident, num_sources,
                   (int)std::min<size_t>(std::max<size_t>(kSsspTeamBytes / each, 1), 1 << 20), &team, &teams);
    }
    hc_status reserved;
    {
        ReclaimScope nothing(nullptr, 0u);
        reserved = reserve();
    }
    if (reserved == HC_ERR_OOM) {  // no room: one source at a time, and what other calls left behind goes
        clear_error();
        if (teams > 1) {
            sssp_teams(g, resident, num_sources, 1, &team, &teams);
            g->ws_sssp.release();
            if (!dist_out) g->ws_out0.release();
            OutPipe::drop_staging(g);
        }
        ReclaimScope own_scope(g, kKeepAdj | kKeepSssp);
        reserved = reserve();
    }
    HC_TRY(reserved);
    char *p = g->ws_sssp.as<char>();
    auto take = [&](size_t b) {
        char *r = p;
        p += up(b);
        return r;
    };
    SsspArgs a{};
    a.index = g->index.as<int64_t>();
    a.nbr = g->nbr.as<int32_t>();
    a.w = g->wgt.as<int32_t>();
    a.n = g->N;
    a.n_active = g->n_active;
    a.m = g->M;
    a.q0 = (int32_t *)take(4 * n);
    a.q1 = (int32_t *)take(4 * n);
    a.far0 = (int32_t *)take(4 * n);
    a.far1 = (int32_t *)take(4 * n);
    a.stamp = (int32_t *)take(4 * n);
    a.fstamp = (int32_t *)take(4 * n);
    a.changed = (uint32_t *)take(4 * W);
    a.tasks = (int2 *)take(sizeof(int2) * ntasks);
    SsspFold *fold = g->ws_ctl.as<SsspFold>();
    a.ctl = reinterpret_cast<SsspCtl *>(g->ws_ctl.as<char>() + fold_bytes);
    a.fold = fold;
    a.team = team;
    a.team_stride = bytes;
    a.plan = g->base_view;
    a.max_epochs = o.max_epochs > 0 ? o.max_epochs : 0x7fffffff;
    a.pull_alpha = pull_alpha;
    if (a.pull_alpha > 0) {
        a.adj = g->sssp_adj.as<int2>();
        a.ws = weight_shift(g->w_max);
    }
    if (o.delta == 0) {
        const double davg = g->n_active ? (double)g->M / (double)g->n_active : 1.0;
        a.delta = (int32_t)std::max(1.0, std::min(1e9, g->w_mean * 32.0 / std::max(davg, 1.0)));
    } else {
        a.delta = o.delta;
    }

    // Candidates can reach the INT32_MAX clamp only when a path of
    // n_active - 1 edges of the largest weight can; then each source's
    // distances are checked after its run (a source over the limit leaves
    // its id in the fold record).
    static_assert(sizeof(SsspCtl) + 256 <= 3072 && sizeof(SsspCtl) <= kCtlSlotBytes, "SsspCtl overlaps its spare slots");
    const bool check_range = (int64_t)g->w_max * std::max<int64_t>(g->n_active - 1, 0) >= (int64_t)kInfDist;
    const int32_t range_limit = kInfDist - 1 - g->w_max;
    double total_ms = 0;
    // Without per-run statistics or a trace the sources of a call run in one
    // launch (a launch per team's worth with staged outputs or scratch
    // distances), and the host waits once, at the end.
    const bool rows_kept = dev_dist || host_dist;
    const int per_launch = per_run ? 1 : staged || !rows_kept ? teams : kSsspLaunchSources;
    a.dist_stride = rows_kept ? n : 0;
    SsspFold *h_fold = nullptr;
    if (!per_run) {
        HC_TRY(ctl_slot(g, 0, (void **)&h_fold, (void **)&a.fold_host));
        { sssp_clear<<<1, 256, 0, g->stream>>>(a.ctl, teams, fold); ::hc::count_launch(); }
        HC_CUDA_TRY(cudaGetLastError());
        HC_CUDA_TRY(cudaEventRecord(g->ev_start, g->stream));
    }
    const void *h_range = nullptr;
    for (int32_t i = 0, l = 0; i < num_sources; i += per_launch, l++) {
        a.nsrc = std::min(per_launch, num_sources - i);
        std::copy(src.begin() + i, src.begin() + i + a.nsrc, a.src);
        int32_t *stage[2] = {nullptr, nullptr};
        if (staged) HC_TRY(pipe.acquire(l, stage));
        a.dist = dev_dist ? dist_out + (size_t)i * n : host_dist ? stage[0] : g->ws_out0.as<int32_t>();
        if (per_run) {
            { sssp_clear<<<1, 256, 0, g->stream>>>(a.ctl, 1, fold); ::hc::count_launch(); }
            HC_CUDA_TRY(cudaEventRecord(g->ev_start, g->stream));
        }
        const int use = std::min(teams, a.nsrc);
        HC_TRY((o.collect_stats ? launch_sssp<true, 2>(g, a, use)
                : wide          ? launch_sssp<false, 3>(g, a, use)
                                : launch_sssp<false, 2>(g, a, use)));
        if (per_run) HC_CUDA_TRY(cudaEventRecord(g->ev_stop, g->stream));
        for (int32_t j = 0; j < a.nsrc; j++) {
            const int32_t *row = a.dist + (size_t)j * n;
            if (parent_out) {
                int32_t *par = dev_parent ? parent_out + (size_t)(i + j) * n : stage[1] + (size_t)j * n;
                { sssp_parent_init<<<g->sm_count * 4, 256, 0, g->stream>>>(par, g->N, a.src[j]); ::hc::count_launch(); }
                { sssp_parents_fill<<<g->sm_count * 8, 256, 0, g->stream>>>(a.index, a.nbr, a.w, row, g->N, a.src[j], par); ::hc::count_launch(); }
            }
            if (check_range) {
                { any_above<<<g->sm_count * 4, 256, 0, g->stream>>>(row, g->N, range_limit, a.src[j], &fold->range_src); ::hc::count_launch(); }
            }
        }
        HC_CUDA_TRY(cudaGetLastError());
        if (staged) {
            void *dst[2] = {host_dist ? (void *)(dist_out + (size_t)i * n) : nullptr,
                            host_parent ? (void *)(parent_out + (size_t)i * n) : nullptr};
            HC_TRY(pipe.release(l, dst, a.nsrc));
        }
        if (!per_run) continue;

        SsspCtl c;
        const void *h_ctl = nullptr, *h_cnt = nullptr;
        if (check_range) HC_TRY(ctl_read(g, &fold->range_src, sizeof(int), 1, &h_range));
        HC_TRY(ctl_read(g, a.ctl, sizeof(c), 0, &h_ctl));
        if (o.collect_stats && stats) {
            unsigned long long *cnt = (unsigned long long *)(g->ws_ctl.as<char>() + 3072);
            HC_TRY(ctl_zero(g, cnt, 8));
            { count_finite<<<g->sm_count * 4, 256, 0, g->stream>>>(a.dist, g->N, cnt); ::hc::count_launch(); }
            HC_TRY(ctl_read(g, cnt, 8, 2, &h_cnt));
        }
        HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
        std::memcpy(&c, h_ctl, sizeof(c));
        int range_src = -1;
        if (h_range) std::memcpy(&range_src, h_range, sizeof(int));
        if (h_cnt) {
            unsigned long long reached = 0;
            std::memcpy(&reached, h_cnt, 8);
            stats->reached += (int32_t)reached;
        }
        if (c.gs.err) return fail((hc_status)c.gs.err, "hc_sssp: device run from source %d ended with status %d",
                                  src[i], c.gs.err);
        if (range_src >= 0)
            return fail(HC_ERR_UNSUPPORTED, "hc_sssp: a distance from source %d comes within the largest weight "
                        "(%d) of INT32_MAX: int32 distances cannot hold it", src[i], g->w_max);
        float ms = 0;
        HC_CUDA_TRY(cudaEventElapsedTime(&ms, g->ev_start, g->ev_stop));
        total_ms += ms;
        if (stats) {
            stats->epochs = std::max(stats->epochs, c.epochs);
            stats->vertices_processed += (int64_t)c.vproc;
            stats->edges_relaxed += (int64_t)c.erelax;
        }
        if (std::getenv("HC_TRACE")) {
            const int ne = std::min(c.epochs, kTraceEpochs);
            std::fprintf(stderr, "[hc sssp] src %d: %d epochs (%d pull), %d phases, delta %d, %.1f us\n", src[i],
                         c.epochs, c.pulls, c.phases, a.delta, ms * 1e3);
            for (int e = 0; e < ne; e++) {
                const int ph = c.trace[e].phase;
                std::fprintf(stderr, "[hc sssp]   E%-4d %s phase %-4d nq=%-9d %8.1f us\n", e, ph < 0 ? "pull" : "push",
                             ph < 0 ? -1 - ph : ph, c.trace[e].nq, (c.trace[e + 1].t_ns - c.trace[e].t_ns) * 1e-3);
            }
        }
    }
    if (!per_run) {
        HC_CUDA_TRY(cudaEventRecord(g->ev_stop, g->stream));
        if (check_range && num_sources > 0) HC_TRY(ctl_read(g, &fold->range_src, sizeof(int), 1, &h_range));
        HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
        if (num_sources > 0) {
            SsspFold f;
            std::memcpy(&f, h_fold, sizeof(f));
            if (f.err) return fail((hc_status)f.err, "hc_sssp: device run from source %d ended with status %d",
                                   f.err_src, f.err);
            int range_src = -1;
            if (h_range) std::memcpy(&range_src, h_range, sizeof(int));
            if (range_src >= 0)
                return fail(HC_ERR_UNSUPPORTED, "hc_sssp: a distance from source %d comes within the largest weight "
                            "(%d) of INT32_MAX: int32 distances cannot hold it", range_src, g->w_max);
            if (stats) stats->epochs = f.epochs;
        }
        float ms = 0;
        HC_CUDA_TRY(cudaEventElapsedTime(&ms, g->ev_start, g->ev_stop));
        total_ms = ms;
    }
    if (host_dist || host_parent) HC_TRY(pipe.finish());
    if (stats) {
        stats->ms = total_ms;
        // 16 B offsets per processed vertex, 8 B (neighbour + weight) per
        // relaxed edge, 4 B distance write per reached vertex.
        stats->bytes_model = 16.0 * (double)stats->vertices_processed + 8.0 * (double)stats->edges_relaxed +
                             4.0 * (double)stats->reached;
    }
    return HC_OK;
}
