// Direction-optimising BFS: one persistent launch for all sources of a call,
// teams of blocks running several of them at a time.
//
// Reference path: bfs_gpu (src/kernels/gpu/bfs.cuh:21-95) runs bottom-up
// epochs only, one launch + blocking 4-byte D2H + cudaMemset per level; the
// direction heuristic lives in the CPU bfs_do_cpu (src/kernels/cpu/bfs.cuh:48-114,
// alpha = 15, beta = 18).  Here the whole level loop runs on the device: every
// block evaluates the same alpha/beta state machine from counters read after a
// grid barrier, so the per-level selector costs no host round trip.
//
// HBM layout of the working set (W = ceil(N/32) words):
//   depth, parent  int32[N]      outputs (caller's device buffer or ours)
//   visited        uint32[W]     claimed vertices
//   fb[3]          uint32[W]     frontier bitmaps of bottom-up levels: level L
//                                reads fb[L%3], writes fb[(L+1)%3], zeroes
//                                fb[(L+2)%3]; top-down levels keep a queue
//                                only, and the first bottom-up level after
//                                one builds its bitmap from the queue
//   q[2]           int32[N]      frontier queues (top-down levels)
//   tasks          int2[]        (vertex, chunk) pieces of long rows
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <cstdlib>
#include <mutex>
#include <thread>
#include <vector>

#include "hc_expand.cuh"
#include "hc_graph.cuh"

namespace hc {
namespace {

constexpr int kBfsThreads = 512;
constexpr int kBuSplitLevels = HC_BFS_SPLIT_LEVELS;
constexpr int kTraceLevels = 64;
// Bottom-up levels copy the first kHubWords words of the frontier bitmap
// (the 131072 highest-degree vertices of a degree-sorted graph, which most
// edges point at) into shared memory and probe them there.
constexpr int kHubWords = 4096;
// Every frontier bitmap has a summary: bit i set when one of its words
// [i << sum_shift, (i + 1) << sum_shift) is non-zero, at most kSumWords words,
// so bottom-up levels keep it in shared memory and probe the bitmap in global
// memory only for neighbours whose summary bit is set (on a sparse frontier,
// few: most rows that find no parent stop reading global memory).
constexpr int kSumWords = 4096;
// Thin top-down levels (at most kSoloCap vertices with at most kSoloEdges
// edges, none of more than kSoloDeg) run on the team's first block alone, a
// block barrier per level and the frontier in shared memory, for up to
// kSoloLevels levels at a time while the other blocks wait at one grid
// barrier.  Such a level is a chain of dependent L2 round trips: on the grid it
// also pays the barrier and the global queue's counters (a 100-vertex level of a
// grid graph: 2.9 us here, 7 us there).  The limits: one block keeps 2048 edges
// in flight, and above one round of those the grid is faster (1023 x 1025
// grid: limit 1024 9.6 ms, 2048 9.1 ms, 4096 10.0 ms, 8192 13.5 ms, no thin
// levels 16 ms); a row longer than kSoloDeg would serialise on one warp.
constexpr int kSoloCap = 1920;
constexpr int kSoloEdges = 2048;
constexpr int kSoloDeg = 128;
constexpr int kSoloLevels = 1024;

struct LevelCnt {
    int nf;                 // vertices in this frontier
    int tasks;              // long-row tasks queued while expanding it
    unsigned long long mf;  // sum of their degrees (top-down only)
};

struct BfsCtl {
    GridSync gs;
    LevelCnt cnt[2][3];     // by run parity: a run's counters are set while blocks may still read the last run's
    int conv;               // bitmap -> queue conversion counter
    int levels, td_levels, bu_levels;
    unsigned long long vscan, escan, reached;
    struct {
        int L, nf, td_levels;
        long long edges_to_check, num_edges;
    } solo;                  // loop state after the first block's thin levels
    struct {
        int mode, nf;
        unsigned long long t_ns;
    } trace[kTraceLevels + 1];  // per-level record for HC_TRACE=1
};

// Results of the runs of one call, folded on the device after each run so
// that the host need not wait for each source: the first failure (status and
// source), the deepest run, the top-down / bottom-up level counts.
struct BfsFold {
    int err, err_src, levels, td_levels, bu_levels;
    int teams_done;  // of the running launch
};

// Sources of one launch.
constexpr int kBfsLaunchSources = 256;
// Bytes that the workspaces of sources run at the same time may take in all;
// past it (and when they cannot be allocated) fewer run at a time.
constexpr size_t kBfsTeamBytes = 1ull << 30;

struct BfsArgs {
    const int64_t *index;
    const int32_t *nbr;
    int32_t n, n_active, n_warp_rows;
    int64_t m;
    int32_t *depth, *parent;
    uint32_t *visited, *fb0, *fb1, *fb2;
    uint32_t *sb0, *sb1, *sb2;  // the frontier bitmaps' summaries (sum_words words each)
    int sum_shift, sum_words;
    int32_t *q0, *q1;
    int2 *tasks;
    BfsCtl *ctl;
    BfsFold *fold, *fold_host;  // fold_host: mapped host copy, written by the launch's last team (null: none)
    // Teams of `team` consecutive blocks run one source at a time each, team t
    // the sources t, t + teams, ...; the pointers above are team 0's, team t's
    // lie t * team_stride bytes (depth, parent: see out_stride) further on.
    int team;
    size_t team_stride;
    // Output row of source i: depth + i * out_stride (out_stride 0: not wanted,
    // one scratch row per team).
    int64_t depth_stride, parent_stride;
    int nsrc;
    int32_t src[kBfsLaunchSources];
    int alpha, beta, direction, bu_variant, max_levels;
    // Per bottom-up level warp/thread split (the per-epoch granularity
    // selector): bottom-up level k (0 = the first) runs warp per vertex on
    // [0, bu_split[min(k, bu_split_levels - 1)]) and thread per vertex after;
    // bu_split_levels 0 = the fixed split of bu_variant.
    int32_t bu_split[kBuSplitLevels];
    int bu_split_levels;
};

// A workspace pointer of this team.
template <class T>
__device__ __forceinline__ T *of_team(T *p, size_t off) {
    return reinterpret_cast<T *>(reinterpret_cast<char *>(p) + off);
}
// What one run works on: the team's share of the workspace and the source's
// outputs.  Kept in shared memory: as registers these pointers would spill the
// levels' inner loops.
struct BfsRun {
    int32_t src;
    int32_t *depth, *parent;
    uint32_t *visited;
    int32_t *q0, *q1;
    int2 *tasks;
    uint32_t *fb[3], *sb[3];
};

// Sets vertex v's bit in a frontier bitmap and, when its word was empty, the
// word's summary bit.
__device__ __forceinline__ void frontier_add(uint32_t *fb, uint32_t *sb, int cs, int32_t v) {
    const int w = v >> 5;
    if (atomicOr(fb + w, 1u << (v & 31)) == 0u) atomicOr(sb + ((w >> cs) >> 5), 1u << ((w >> cs) & 31));
}

// Word of the frontier bitmap that holds vertex u's bit: the shared copy of
// the hub prefix for u < hub_v, else 0 when u's summary bit (shared) is clear,
// else the bitmap in global memory.  u < 0 (no edge) reads as 0.
__device__ __forceinline__ uint32_t frontier_word_sum(const uint32_t *s_fb, int hub_v, const uint32_t *s_sum, int cs,
                                                      const uint32_t *fb, int32_t u) {
    const bool hub = u >= 0 && u < hub_v;
    const int sw_i = (max(u, 0) >> 5) >> cs;
    const bool need = u >= 0 && !hub && ((s_sum[sw_i >> 5] >> (sw_i & 31)) & 1u);
    const uint32_t hw = s_fb[hub ? (u >> 5) : 0];
    const uint32_t gw = need ? __ldcg(fb + (u >> 5)) : 0u;
    return hub ? hw : gw;
}

// Top-down edge visitor: claim an unvisited neighbour with a CAS on its
// parent, mark it visited, queue it.
struct TopDownVisit {
    const int64_t *index;
    const int32_t *nbr;
    int32_t *parent, *depth;
    uint32_t *visited;
    int32_t *qnext;
    int *qlen;
    int next_depth;
    unsigned long long mf;  // degree sum of the claimed vertices (this thread)
    struct Item {
        int32_t u, v;
        uint32_t word;
    };
    __device__ __forceinline__ void load(Item &it, int32_t u, int64_t e) {
        it.u = u;
        it.v = __ldg(nbr + e);
    }
    __device__ __forceinline__ void probe(Item &it) { it.word = __ldcg(visited + (it.v >> 5)); }
    // Stages across the round's items: all CASes in flight, then the marks,
    // then one queue append for the whole warp.
    __device__ __forceinline__ void commit(Item (&it)[kUnroll], const bool (&act)[kUnroll]) {
        bool take[kUnroll];
        int32_t old[kUnroll], v[kUnroll];
#pragma unroll
        for (int j = 0; j < kUnroll; j++) {
            take[j] = act[j] && !((it[j].word >> (it[j].v & 31)) & 1u);
            old[j] = take[j] ? atomicCAS(parent + it[j].v, -1, it[j].u) : 0;
        }
#pragma unroll
        for (int j = 0; j < kUnroll; j++) {
            take[j] = take[j] && old[j] == -1;
            v[j] = take[j] ? it[j].v : 0;
            if (take[j]) {
                depth[v[j]] = next_depth;
                atomicOr(visited + (v[j] >> 5), 1u << (v[j] & 31));
            }
        }
#pragma unroll
        for (int j = 0; j < kUnroll; j++)
            if (take[j]) mf += (unsigned long long)(__ldg(index + v[j] + 1) - __ldg(index + v[j]));
        warp_append_n(take, v, qnext, qlen);
    }
};

// Shared-memory queue of the thin levels: vertex, and its row's first slot and
// degree packed (44 + 20 bits, the degree clamped).
struct SoloQueue {
    int32_t u[kSoloCap];
    unsigned long long row[kSoloCap];
};
constexpr unsigned long long kSoloDegMask = (1ull << 20) - 1ull;
__device__ __forceinline__ unsigned long long solo_row(int64_t b, int64_t d) {
    return ((unsigned long long)b << 20) | min((unsigned long long)d, kSoloDegMask);
}

// Thin top-down levels from level *L on, by one block (every thread calls it).
// The same level as the grid's (claim by CAS on parent, mark, queue), with the
// queue in shared memory and mirrored in the global queue, so that the grid can
// take any level over.  Stops before a level that is too wide, that the
// direction rule turns bottom-up, after kSoloLevels levels, or when the queue
// is empty.  Returns with the loop state updated in every thread.
struct SoloState {
    int L, nf, td_levels;
    long long edges_to_check, num_edges;
    unsigned long long vscan, escan;
};
struct SoloArgs {
    const int64_t *index;
    const int32_t *nbr;
    int direction, alpha, max_levels;
};
// Not inlined: its registers would spill the grid's levels.
template <bool kStats>
__device__ __noinline__ SoloState solo_levels(SoloArgs a, const BfsRun &r, BfsCtl *ctl, SoloQueue *sq, SoloState st) {
    int L = st.L, nf = st.nf, td_levels = st.td_levels;
    int32_t *const parent = r.parent, *const depth = r.depth;
    uint32_t *const visited = r.visited;
    long long edges_to_check = st.edges_to_check, num_edges = st.num_edges;
    unsigned long long my_vscan = st.vscan, my_escan = st.escan;
    __shared__ int s_n[3];
    __shared__ unsigned long long s_sum;
    __shared__ unsigned s_mf[3];  // exact while no row is long (see the end)
    __shared__ int s_wide[3];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int32_t *qin = (L & 1) ? r.q1 : r.q0;
    if (threadIdx.x < 3) {
        s_n[threadIdx.x] = 0;
        s_mf[threadIdx.x] = 0u;
        s_wide[threadIdx.x] = 0;
    }
    __syncthreads();
    unsigned edges = 0;
    for (int i = threadIdx.x; i < nf; i += blockDim.x) {
        const int32_t u = __ldcg(qin + i);
        const int64_t b = __ldg(a.index + u), d = __ldg(a.index + u + 1) - b;
        sq[0].u[i] = u;
        sq[0].row[i] = solo_row(b, d);
        edges += (unsigned)min(d, (int64_t)kSoloEdges);
        if (d > kSoloDeg) s_wide[0] = 1;
    }
    // The frontier's own edges: after a bottom-up level num_edges is not their count.
    edges = __reduce_add_sync(kFull, edges);
    if (lane == 0 && edges) atomicAdd(&s_mf[0], edges);
    __syncthreads();
    bool wide = s_wide[0] || s_mf[0] > (unsigned)kSoloEdges;
    for (int step = 0; step < kSoloLevels; step++) {
        const int ns = (step + 1) % 3;
        if (nf == 0 || nf > kSoloCap || wide || L >= a.max_levels ||
            (a.direction == 0 && num_edges > edges_to_check / a.alpha))
            break;
        const SoloQueue &cq = sq[step & 1];
        SoloQueue &nq = sq[(step + 1) & 1];
        int32_t *qnext = (L & 1) ? r.q0 : r.q1;
        edges_to_check -= num_edges;
        td_levels++;
        if (threadIdx.x == 0) {
            s_n[(step + 2) % 3] = 0;
            s_mf[(step + 2) % 3] = 0u;
            s_wide[(step + 2) % 3] = 0;
            if (L < kTraceLevels) {
                ctl->trace[L].mode = 1;
                ctl->trace[L].nf = nf;
                ctl->trace[L].t_ns = globaltimer_ns();
            }
            if (kStats) {
                my_vscan += nf;
                my_escan += s_mf[step % 3];  // num_edges is 1 after a bottom-up level
            }
        }
        const int per = min(32, max(1, (nf + nwarps - 1) / nwarps));
        for (int base = wib * per; base < nf; base += nwarps * per) {
            const int i = base + lane;
            const bool mine = lane < per && i < nf;
            const int32_t u = mine ? cq.u[i] : -1;
            const unsigned long long row = mine ? cq.row[i] : 0ull;
            const long long beg = (long long)(row >> 20);
            int total;
            const int excl = warp_exclusive_scan((int)(row & kSoloDegMask), &total);
            for (int k0 = 0; k0 < total; k0 += 32 * kUnroll) {
                int32_t v[kUnroll], from[kUnroll];
                uint32_t word[kUnroll];
                bool take[kUnroll];
#pragma unroll
                for (int j = 0; j < kUnroll; j++) {
                    const int k = k0 + 32 * j + lane;
                    int lo = 0;
#pragma unroll
                    for (int st = 16; st > 0; st >>= 1) {
                        const int c = __shfl_sync(kFull, excl, lo + st);
                        if (c <= k) lo += st;
                    }
                    from[j] = __shfl_sync(kFull, u, lo);
                    const long long bo = __shfl_sync(kFull, beg, lo);
                    const int off = k - __shfl_sync(kFull, excl, lo);
                    take[j] = k < total;
                    v[j] = take[j] ? __ldg(a.nbr + bo + off) : 0;
                }
#pragma unroll
                for (int j = 0; j < kUnroll; j++) word[j] = take[j] ? __ldcg(visited + (v[j] >> 5)) : ~0u;
#pragma unroll
                for (int j = 0; j < kUnroll; j++)
                    from[j] = (word[j] >> (v[j] & 31)) & 1u ? 0 : atomicCAS(parent + v[j], -1, from[j]);
#pragma unroll
                for (int j = 0; j < kUnroll; j++) take[j] = from[j] == -1;
                unsigned bal[kUnroll];
                int count = 0;
#pragma unroll
                for (int j = 0; j < kUnroll; j++) {
                    bal[j] = __ballot_sync(kFull, take[j]);
                    count += __popc(bal[j]);
                }
                if (count == 0) continue;
                int pos = 0;
                if (lane == 0) pos = atomicAdd(&s_n[ns], count);
                pos = __shfl_sync(kFull, pos, 0);
                int64_t nb[kUnroll], nd[kUnroll];
#pragma unroll
                for (int j = 0; j < kUnroll; j++) {
                    nb[j] = take[j] ? __ldg(a.index + v[j]) : 0;
                    nd[j] = take[j] ? __ldg(a.index + v[j] + 1) : 0;
                }
                unsigned dsum = 0;
#pragma unroll
                for (int j = 0; j < kUnroll; j++) {
                    if (take[j]) {
                        const int p = pos + __popc(bal[j] & lt);
                        depth[v[j]] = L + 1;
                        atomicOr(visited + (v[j] >> 5), 1u << (v[j] & 31));
                        qnext[p] = v[j];
                        if (p < kSoloCap) {
                            nq.u[p] = v[j];
                            nq.row[p] = solo_row(nb[j], nd[j] - nb[j]);
                        }
                        dsum += (unsigned)min(nd[j] - nb[j], (int64_t)kSoloEdges);
                        if (nd[j] - nb[j] > kSoloDeg) s_wide[ns] = 1;
                    }
                    pos += __popc(bal[j]);
                }
                dsum = __reduce_add_sync(kFull, dsum);
                if (lane == 0) atomicAdd(&s_mf[ns], dsum);
            }
        }
        __syncthreads();
        nf = s_n[ns];
        num_edges = (long long)s_mf[ns];
        wide = s_wide[ns] || num_edges > kSoloEdges;
        L++;
    }
    if (wide && L != st.L) {
        // The sum of a frontier with long rows, exactly: the direction rule reads it.
        __syncthreads();
        if (threadIdx.x == 0) s_sum = 0ull;
        __syncthreads();
        const int32_t *q = (L & 1) ? r.q1 : r.q0;
        unsigned long long sum = 0;
        for (int i = threadIdx.x; i < nf; i += blockDim.x) {
            const int32_t u = __ldcg(q + i);
            sum += (unsigned long long)(__ldg(a.index + u + 1) - __ldg(a.index + u));
        }
        sum = warp_sum(sum);
        if (lane == 0 && sum) atomicAdd(&s_sum, sum);
        __syncthreads();
        num_edges = (long long)s_sum;
    }
    return SoloState{L, nf, td_levels, edges_to_check, num_edges, my_vscan, my_escan};
}

// Shared memory of one block: the hub prefix and the summary of the frontier
// bitmap (bottom-up levels), or the two queues of the thin levels.
union BfsShared {
    struct {
        uint32_t fb[kHubWords];
        uint32_t sum[kSumWords];
    } bu;
    SoloQueue solo[2];
};

// kBlocks resident blocks per SM: two, or three for many sources at a time.  The
// levels wait on dependent loads (issue slots 32 % used, DRAM 14 %), and with
// enough work to fill them a third block's warps are worth the spills they cost:
// from kBfsWideWork edges times sources on, two sources at least.  Two / three
// blocks in us: Kronecker scale 22, 1 source 273 / 283, 2 410 / 401, 16 2043 / 1606;
// scale 20, 2 169 / 185, 4 220 / 214; scale 18, 8 160 / 166, 16 210 / 199; scale 16,
// 16 123 / 130, 64 218 / 209; uniform 2^18 vertices, 4 194 / 197, 16 454 / 453; 2^16, 16
// 134 / 136, 64 322 / 276.
constexpr int64_t kBfsWideWork = 1ll << 26;
template <bool kStats, int kBlocks>
__global__ void __launch_bounds__(kBfsThreads, kBlocks) bfs_persistent(BfsArgs a) {
    __shared__ unsigned long long s_red[32];
    __shared__ BfsShared sh;
    __shared__ int s_stop;
    uint32_t *const s_fb = sh.bu.fb, *const s_sum = sh.bu.sum;
    const int lane = threadIdx.x & 31;
    const int team = blockIdx.x / a.team, team_block = blockIdx.x - team * a.team;
    const int nteams = gridDim.x / a.team;
    BfsCtl *ctl = a.ctl + team;
    const size_t toff = (size_t)team * a.team_stride;
    const int gtid = team_block * blockDim.x + threadIdx.x;
    const int nthreads = a.team * blockDim.x;
    const int gwarp = gtid >> 5, nwarps = nthreads >> 5;
    const int W = (a.n + 31) >> 5;
    const int W_act = (a.n_active + 31) >> 5;
    // A team of one block needs no more than its own block barrier.
    bool stop = false;  // thread 0 of a one-block team: it recorded a failure
    auto team_sync = [&]() -> bool {
        if (a.team > 1) return grid_barrier(&ctl->gs, (unsigned)a.team);
        __syncthreads();
        if (threadIdx.x == 0) s_stop = stop;
        __syncthreads();
        return !s_stop;
    };

    __shared__ BfsRun r;
    if (threadIdx.x == 0) {
        r.visited = of_team(a.visited, toff);
        r.q0 = of_team(a.q0, toff);
        r.q1 = of_team(a.q1, toff);
        r.tasks = of_team(a.tasks, toff);
        r.fb[0] = of_team(a.fb0, toff);
        r.fb[1] = of_team(a.fb1, toff);
        r.fb[2] = of_team(a.fb2, toff);
        r.sb[0] = of_team(a.sb0, toff);
        r.sb[1] = of_team(a.sb1, toff);
        r.sb[2] = of_team(a.sb2, toff);
    }
    unsigned long long my_vscan = 0, my_escan = 0;
    bool failed = false;
    int run = 0;

    for (int si = team; si < a.nsrc && !failed; si += nteams, run++) {
    __syncthreads();  // the last run's reads of r
    if (threadIdx.x == 0) {
        r.src = a.src[si];
        r.depth = a.depth + (a.depth_stride ? (size_t)si * a.depth_stride : (size_t)team * a.n);
        r.parent = a.parent + (a.parent_stride ? (size_t)si * a.parent_stride : (size_t)team * a.n);
    }
    __syncthreads();
    LevelCnt *const cnt = ctl->cnt[run & 1];
    {
        const int32_t src = r.src;
        int32_t *const depth = r.depth, *const parent = r.parent;
        for (int i = gtid; i < a.n; i += nthreads) {
            depth[i] = i == src ? 0 : -1;
            parent[i] = i == src ? i : -1;
        }
        uint32_t *const vis = r.visited, *const f0 = r.fb[0], *const f1 = r.fb[1], *const f2 = r.fb[2];
        for (int i = gtid; i < W; i += nthreads) {
            vis[i] = i == (src >> 5) ? 1u << (src & 31) : 0u;
            f0[i] = 0;
            f1[i] = 0;
            f2[i] = 0;
        }
        uint32_t *const s0 = r.sb[0], *const s1 = r.sb[1], *const s2 = r.sb[2];
        for (int i = gtid; i < a.sum_words; i += nthreads) {
            s0[i] = 0;
            s1[i] = 0;
            s2[i] = 0;
        }
    }
    const unsigned long long t_start = globaltimer_ns();
    if (gtid == 0) {
        r.q0[0] = r.src;
        cnt[0] = LevelCnt{1, 0, (unsigned long long)(a.index[r.src + 1] - a.index[r.src])};
        cnt[1] = LevelCnt{0, 0, 0ull};
        cnt[2] = LevelCnt{0, 0, 0ull};
    }
    failed = !team_sync();

    // Direction state (identical in every block).
    bool push = a.direction != 2;
    bool have_queue = true;
    // Thin levels may go to one block; a level of the whole grid lies between two
    // such turns, so that nobody still reads the state of the last one.
    bool solo_ok = true;
    bool bitmaps_clear = true;  // all three frontier bitmaps are zero (no bottom-up level yet)
    long long edges_to_check = a.m;
    long long num_edges = (long long)(a.index[r.src + 1] - a.index[r.src]);
    int L = 0, td_levels = 0, bu_levels = 0;
    // The level counters rotate with the levels that the whole grid runs: the
    // thin levels of one block leave them alone, since other blocks may still
    // be reading those of the last one.
    int C = 0;
    int solo_nf = -1;  // frontier size after thin levels (-1: in the counters)

    while (!failed) {
        const int cur = L % 3, nxt = (L + 1) % 3, old = (L + 2) % 3;
        LevelCnt *const ccur = &cnt[C % 3], *const cnxt = &cnt[(C + 1) % 3];
        int nf = solo_nf >= 0 ? solo_nf : __ldcg(&ccur->nf);
        solo_nf = -1;
        if (nf == 0) break;
        if (L >= a.max_levels) {
            if (gtid == 0) atomicExch(&ctl->gs.err, (int)HC_ERR_NOT_CONVERGED);
            break;
        }
        if (gtid == 0) {
            if (globaltimer_ns() - t_start > c_limits.run_ns) {
                atomicExch(&ctl->gs.err, (int)HC_ERR_TIMEOUT);
                stop = true;
            }
            LevelCnt *const cold = &cnt[(C + 2) % 3];
            cold->nf = 0;
            cold->tasks = 0;
            cold->mf = 0;
        }
        uint32_t *fcur = r.fb[cur], *fnext = r.fb[nxt], *fold = r.fb[old];
        uint32_t *scur = r.sb[cur], *snext = r.sb[nxt], *sold = r.sb[old];
        int32_t *qcur = (L & 1) ? r.q1 : r.q0;
        int32_t *qnext = (L & 1) ? r.q0 : r.q1;

        if (a.direction == 0 && push && num_edges > edges_to_check / a.alpha) push = false;
        if (gtid == 0 && L < kTraceLevels) {
            ctl->trace[L].mode = push ? 1 : 2;
            ctl->trace[L].nf = nf;
            ctl->trace[L].t_ns = globaltimer_ns();
        }

        if (push) {
            if (!have_queue) {
                // Frontier came from a bottom-up level: compact its bitmap.
                for (int w0 = gwarp * 32; w0 < W_act; w0 += nwarps * 32) {
                    const int w = w0 + lane;
                    uint32_t bits = w < W_act ? __ldcg(fcur + w) : 0u;
                    int total;
                    int pos = warp_exclusive_scan(__popc(bits), &total);
                    int base = 0;
                    if (lane == 0 && total) base = atomicAdd(&ctl->conv, total);
                    pos += __shfl_sync(kFull, base, 0);
                    while (bits) {
                        const int b = __ffs(bits) - 1;
                        bits &= bits - 1;
                        qcur[pos++] = w * 32 + b;
                    }
                }
                if ((failed = !team_sync())) break;
                nf = __ldcg(&ctl->conv);
                have_queue = true;
            }
            if (solo_ok && nf <= kSoloCap && num_edges <= kSoloEdges) {
                const int L0 = L;
                solo_ok = false;
                if (team_block == 0) {
                    const SoloState st = solo_levels<kStats>(
                        SoloArgs{a.index, a.nbr, a.direction, a.alpha, a.max_levels}, r, ctl, sh.solo,
                        SoloState{L, nf, td_levels, edges_to_check, num_edges, my_vscan, my_escan});
                    L = st.L;
                    nf = st.nf;
                    td_levels = st.td_levels;
                    edges_to_check = st.edges_to_check;
                    num_edges = st.num_edges;
                    my_vscan = st.vscan;
                    my_escan = st.escan;
                    if (threadIdx.x == 0) {
                        ctl->solo.L = L;
                        ctl->solo.nf = nf;
                        ctl->solo.td_levels = td_levels;
                        ctl->solo.edges_to_check = edges_to_check;
                        ctl->solo.num_edges = num_edges;
                    }
                }
                if ((failed = !team_sync())) break;
                L = __ldcg(&ctl->solo.L);
                if (L != L0) {
                    solo_nf = __ldcg(&ctl->solo.nf);
                    td_levels = __ldcg(&ctl->solo.td_levels);
                    edges_to_check = __ldcg(&ctl->solo.edges_to_check);
                    num_edges = __ldcg(&ctl->solo.num_edges);
                    continue;
                }
            }
            edges_to_check -= num_edges;
            td_levels++;
            const int next_depth = L + 1;
            TopDownVisit visit{a.index, a.nbr, r.parent, r.depth, r.visited, qnext, &cnxt->nf, next_depth,
                               0ull};
            if (kStats) {
                for (int i = gtid; i < nf; i += nthreads) {
                    const int32_t u = __ldcg(qcur + i);
                    my_escan += (unsigned long long)(a.index[u + 1] - a.index[u]);
                }
                if (gtid == 0) my_vscan += nf;
            }
            expand_small(a.index, qcur, nf, r.tasks, &ccur->tasks, gwarp, nwarps, visit);
            unsigned long long mf_blk = block_sum(visit.mf, s_red);
            if (threadIdx.x == 0 && mf_blk) atomicAdd(&cnxt->mf, mf_blk);
            if ((failed = !team_sync())) break;
            const int nt = __ldcg(&ccur->tasks);
            if (nt > 0) {
                visit.mf = 0;
                expand_tasks(a.index, r.tasks, nt, gwarp, nwarps, visit);
                mf_blk = block_sum(visit.mf, s_red);
                if (threadIdx.x == 0 && mf_blk) atomicAdd(&cnxt->mf, mf_blk);
                if ((failed = !team_sync())) break;
            }
            num_edges = (long long)__ldcg(&cnxt->mf);
            have_queue = true;
        } else {
            if (have_queue) {
                // Frontier came from a top-down level: set its bits.  This
                // level's and the next one's bitmaps must be zero first.
                if (!bitmaps_clear) {
                    for (int i = gtid; i < W_act; i += nthreads) {
                        fcur[i] = 0;
                        fnext[i] = 0;
                    }
                    for (int i = gtid; i < a.sum_words; i += nthreads) {
                        scur[i] = 0;
                        snext[i] = 0;
                    }
                    if ((failed = !team_sync())) break;
                }
                for (int i = gtid; i < nf; i += nthreads) frontier_add(fcur, scur, a.sum_shift, __ldcg(qcur + i));
                if ((failed = !team_sync())) break;
            }
            bitmaps_clear = false;
            for (int i = gtid; i < W_act; i += nthreads) fold[i] = 0;
            for (int i = gtid; i < a.sum_words; i += nthreads) sold[i] = 0;
            bu_levels++;
            const int next_depth = L + 1;
            int found_local = 0;
            // The frontier bitmap is complete (grid barrier) and read-only in
            // this level: copy its hub prefix.
            const int hub_w = min(kHubWords, W_act);
            const int hub_v = hub_w << 5;
            for (int i = threadIdx.x; i < hub_w; i += blockDim.x) s_fb[i] = __ldcg(fcur + i);
            for (int i = threadIdx.x; i < a.sum_words; i += blockDim.x) s_sum[i] = __ldcg(scur + i);
            __syncthreads();
            const int cs = a.sum_shift;
            // Rows of degree >= 32: warp per vertex, 32 probes per step.
            // AUTO = thread granularity with four probes in flight: on the
            // degree-sorted Kronecker graphs it beats warp-per-row for the
            // >= 32-edge prefix (0.36 vs 0.68 ms per source at scale 22), since
            // the first probes of a sorted row usually hit.  BLOCK selects the
            // warp path only for that prefix.
            const int n_warp = a.bu_split_levels > 0
                                   ? a.bu_split[min(bu_levels - 1, a.bu_split_levels - 1)]
                                   : a.bu_variant == HC_VARIANT_WARP
                                         ? a.n_active
                                         : (a.bu_variant == HC_VARIANT_BLOCK ? a.n_warp_rows : 0);
            const int n_warp_al = min(((n_warp + 31) >> 5) << 5, W_act << 5);
            for (int v = gwarp; v < n_warp_al; v += nwarps) {
                if (v >= a.n_active) break;
                const uint32_t bit = 1u << (v & 31);
                if (__ldcg(r.visited + (v >> 5)) & bit) continue;
                const int64_t b = a.index[v], e = a.index[v + 1];
                int32_t par = -1;
                int64_t probes = 0;
                for (int64_t e0 = b; e0 < e; e0 += 32) {
                    const int64_t i = e0 + lane;
                    bool hit = false;
                    int32_t u = 0;
                    if (i < e) {
                        u = a.nbr[i];
                        hit = (frontier_word_sum(s_fb, hub_v, s_sum, cs, fcur, u) >> (u & 31)) & 1u;
                    }
                    const unsigned bal = __ballot_sync(kFull, hit);
                    if (kStats) probes += bal ? (int64_t)__ffs(bal) : ((e - e0) < 32 ? (e - e0) : (int64_t)32);
                    if (bal) {
                        par = __shfl_sync(kFull, u, __ffs(bal) - 1);
                        break;
                    }
                }
                if (kStats && lane == 0) {
                    my_vscan++;
                    my_escan += probes;
                }
                if (par >= 0 && lane == 0) {
                    r.parent[v] = par;
                    r.depth[v] = next_depth;
                    atomicOr(r.visited + (v >> 5), bit);
                    frontier_add(fnext, snext, cs, v);
                    found_local++;
                }
            }
            // Remaining rows: thread per vertex, warp owns one bitmap word.
            for (int w = (n_warp_al >> 5) + gwarp; w < W_act; w += nwarps) {
                const uint32_t vis = __ldcg(r.visited + w);
                const int v = w * 32 + lane;
                int32_t par = -1;
                if (v < a.n_active && !((vis >> lane) & 1u)) {
                    const int64_t b = a.index[v], e = a.index[v + 1];
                    // Four probes in flight per round; any frontier neighbour is a valid parent.
                    for (int64_t i = b; i < e && par < 0; i += 4) {
                        int32_t u[4];
                        uint32_t wd[4];
#pragma unroll
                        for (int j = 0; j < 4; j++) u[j] = i + j < e ? a.nbr[i + j] : -1;
#pragma unroll
                        for (int j = 0; j < 4; j++) wd[j] = frontier_word_sum(s_fb, hub_v, s_sum, cs, fcur, u[j]);
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            if (par < 0 && u[j] >= 0 && ((wd[j] >> (u[j] & 31)) & 1u)) {
                                par = u[j];
                                if (kStats) my_escan += (unsigned long long)(i + j - b + 1);
                            }
                    }
                    if (kStats) {
                        my_vscan++;
                        if (par < 0) my_escan += (unsigned long long)(e - b);
                    }
                }
                const unsigned bal = __ballot_sync(kFull, par >= 0);
                if (par >= 0) {
                    r.parent[v] = par;
                    r.depth[v] = next_depth;
                }
                if (lane == 0) {
                    fnext[w] = bal;
                    if (bal) {
                        r.visited[w] = vis | bal;
                        atomicOr(snext + ((w >> cs) >> 5), 1u << ((w >> cs) & 31));
                    }
                    found_local += __popc(bal);
                }
            }
            unsigned long long f_blk = block_sum((unsigned long long)found_local, s_red);
            if (threadIdx.x == 0 && f_blk) atomicAdd((unsigned long long *)&ctl->reached, f_blk);
            if (threadIdx.x == 0 && f_blk) atomicAdd(&cnxt->nf, (int)f_blk);
            if (gtid == 0) ctl->conv = 0;
            if ((failed = !team_sync())) break;
            const int nf_next = __ldcg(&cnxt->nf);
            if (a.direction == 0 && !(nf_next > nf || nf_next > a.n / a.beta)) {
                push = true;
                num_edges = 1;
            }
            have_queue = false;
        }
        L++;
        C++;
        solo_ok = true;
    }

    if (gtid == 0) {
        ctl->levels = L;
        ctl->trace[L < kTraceLevels ? L : kTraceLevels].t_ns = globaltimer_ns();
        ctl->td_levels = td_levels;
        ctl->bu_levels = bu_levels;
        const int err = *(volatile int *)&ctl->gs.err;
        if (err && atomicCAS(&a.fold->err, 0, err) == 0) a.fold->err_src = r.src;
        atomicMax(&a.fold->levels, L);
        atomicAdd(&a.fold->td_levels, td_levels);
        atomicAdd(&a.fold->bu_levels, bu_levels);
    }
    }  // next source

    if (gtid == 0) {
        __threadfence();
        if (atomicAdd(&a.fold->teams_done, 1) == nteams - 1) {
            __threadfence();
            a.fold->teams_done = 0;
            if (a.fold_host) {
                a.fold_host->err = __ldcg(&a.fold->err);
                a.fold_host->err_src = __ldcg(&a.fold->err_src);
                a.fold_host->levels = __ldcg(&a.fold->levels);
                a.fold_host->td_levels = __ldcg(&a.fold->td_levels);
                a.fold_host->bu_levels = __ldcg(&a.fold->bu_levels);
                __threadfence_system();
            }
        }
    }

    if (kStats) {
        unsigned long long v = block_sum(my_vscan, s_red);
        if (threadIdx.x == 0 && v) atomicAdd(&ctl->vscan, v);
        unsigned long long e = block_sum(my_escan, s_red);
        if (threadIdx.x == 0 && e) atomicAdd(&ctl->escan, e);
    }
}

// Discovered count for top-down levels is the queue length; add it up after
// the run from the per-level counters is not possible (they rotate), so the
// reached total is recounted from the depth array.
__global__ void count_reached(const int32_t *depth, int32_t n, unsigned long long *out) {
    __shared__ unsigned long long s_red[32];
    unsigned long long c = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        c += depth[i] >= 0;
    c = block_sum(c, s_red);
    if (threadIdx.x == 0 && c) atomicAdd(out, c);
}

// Host outputs on a degree-sorted graph: the vertices [n_copy, n) have no
// edges, so every run leaves their depth and parent at -1 (a source among
// them aside: depth 0, parent itself).  A few host threads write those
// suffixes while the GPU runs, and only the first n_copy entries of each
// source's rows cross PCIe.  The threads are joined by the destructor, on
// every return path.
struct SuffixFill {
    std::vector<std::thread> th;
    void start(int32_t *depth, int32_t *parent, const std::vector<int32_t> &src, int64_t n, int64_t n_copy) {
        const int k = (int)src.size();
        const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
        const int nt = std::max(1, std::min({(int)(hw / 2), 8, k}));
        auto part = [=, &src](int t) {
            for (int i = t; i < k; i += nt) {
                for (int32_t *out : {depth, parent}) {
                    if (!out) continue;
                    // -1 in every byte is -1 in every int32; a large memset streams its
                    // stores without reading the lines first.
                    std::memset(out + (size_t)i * n + n_copy, 0xFF, sizeof(int32_t) * (size_t)(n - n_copy));
                }
                const int32_t s = src[i];
                if (s >= n_copy) {
                    if (depth) depth[(size_t)i * n + s] = 0;
                    if (parent) parent[(size_t)i * n + s] = s;
                }
            }
        };
        for (int t = 0; t < nt; t++) {
            try {
                th.emplace_back(part, t);
            } catch (...) {  // no thread to be had: this share runs here (nothing throws past the C ABI)
                part(t);
            }
        }
    }
    ~SuffixFill() {
        for (auto &t : th) t.join();
    }
};

// Clears the fold record and what the teams' control blocks must start from.
__global__ void bfs_clear(BfsCtl *ctl, int teams, BfsFold *f) {
    if (threadIdx.x == 0) *f = BfsFold{0, 0, 0, 0, 0, 0};
    for (int t = threadIdx.x; t < teams; t += blockDim.x) {
        ctl[t].gs = GridSync{0ull, 0, 0};
        ctl[t].conv = 0;
        ctl[t].vscan = ctl[t].escan = ctl[t].reached = 0ull;
    }
}

// Blocks of bfs_persistent that are resident at a time.
template <bool kStats, int kBlocks>
hc_status bfs_resident(hc_graph *g, int *blocks) {
    static int blocks_per_sm = 0;
    if (blocks_per_sm == 0) {
        HC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, bfs_persistent<kStats, kBlocks>,
                                                                  kBfsThreads, 0));
        if (blocks_per_sm < 1) return fail(HC_ERR_CUDA, "BFS kernel cannot be resident");
    }
    *blocks = blocks_per_sm * g->sm_count;
    return HC_OK;
}

template <bool kStats, int kBlocks>
hc_status launch_bfs(hc_graph *g, BfsArgs &a, int teams) {
    dim3 grid(a.team * teams), block(kBfsThreads);
    ::hc::count_launch();
    if (a.team == 1) {  // no block waits for another
        bfs_persistent<kStats, kBlocks><<<grid, block, 0, g->stream>>>(a);
        HC_CUDA_TRY(cudaGetLastError());
        return HC_OK;
    }
    void *params[] = {&a};
    HC_CUDA_TRY(cudaLaunchCooperativeKernel((void *)bfs_persistent<kStats, kBlocks>, grid, block, params, 0, g->stream));
    return HC_OK;
}

// Blocks per team and teams for k sources on a graph of m edges (at most `room`
// teams), from sweeps of team sizes on Kronecker and uniform graphs of 20k to 128M edges.  A team is no
// smaller than sqrt(m) / 300 blocks: below that the sources run at a time
// outgrow the L2 (64 sources, 128M edges: 8 teams 7.6 ms, 12 teams 10.4 ms, 1
// team 12.9 ms; 16 sources, 8M edges: 16 teams 0.41 ms, 1 team 1.45 ms).  It is
// no larger than sqrt(m) / 19: above that a barrier and the queue's counters
// cost more than the blocks bring (one source, 20k edges: 8 blocks 79 us, 296
// blocks 97 us; 8M edges: 148 blocks 108 us, 296 blocks 120 us).  Between the
// two, as many teams as end the sources in the fewest rounds.
void bfs_teams(int64_t m, int resident, int k, int room, int *team, int *teams) {
    const double root = std::sqrt((double)std::max<int64_t>(m, 1));
    const int least = std::max(1, std::min(resident, (int)std::lround(root / 300.0)));
    const int most = std::max(1, std::min(resident, (int)std::lround(root / 19.0)));
    const int at_a_time = std::max(1, std::min({k, room, resident / least, kBfsLaunchSources}));
    const int rounds = (std::max(k, 1) + at_a_time - 1) / at_a_time;
    *teams = (std::max(k, 1) + rounds - 1) / rounds;
    *team = std::max(least, std::min(most, resident / *teams));
}

}  // namespace
}  // namespace hc

using namespace hc;

extern "C" hc_status hc_bfs(hc_graph *g, const int32_t *sources, int32_t num_sources, int32_t *depth_out,
                            int32_t *parent_out, const hc_bfs_opts *opts, hc_bfs_stats *stats) {
    clear_error();
    HC_TRY(activate(g));
    if (!sources || num_sources < 0) return fail(HC_ERR_INVALID_ARG, "hc_bfs: bad source list");
    hc_bfs_opts o{};
    if (opts) o = *opts;
    // Zero fields: the handle's tuned values, else Beamer's alpha = 15, beta = 18.
    if (o.alpha <= 0) o.alpha = g->tune.bfs_alpha > 0 ? g->tune.bfs_alpha : 15;
    if (o.beta <= 0) o.beta = g->tune.bfs_beta > 0 ? g->tune.bfs_beta : 18;
    // AUTO: the handle's per-level split table when the autotuner left one,
    // else its tuned variant.
    const bool by_level = o.bu_variant == HC_VARIANT_AUTO && g->tune.bfs_bu_split_levels > 0;
    if (o.bu_variant == HC_VARIANT_AUTO) o.bu_variant = (hc_variant)g->tune.bfs_bu_variant;
    if (o.direction < 0 || o.direction > 2) return fail(HC_ERR_INVALID_ARG, "hc_bfs: direction must be 0, 1 or 2");
    if (stats) std::memset(stats, 0, sizeof(*stats));

    std::vector<int32_t> src(num_sources);
    if (is_device_pointer(sources))
        HC_CUDA_TRY(cudaMemcpy(src.data(), sources, sizeof(int32_t) * num_sources, cudaMemcpyDefault));
    else
        std::copy(sources, sources + num_sources, src.begin());
    for (int32_t s : src)
        if (s < 0 || s >= g->N) return fail(HC_ERR_INVALID_ARG, "hc_bfs: source %d outside [0, %d)", s, g->N);
    HC_TRY(after_default_stream(g));

    const int64_t n = g->N;
    const int64_t W = (n + 31) / 32;
    const int64_t ntasks = max_expand_tasks(g->M, n);
    int sum_shift = 0;
    while (((W + (1ll << sum_shift) - 1) >> sum_shift) > (int64_t)kSumWords * 32) sum_shift++;
    const int sum_words = (int)((((W + (1ll << sum_shift) - 1) >> sum_shift) + 31) / 32);
    // Without per-run statistics or a trace the sources of a call run in one
    // launch, several at a time, and the host waits once, at the end (with
    // them, it runs one at a time and reads its control block after it).
    const bool per_run = (o.collect_stats && stats) || std::getenv("HC_TRACE");
    const bool dev_depth = is_device_pointer(depth_out);
    const bool dev_parent = is_device_pointer(parent_out);
    // Host outputs: staged on the device and copied while the next sources run.
    const bool host_depth = depth_out && !dev_depth, host_parent = parent_out && !dev_parent;
    const size_t bytes = [&] {
        auto up = [](size_t b) { return (b + 255) / 256 * 256; };
        return 4 * up(4 * (size_t)W) + 3 * up(4 * (size_t)sum_words) + 2 * up(4 * (size_t)n) +
               up(sizeof(int2) * (size_t)ntasks);
    }();
    int resident = 0;
    const bool wide = !per_run && num_sources >= 2 && g->M * num_sources >= kBfsWideWork;
    HC_TRY((o.collect_stats ? bfs_resident<true, 2>(g, &resident)
            : wide          ? bfs_resident<false, 3>(g, &resident)
                            : bfs_resident<false, 2>(g, &resident)));
    OutPipe pipe;
    int team = resident, teams = 1;
    const size_t fold_bytes = 256;
    auto reserve = [&]() -> hc_status {
        HC_TRY(g->ws_bfs.ensure(bytes * teams));
        HC_TRY(g->ws_ctl.ensure(std::max<size_t>(4096, fold_bytes + sizeof(BfsCtl) * (size_t)teams)));
        if (!depth_out) HC_TRY(g->ws_out0.ensure(4 * n * (size_t)teams));
        if (!parent_out) HC_TRY(g->ws_out1.ensure(4 * n * (size_t)teams));
        if (host_depth || host_parent) HC_TRY(pipe.init(g, 2, 4 * n, teams));
        return HC_OK;
    };
    if (per_run) {
        bfs_teams(g->M, resident, 1, 1, &team, &teams);
    } else {
        // Bytes of one source at a time: workspace, staging (both arrays, two
        // slots), scratch rows of outputs nobody asked for.
        const size_t each = bytes + 4 * (size_t)n * ((host_depth || host_parent ? 4 : 0) + !depth_out + !parent_out);
        bfs_teams(g->M, resident, num_sources, (int)std::min<size_t>(std::max<size_t>(kBfsTeamBytes / each, 1), 1 << 20),
                  &team, &teams);
    }
    hc_status reserved;
    {
        ReclaimScope nothing(nullptr, 0u);
        reserved = reserve();
    }
    if (reserved == HC_ERR_OOM) {  // no room: one source at a time, and what other calls left behind goes
        clear_error();
        if (teams > 1) {
            bfs_teams(g->M, resident, num_sources, 1, &team, &teams);
            g->ws_bfs.release();
            if (!depth_out) g->ws_out0.release();
            if (!parent_out) g->ws_out1.release();
            OutPipe::drop_staging(g);
        }
        ReclaimScope reclaim_scope(g, kKeepBfs);
        reserved = reserve();
    }
    HC_TRY(reserved);
    char *p = g->ws_bfs.as<char>();
    auto take = [&](size_t b) {
        char *r = p;
        p += (b + 255) / 256 * 256;
        return r;
    };
    BfsArgs a{};
    a.index = g->index.as<int64_t>();
    a.nbr = g->nbr.as<int32_t>();
    a.n = g->N;
    a.n_active = g->n_active;
    a.n_warp_rows = g->n_warp_rows;
    a.m = g->M;
    a.visited = (uint32_t *)take(4 * W);
    a.fb0 = (uint32_t *)take(4 * W);
    a.fb1 = (uint32_t *)take(4 * W);
    a.fb2 = (uint32_t *)take(4 * W);
    a.sb0 = (uint32_t *)take(4 * (size_t)sum_words);
    a.sb1 = (uint32_t *)take(4 * (size_t)sum_words);
    a.sb2 = (uint32_t *)take(4 * (size_t)sum_words);
    a.sum_shift = sum_shift;
    a.sum_words = sum_words;
    a.q0 = (int32_t *)take(4 * n);
    a.q1 = (int32_t *)take(4 * n);
    a.tasks = (int2 *)take(sizeof(int2) * ntasks);
    BfsFold *fold = g->ws_ctl.as<BfsFold>();
    a.ctl = reinterpret_cast<BfsCtl *>(g->ws_ctl.as<char>() + fold_bytes);
    a.fold = fold;
    a.team = team;
    a.team_stride = bytes;
    a.alpha = o.alpha;
    a.beta = o.beta;
    a.direction = o.direction;
    a.bu_variant = (int)o.bu_variant;
    a.max_levels = g->N + 1;
    a.bu_split_levels = 0;
    if (by_level) {
        a.bu_split_levels = std::min(g->tune.bfs_bu_split_levels, kBuSplitLevels);
        for (int k = 0; k < a.bu_split_levels; k++)
            a.bu_split[k] = std::max(0, std::min(g->tune.bfs_bu_split[k], g->n_active));
    }

    SuffixFill fill;  // declared after the pipe: its threads are joined first on any return
    if (host_depth || host_parent) {
        const int64_t n_copy = g->degree_sorted ? (int64_t)g->n_active : n;
        if (n_copy < n) {
            pipe.copy_bytes = sizeof(int32_t) * (size_t)n_copy;
            fill.start(host_depth ? depth_out : nullptr, host_parent ? parent_out : nullptr, src, n, n_copy);
        }
    }

    double total_ms = 0;
    if (!per_run) {
        BfsFold *h_fold = nullptr;
        HC_TRY(ctl_slot(g, 0, (void **)&h_fold, (void **)&a.fold_host));
        { bfs_clear<<<1, 256, 0, g->stream>>>(a.ctl, teams, fold); ::hc::count_launch(); }
        HC_CUDA_TRY(cudaGetLastError());
        HC_CUDA_TRY(cudaEventRecord(g->ev_start, g->stream));
        // Host outputs are copied a launch at a time, so a launch runs one source per team.
        const bool staged = host_depth || host_parent;
        const int per_launch = staged ? teams : kBfsLaunchSources;
        a.depth_stride = depth_out ? n : 0;
        a.parent_stride = parent_out ? n : 0;
        for (int32_t i = 0, l = 0; i < num_sources; i += per_launch, l++) {
            a.nsrc = std::min(per_launch, num_sources - i);
            std::copy(src.begin() + i, src.begin() + i + a.nsrc, a.src);
            int32_t *stage[2] = {nullptr, nullptr};
            if (staged) HC_TRY(pipe.acquire(l, stage));
            a.depth = dev_depth ? depth_out + (size_t)i * n : host_depth ? stage[0] : g->ws_out0.as<int32_t>();
            a.parent = dev_parent ? parent_out + (size_t)i * n : host_parent ? stage[1] : g->ws_out1.as<int32_t>();
            HC_TRY((wide ? launch_bfs<false, 3>(g, a, std::min(teams, a.nsrc))
                         : launch_bfs<false, 2>(g, a, std::min(teams, a.nsrc))));
            if (staged) {
                void *dst[2] = {host_depth ? (void *)(depth_out + (size_t)i * n) : nullptr,
                                host_parent ? (void *)(parent_out + (size_t)i * n) : nullptr};
                HC_TRY(pipe.release(l, dst, a.nsrc));
            }
        }
        HC_CUDA_TRY(cudaEventRecord(g->ev_stop, g->stream));
        HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
        if (num_sources > 0) {
            BfsFold f;
            std::memcpy(&f, h_fold, sizeof(f));
            if (f.err) return fail((hc_status)f.err, "hc_bfs: device run from source %d ended with status %d",
                                   f.err_src, f.err);
            if (stats) {
                stats->levels = f.levels;
                stats->td_levels = f.td_levels;
                stats->bu_levels = f.bu_levels;
            }
        }
        float ms = 0;
        HC_CUDA_TRY(cudaEventElapsedTime(&ms, g->ev_start, g->ev_stop));
        total_ms = ms;
    }
    for (int32_t i = 0; per_run && i < num_sources; i++) {
        a.nsrc = 1;
        a.src[0] = src[i];
        int32_t *stage[2] = {nullptr, nullptr};
        if (host_depth || host_parent) HC_TRY(pipe.acquire(i, stage));
        a.depth = dev_depth ? depth_out + (size_t)i * n : host_depth ? stage[0] : g->ws_out0.as<int32_t>();
        a.parent = dev_parent ? parent_out + (size_t)i * n : host_parent ? stage[1] : g->ws_out1.as<int32_t>();
        { bfs_clear<<<1, 256, 0, g->stream>>>(a.ctl, 1, fold); ::hc::count_launch(); }
        HC_CUDA_TRY(cudaEventRecord(g->ev_start, g->stream));
        HC_TRY((o.collect_stats ? launch_bfs<true, 2>(g, a, 1) : launch_bfs<false, 2>(g, a, 1)));
        HC_CUDA_TRY(cudaEventRecord(g->ev_stop, g->stream));
        if (host_depth || host_parent) {
            void *dst[2] = {host_depth ? (void *)(depth_out + (size_t)i * n) : nullptr,
                            host_parent ? (void *)(parent_out + (size_t)i * n) : nullptr};
            HC_TRY(pipe.release(i, dst, 1));
        }
        static_assert(sizeof(BfsCtl) + 256 + 64 <= 2560 && sizeof(BfsCtl) <= kCtlSlotBytes, "BfsCtl exceeds a control-read slot");
        BfsCtl c;
        const void *h_ctl = nullptr, *h_cnt = nullptr;
        HC_TRY(ctl_read(g, a.ctl, sizeof(c), 0, &h_ctl));
        if (o.collect_stats && stats) {
            unsigned long long *cnt = (unsigned long long *)(g->ws_ctl.as<char>() + 3072);
            HC_TRY(ctl_zero(g, cnt, 8));
            { count_reached<<<g->sm_count * 4, 256, 0, g->stream>>>(a.depth, g->N, cnt); ::hc::count_launch(); }
            HC_TRY(ctl_read(g, cnt, 8, 1, &h_cnt));
        }
        HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
        std::memcpy(&c, h_ctl, sizeof(c));
        if (h_cnt) {
            unsigned long long reached = 0;
            std::memcpy(&reached, h_cnt, 8);
            stats->reached += (int32_t)reached;
        }
        if (c.gs.err) return fail((hc_status)c.gs.err, "hc_bfs: device run from source %d ended with status %d",
                                  src[i], c.gs.err);
        float ms = 0;
        HC_CUDA_TRY(cudaEventElapsedTime(&ms, g->ev_start, g->ev_stop));
        total_ms += ms;
        if (stats) {
            stats->levels = std::max(stats->levels, c.levels);
            stats->td_levels += c.td_levels;
            stats->bu_levels += c.bu_levels;
            stats->vertices_scanned += (int64_t)c.vscan;
            stats->edges_scanned += (int64_t)c.escan;
        }
        if (std::getenv("HC_TRACE")) {
            const int nl = std::min(c.levels, kTraceLevels);
            std::fprintf(stderr, "[hc bfs] src %d: %d levels, %.1f us\n", src[i], c.levels, ms * 1e3);
            for (int l = 0; l < nl; l++)
                std::fprintf(stderr, "[hc bfs]   L%-3d %s nf=%-9d %8.1f us\n", l, c.trace[l].mode == 1 ? "TD" : "BU",
                             c.trace[l].nf, (c.trace[l + 1].t_ns - c.trace[l].t_ns) * 1e-3);
        }
    }
    if (host_depth || host_parent) HC_TRY(pipe.finish());
    if (stats) {
        stats->ms = total_ms;
        // Streamed bytes: 16 B offsets per scanned vertex, 4 B per scanned edge,
        // 4 B per discovered vertex, and for bottom-up levels two bitmap sweeps.
        stats->bytes_model = 16.0 * (double)stats->vertices_scanned + 4.0 * (double)stats->edges_scanned +
                             4.0 * (double)stats->reached +
                             2.0 * ((double)g->N / 8.0) * (double)stats->bu_levels;
    }
    return HC_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free BFS.
//
// Some callers cannot allocate device memory at the moment they need a BFS:
// code running inside another framework's caching allocator or memory pool
// (where a cudaMalloc would bypass or fragment the pool), paths that must not
// trigger the implicit device synchronisation a cudaMalloc / cudaFree can
// cause, and hosts that pre-plan every byte of HBM.  hc_bfs_noalloc serves
// them: the caller passes the graph and the outputs in its own device memory,
// and the working set (visited and frontier bitmaps, the two queues, the
// long-row task list and the control block) lives in one fixed file-scope
// device array, g_bfs_scratch, sized for graphs of up to kNoAllocMaxNodes
// vertices and kNoAllocMaxEdges edges (about 13 MB, held by every GPU that
// loads this library until the process exits).  It runs the same persistent
// direction-optimising kernel as hc_bfs.
namespace hc {
namespace {

constexpr int32_t kNoAllocMaxNodes = 1 << 20;
constexpr int64_t kNoAllocMaxEdges = 1ll << 24;
constexpr size_t na_align(size_t b) { return (b + 255) / 256 * 256; }
constexpr size_t kNaWords = (size_t)kNoAllocMaxNodes / 32;
constexpr size_t kNaTasks = (size_t)(kNoAllocMaxEdges / kTaskEdges + kNoAllocMaxEdges / (kSmallDeg + 1) + 64);
// Frontier summaries: one bit per bitmap word (kNaWords <= 32 * kSumWords).
constexpr size_t kNaSumWords = (kNaWords + 31) / 32;
static_assert(kNaWords <= (size_t)kSumWords * 32, "summary of the fixed-size bitmaps needs a shift");
constexpr size_t kNoAllocBytes = na_align(sizeof(BfsCtl)) + na_align(sizeof(BfsFold)) + na_align(sizeof(int)) + 4 * na_align(4 * kNaWords) +
                                 3 * na_align(4 * kNaSumWords) + 2 * na_align(4 * (size_t)kNoAllocMaxNodes) +
                                 na_align(sizeof(int2) * kNaTasks);

static __device__ __align__(256) unsigned char g_bfs_scratch[kNoAllocBytes];

// In host code g_bfs_scratch names a host-side shadow, not device memory: the
// device address comes from cudaGetSymbolAddress, once per device, with that
// device current, and is cached here.
constexpr int kNaMaxDevices = 64;
std::mutex g_na_mutex;
void *g_na_addr[kNaMaxDevices] = {};

hc_status noalloc_scratch(int dev, unsigned char **out) {
    if (dev < 0 || dev >= kNaMaxDevices) return fail(HC_ERR_UNSUPPORTED, "hc_bfs_noalloc: device %d out of range", dev);
    std::lock_guard<std::mutex> lock(g_na_mutex);
    if (!g_na_addr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_bfs_scratch);
        if (e != cudaSuccess || !p) {
            cudaGetLastError();
            return fail(HC_ERR_CUDA, "hc_bfs_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
        }
        g_na_addr[dev] = p;
    }
    *out = static_cast<unsigned char *>(g_na_addr[dev]);
    return HC_OK;
}

bool on_device(const void *p, int dev) {
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return (attr.type == cudaMemoryTypeDevice || attr.type == cudaMemoryTypeManaged) && attr.device == dev;
}

}  // namespace
}  // namespace hc

extern "C" hc_status hc_bfs_noalloc(const int64_t *index, const int32_t *neighbors, int32_t num_nodes,
                                    int64_t num_edges, int32_t source, int32_t *depth_out, int32_t *parent_out,
                                    void *stream) {
    using namespace hc;
    clear_error();
    if (num_nodes < 1 || num_nodes > kNoAllocMaxNodes || num_edges < 0 || num_edges > kNoAllocMaxEdges)
        return fail(HC_ERR_INVALID_ARG,
                    "hc_bfs_noalloc: graph of %d vertices / %lld edges exceeds the fixed working set "
                    "(at most %d vertices and %lld edges); use hc_bfs",
                    num_nodes, (long long)num_edges, kNoAllocMaxNodes, (long long)kNoAllocMaxEdges);
    if (source < 0 || source >= num_nodes)
        return fail(HC_ERR_INVALID_ARG, "hc_bfs_noalloc: source %d outside [0, %d)", source, num_nodes);
    int dev = 0;
    HC_CUDA_TRY(cudaGetDevice(&dev));
    if (!index || !neighbors || !depth_out || !parent_out || !on_device(index, dev) ||
        (num_edges > 0 && !on_device(neighbors, dev)) || !on_device(depth_out, dev) || !on_device(parent_out, dev))
        return fail(HC_ERR_INVALID_ARG,
                    "hc_bfs_noalloc: index, neighbors, depth_out and parent_out must be device memory of the "
                    "current device");
    unsigned char *base = nullptr;
    HC_TRY(noalloc_scratch(dev, &base));
    int sms = 0, bps = 0;
    HC_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    HC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, (bfs_persistent<false, 2>), kBfsThreads, 0));
    if (bps < 1) return fail(HC_ERR_CUDA, "hc_bfs_noalloc: BFS kernel cannot be resident");

    unsigned char *p = base;
    auto take = [&](size_t b) {
        unsigned char *r = p;
        p += na_align(b);
        return r;
    };
    BfsArgs a{};
    a.ctl = reinterpret_cast<BfsCtl *>(take(sizeof(BfsCtl)));
    a.fold = reinterpret_cast<BfsFold *>(take(sizeof(BfsFold)));
    int *check_flag = reinterpret_cast<int *>(take(sizeof(int)));
    a.visited = reinterpret_cast<uint32_t *>(take(4 * kNaWords));
    a.fb0 = reinterpret_cast<uint32_t *>(take(4 * kNaWords));
    a.fb1 = reinterpret_cast<uint32_t *>(take(4 * kNaWords));
    a.fb2 = reinterpret_cast<uint32_t *>(take(4 * kNaWords));
    a.sb0 = reinterpret_cast<uint32_t *>(take(4 * kNaSumWords));
    a.sb1 = reinterpret_cast<uint32_t *>(take(4 * kNaSumWords));
    a.sb2 = reinterpret_cast<uint32_t *>(take(4 * kNaSumWords));
    a.sum_shift = 0;
    a.sum_words = (int)((((num_nodes + 31) / 32) + 31) / 32);
    a.q0 = reinterpret_cast<int32_t *>(take(4 * (size_t)kNoAllocMaxNodes));
    a.q1 = reinterpret_cast<int32_t *>(take(4 * (size_t)kNoAllocMaxNodes));
    a.tasks = reinterpret_cast<int2 *>(take(sizeof(int2) * kNaTasks));
    a.index = index;
    a.nbr = neighbors;
    a.n = num_nodes;
    a.n_active = num_nodes;  // no degree analysis here: scan every vertex
    a.n_warp_rows = 0;
    a.m = num_edges;
    a.depth = depth_out;
    a.parent = parent_out;
    a.nsrc = 1;
    a.src[0] = source;
    // The blocks that suit the graph's size: all that fit made every barrier dearer
    // (Kronecker scale 16: 148 us with 296 blocks, 136 us so; scale 10: 110 and 91).
    int teams = 1;
    bfs_teams(num_edges, sms * bps, 1, 1, &a.team, &teams);
    a.alpha = 15;
    a.beta = 18;
    a.direction = 0;
    a.bu_variant = HC_VARIANT_THREAD;
    a.max_levels = num_nodes + 1;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    // The caller's CSR is checked before the traversal reads it (offsets
    // rising from 0 to num_edges, neighbour ids in [0, num_nodes)); the check
    // writes its flag into the fixed array too.
    HC_TRY(csr_check_async(index, neighbors, 1, num_nodes, num_edges, check_flag, sms, s));
    int bad = 0;
    HC_CUDA_TRY(cudaMemcpyAsync(&bad, check_flag, sizeof(int), cudaMemcpyDeviceToHost, s));
    HC_CUDA_TRY(cudaStreamSynchronize(s));
    if (bad & 1) return fail(HC_ERR_INVALID_ARG, "hc_bfs_noalloc: offsets must rise from 0 to num_edges");
    if (bad & 2) return fail(HC_ERR_INVALID_ARG, "hc_bfs_noalloc: neighbour id outside [0, num_nodes)");
    // The array keeps the previous call's contents; the control block must
    // start at zero (the kernel initialises everything else it reads).
    HC_CUDA_TRY(cudaMemsetAsync(a.ctl, 0, sizeof(BfsCtl), s));
    HC_CUDA_TRY(cudaMemsetAsync(a.fold, 0, sizeof(BfsFold), s));
    void *params[] = {&a};
    ::hc::count_launch();
    HC_CUDA_TRY(cudaLaunchCooperativeKernel((void *)bfs_persistent<false, 2>, dim3(a.team), dim3(kBfsThreads), params, 0,
                                            s));
    int err = 0;
    HC_CUDA_TRY(cudaMemcpyAsync(&err, &a.ctl->gs.err, sizeof(int), cudaMemcpyDeviceToHost, s));
    HC_CUDA_TRY(cudaStreamSynchronize(s));
    if (err) return fail((hc_status)err, "hc_bfs_noalloc: device run ended with status %d", err);
    return HC_OK;
}
