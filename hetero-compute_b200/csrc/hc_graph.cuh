// The device graph handle shared by every kernel translation unit.
#pragma once

#include "hc_device.cuh"

namespace hc {
// Row plans of the PageRank sweeps and the SSSP pull sweep, built once per graph
// from the offsets of the rows with edges:
//   stream groups  32 consecutive rows, one warp
//   long rows      one warp per row
//   hub rows       more than two chunks of edges, cut into tasks of one chunk
// A long row, a task or a PageRank stream group is a serial chain of its warp's
// 128-edge steps (about a microsecond each), so on a small graph, whose sweep is
// no more than a few of those, they are short; on a large one they are long, as
// a task ends with a fence and a counter and a warp per short row wastes lanes.
//   chunk          M / 4096 edges rounded down to a power of two, in [256, 2048]
//   stream group   at most M / 8192 edges, rounded likewise, in [256, 2048]; at
//                  least 1024 when more than kMaxSingle1 rows in groups of up to
//                  1024 edges would be single otherwise, and 2048 when more than
//                  kMaxSingle2 in groups of 1024 to 2048 would: a warp a row of 16
//                  to 64 edges is then many rounds of mostly idle lanes, where a
//                  group is a few (uniform, ms a solve: 2^18 vertices, rows of 16,
//                  0.57 with the limit at 512, 0.32 at 1024; rows of 48, 0.47 at
//                  1024, 0.42 at 2048; 2^19, rows of 32, 0.69 and 0.65; but 2^14,
//                  rows of 32, 0.10 at 256, 0.18 at 1024)
// The SSSP pull (a lane per row) and the adjoint's conjugate gradients use the
// plan of 2048 edges at every size.  The gradient of a weight is a difference of
// two nearly equal numbers, so another order of the sums in the solve would show
// in its last digits.
constexpr int kMinChunk = 256;
constexpr int kMaxChunk = 2048;
constexpr int64_t kMaxSingle1 = 40000, kMaxSingle2 = 200000;
// Batched SSSP keeps 16-bit distances when no weight exceeds this.
constexpr int32_t kMsspNarrowMaxW = 0x0FFF;

struct HubInfo {
    int32_t row;
    int32_t first;  // first partial slot
    int32_t nchunks;
    int32_t pad;
};

struct PrPlanDev {
    const int32_t *stream;  // group ids (rows 32*id .. 32*id+31)
    const int32_t *longrows;
    const int2 *tasks;      // (hub index, chunk)
    const HubInfo *hubs;
    int n_stream, n_long, n_tasks, n_hub;
    int chunk;              // edges per hub task
};

// Row plan of the multi-column PageRank sweeps:
//   tasks   chunks of rows longer than one chunk (hub index, chunk)
//   longs   rows of more than kSpmmLong edges, a warp each
//   the rest, `rows` consecutive rows to a warp: as many as make about a warp's
//   work of each (at most kSpmmRows)
constexpr int kSpmmLong = 64;
constexpr int kSpmmRows = 8;
struct SpmmPlanDev {
    const int32_t *longs;
    const int2 *tasks;
    const HubInfo *hubs;
    int n_long, n_tasks, n_hub, chunk, rows;
};
}  // namespace hc

// Layout in HBM (one allocation per array, 256-byte aligned by cudaMalloc):
//   index     int64[N+1]                 row offsets
//   nbr       int32[M + kNbrPad]         neighbours; the pad keeps 128-bit
//                                        loads of a row's last aligned window
//                                        inside the allocation
//   wgt       int32/f32[M + kNbrPad]     weights, same slots as nbr (SoA)
// Derived arrays (inverse degrees, transposed weights, PageRank row plan)
// and per-algorithm workspaces are built lazily and kept with the handle.
struct hc_graph {
    int device = 0;
    int sm_count = 0;
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev_start = nullptr, ev_stop = nullptr;
    cudaEvent_t ev_default = nullptr;  // after_default_stream

    int32_t N = 0;
    int64_t M = 0;
    int32_t n_active = 0;      // vertices [0, n_active) may have edges
    int32_t n_warp_rows = 0;   // degree-sorted: [0, n_warp_rows) have degree >= 32 (32-aligned)
    int32_t degree_sorted = 0;
    int32_t rows_sorted = 0;      // every row strictly increasing
    int32_t max_degree = 0;
    hc_wtype wtype = HC_W_NONE;

    hc::DevBuf index, nbr, wgt;

    // lazily built derived data
    hc::DevBuf inv_deg;        // f32[N]: 1/deg (0 for isolated)
    hc::DevBuf inv_wsum;       // f32[N]: 1/sum_k w_uk (weighted PageRank)
    hc::DevBuf wtn;            // f32[M]: slot (v,i) holds w_{u v}/sum_k w_uk, u = nbr[v][i]
    hc::DevBuf wf32;           // f32[M]: int32 weights as floats (weighted PageRank on int32 graphs)
    hc::DevBuf pr_plan;        // row plan (device arrays; empty where base_plan is the same)
    hc::PrPlanDev pr_view{};   // host copy of its pointers and counts
    int32_t pr_partial_slots = 0;
    hc::DevBuf base_plan;      // the plan of 2048 edges (SSSP pull, adjoint)
    hc::PrPlanDev base_view{};
    int32_t base_partial_slots = 0;
    hc::DevBuf pr_plan_huge_rows;
    hc::DevBuf spmm_plan;          // multi-column row plan (device arrays)
    hc::SpmmPlanDev spmm_view{};
    int32_t spmm_partial_slots = 0;
    // level schedule of the reference-order PageRank sweep (hc_pr_ordered.cu):
    // order[N] | level_off[levels + 1] | level_long[levels] | deg as fp32 [N];
    // levels -1 = not built
    hc::DevBuf pr_ord;
    int32_t pr_ord_levels = -1;

    // symmetry of the PageRank transition (-1: not checked yet)
    int pr_sym_struct = -1;    // every edge u->v has v->u (rows sorted)
    int pr_sym_w = -1;         // ... with the same weight

    // weight statistics, computed once
    int wstats_done = 0;
    int w_negative = 0;
    int32_t w_max = 0;         // largest weight (0 when none is positive)
    double w_mean = 0.0;
    int w_symmetric = 0;       // w(u->v) == w(v->u) for every edge (rows sorted)
    // SSSP pull sweeps: int2[M + 64] (neighbour, weight) pairs of each row in
    // weight-bucket order (stable), built on the first pull-enabled call
    hc::DevBuf sssp_adj;
    int sssp_adj_ready = 0;

    // batched-BFS hub plan (rows above its split threshold, (row, chunk) tasks)
    hc::DevBuf ws_plan_ms;
    int32_t ms_hubs = -1, ms_tasks = 0;
    // batched-SSSP pull plan: (row, chunk) tasks of the rows above its chunk size
    hc::DevBuf ws_plan_mssp;
    int32_t mssp_tasks = -1;
    int32_t mssp_hub_rows = -1;  // degree-sorted: the row prefix holding half the edges

    // autotuned launch parameters (zero fields: built-in defaults)
    hc_tuning tune{};

    // host-output pipeline (per-source results copied while the next computes)
    hc::DevBuf ws_stage[2][2];  // [slot][array]
    cudaStream_t copy_stream = nullptr;
    cudaEvent_t ev_ready[2] = {nullptr, nullptr}, ev_done[2] = {nullptr, nullptr};

    // workspaces
    hc::DevBuf ws_bfs, ws_sssp, ws_pr, ws_batch, ws_out0, ws_out1, ws_ctl, ws_src;
    hc::PinnedBuf pinned;
    // mapped pinned slots for control-block reads (ctl_read), and their device address
    void *ctl_host = nullptr;
    void *ctl_host_dev = nullptr;

    int bfs_grid = 0, sssp_grid = 0;
    int64_t bytes_held() const;
};

namespace hc {
// Make the handle's device current; returns HC_ERR_CUDA on failure.
hc_status activate(hc_graph *g);
// Orders the handle's stream after what the caller has queued on the legacy
// default stream so far.  The handle's own stream does not wait for it by
// itself, and a caller's output may be memory that a kernel queued there still
// uses (a tensor that an allocator handed on in the order of that stream).
hc_status after_default_stream(hc_graph *g);
// Builds inv_deg (and, for weighted graphs, inv_wsum / wtn) if missing.
hc_status ensure_pr_derived(hc_graph *g, bool weighted);
// Outputs bound for host memory, double-buffered: launch i of a call writes the
// rows of its sources to staging slot i & 1 on the compute stream, and their copy
// to the caller runs on a copy stream while the next launch computes (overlapped
// when the destination is pinned).  Before a slot is written again the compute
// stream waits for that slot's previous copy.
struct OutPipe {
    hc_graph *g = nullptr;
    int narr = 0;
    int pend_rows = 1;
    size_t bytes = 0;       // of one row
    size_t copy_bytes = 0;  // bytes of each row copied out (init: all; a caller may shorten it)
    bool pending = false;
    int pend_slot = 0;
    void *pend_dst[2] = {nullptr, nullptr};
    // Staging and events for `arrays` outputs of up to `rows` rows of `each` bytes.
    hc_status init(hc_graph *graph, int arrays, size_t each, int rows = 1);
    // Staging buffers of launch i (after the wait for the slot's last copy).
    hc_status acquire(int i, int32_t **bufs);
    // Launch i's results are complete on the compute stream once what is queued
    // there has run; copy `rows` consecutive rows of each array to dst[] (null
    // entries are skipped).  The copy is issued by the next acquire or by finish.
    hc_status release(int i, void *const *dst, int rows = 1);
    hc_status flush();
    // Releases the staging (no copy in flight).
    static void drop_staging(hc_graph *g);
    hc_status finish();
};

// A handle for an N-vertex, M-edge graph on `device` with its CSR arrays
// allocated (neighbour and weight pads zeroed) and not yet filled.
hc_status graph_alloc(int32_t num_nodes, int64_t num_edges, hc_wtype wtype, int32_t device, hc_graph **out);
// Validates the filled CSR (offsets 0..M non-decreasing, ids in [0, N)) and
// records its degree analysis; `who` names the caller in error messages.
hc_status graph_finish(hc_graph *g, const char *who);
// Checks a caller's CSR on the device (offsets rising from 0 to m, neighbour
// ids in [0, n); `stride` 2 for interleaved {id, weight} edges): clears
// *flag_dev, then sets bit 0 (offsets) / bit 1 (ids) on a violation.
hc_status csr_check_async(const int64_t *index, const int32_t *nbr, int stride, int32_t n, int64_t m, int *flag_dev,
                          int sm_count, cudaStream_t s);
// Whether the PageRank transition is a reversible walk (symmetric structure,
// and symmetric weights when `weighted`), checked once per graph.
hc_status ensure_pr_symmetry(hc_graph *g, bool weighted, bool *symmetric);
// Whether every edge u->v has a reverse v->u (as multisets), and whether the
// reverse carries the same weight bits (`wbits` may be null).
hc_status edge_symmetry(hc_graph *g, const uint32_t *wbits, bool *structure, bool *weights);
// The edge weights as fp32 for weighted PageRank: the weight array itself
// (fp32 graphs) or its converted copy (int32 graphs, built by ensure_pr_derived).
const float *pr_weights(const hc_graph *g);
// Builds those of the row plans that are missing: PageRank's (g->pr_view,
// g->pr_partial_slots), the plan of 2048 edges (g->base_view,
// g->base_partial_slots), the multi-column one (g->spmm_view,
// g->spmm_partial_slots).
enum : unsigned { kPlanPr = 1u, kPlanBase = 2u, kPlanSpmm = 4u };
hc_status ensure_plans(hc_graph *g, unsigned which);
// Whether a batched loop left to choose becomes a CUDA graph at once: on a graph of
// at most 8 edges a row, road-like, it runs hundreds of epochs (33 sources on a 60 x
// 70 grid: batched SSSP 3.0 ms with a graph, 3.6 with launches first, BFS 2.5 and
// 2.6).
inline bool long_loop(const hc_graph *g) { return g->M <= 8ll * g->n_active; }
// Computes w_negative, w_max, w_mean and w_symmetric once (int32 weights).
hc_status ensure_weight_stats(hc_graph *g);
// Per-run control traffic kept off the copy engines.  A host-output call
// keeps a large copy on the copy stream while the next source runs; a small
// cudaMemcpyAsync or cudaMemsetAsync of a control block on the compute stream
// can queue on the same engine behind it and serialise the two.  ctl_zero
// clears device words with a one-block kernel on the graph's stream; ctl_read
// has a one-block kernel write `bytes` (at most kCtlSlotBytes) of device memory
// into mapped pinned slot `slot` (0..kCtlSlots-1) and returns its host address,
// valid once the stream has been synchronised.
constexpr size_t kCtlSlotBytes = 4096;
constexpr int kCtlSlots = 4;
hc_status ctl_zero(hc_graph *g, void *dev, size_t bytes);
hc_status ctl_read(hc_graph *g, const void *dev, size_t bytes, int slot, const void **host);
// Slot `slot` itself: its host address, and the device address of the same
// memory for a kernel that writes its result there.
hc_status ctl_slot(hc_graph *g, int slot, void **host, void **dev);
// Device memory pressure.  Derived arrays that can be built again (the
// pull sweeps' pair array, the reference-order schedule, the weighted
// PageRank arrays), the batched workspace and the BFS and SSSP workspaces and
// staging are released, when an allocation fails, unless the running call
// needs them; the allocation is then tried once more.  A call states what it
// needs for its lifetime.  Workspaces for several sources at a time are asked
// for under a scope of no graph (nothing is released for them); when they
// cannot be had, those of one source are, under the call's own scope.
enum : unsigned { kKeepAdj = 1u, kKeepPrOrd = 2u, kKeepPrWeighted = 4u, kKeepBatch = 8u, kKeepSssp = 16u, kKeepBfs = 32u };
struct ReclaimScope {
    ReclaimScope(hc_graph *g, unsigned keep);
    ~ReclaimScope();
    ReclaimScope(const ReclaimScope &) = delete;
    ReclaimScope &operator=(const ReclaimScope &) = delete;
    hc_graph *prev_g;
    unsigned prev_keep;
};
// The pull sweeps' weight-ordered (neighbour, weight) pairs (hc_graph::sssp_adj),
// after the weight statistics; bucket(w) = w >> weight_shift(w_max) < 256.
hc_status ensure_weight_order(hc_graph *g);
int weight_shift(int32_t w_max);
}  // namespace hc
