// Pull PageRank: forward, adjoint and multi-column (personalised) forms.
//
// Reference path: pr_pull_gpu (src/kernels/gpu/pr.cuh:42-118) with the
// in-place epochs of src/kernels/gpu/pr.cuh:140-318: score[v] = (1-d)/N +
// d * sum_u score[u]/deg[u], reading an 8-byte wnode_t and an 8-byte int64
// degree per edge.  Here each iteration is a Jacobi pull over a gathered
// vector that already carries the 1/deg factor (4-byte neighbour stream +
// 4-byte gather), with the L1 / per-vertex residual reduced in the same pass.
//
// Work plan (built once per graph from the row offsets, see hc_graph.cuh):
//   stream groups  32 consecutive rows of few edges in total; one warp streams
//                  the whole edge range coalesced and reduces it segment by
//                  segment (CSR-stream, Greathouse & Daga 2014)
//   long rows      one warp per row, 128-bit neighbour loads
//   hub rows       cut into chunks; each chunk's warp writes a partial, the last
//                  one to finish sums the partials in chunk order
//                  (deterministic) and finalises
// Vertices without edges keep (1-d) t_v, written once before the iterations.
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>
#include <memory>
#include <new>
#include <vector>

#include "hc_graph.cuh"

namespace hc {
namespace {

constexpr int kPrThreads = 256;
constexpr int kPrBlocks = 6;  // per SM: the gathers want warps more than registers
constexpr int kMaxIterSlots = 4096;

// Grid barrier and per-iteration sums of one solve: a slot per iteration, all
// zero at the start, so that no block resets a sum another still reads (past
// kMaxIterSlots iterations they come round, cleared two iterations ahead).
struct IterSlot {
    double l1;       // Jacobi: sum |change|; conjugate gradients: p . q
    double rz, z1;   // conjugate gradients: r . z, sum |z|
    int changed, pad;
};
struct IterState {
    GridSync gs;
    int done, blocks_done;   // sweeps launched one by one
    int pause_after, pad;    // 1 + the iteration after which the launch ends (see past_run_limit)
    IterSlot slot[kMaxIterSlots];
};
// What a solve reports, in mapped host memory.  done: 1 converged, 2 stopped, 0
// paused at the run limit: another launch goes on from iteration `iters`.
struct SolveOut {
    int err, iters, done, changed;
    double l1, omega;
};

// One pull sweep: out[v] = base_v + d * rs_v * sum_{e in row v} ew_e * gin[nbr_e].
struct SweepArgs {
    const int64_t *index;
    const int32_t *nbr;
    const float *ew;        // per-slot edge weight (kEW)
    const float *basev;     // per-vertex base (kBaseVec), already scaled by (1-d)
    float base_scalar;
    float d;
    const float *rs;        // per-row scale (kRS)
    const float *ps;        // gather-out scale (kPS)
    float *x[2], *g[2];     // iterates and their gather vectors (g == x without kPS)
    float *partials;
    unsigned *hub_count;
    IterState *st;
    SolveOut *out;
    float *final_x;         // the result is copied here too (null: not)
    float cheb_rho;         // > 0: Chebyshev weights (0: plain Jacobi)
    float tol_l1, eps;
    int max_iters;
    int first_iter;         // where this launch goes on, and the Chebyshev weight it left off with
    double first_omega;
    int32_t n, n_active;
};
// The vectors of one sweep.  They are written by other blocks of the same
// launch, so they are read through L1 by coherent loads; the grid barrier's
// acquire drops what L1 holds of the last sweep's.
struct SweepIter {
    const float *gin;       // gathered vector
    const float *xin;       // previous iterate (residual)
    float *xout;
    float *gout;            // gather vector for the next sweep (kPS) -- else == xout
    float omega;            // Chebyshev weight of this iteration (1: plain Jacobi)
};

template <bool kEW, bool kRS, bool kPS, bool kBaseVec, bool kCG = false>
__device__ __forceinline__ void finish_row(const SweepArgs &a, const SweepIter &v, int32_t r, float sum, float &l1, int &chg) {
    if constexpr (kCG) {
        // Conjugate-gradient product (gin = p): xout = (S p)_r, and
        // p_r q_r with q = s p - d S p summed where the residual goes.
        const float pr = v.gin[r];
        const float rsr = a.rs[r];
        const float sr = rsr > 0.f ? 1.0f / rsr : 0.f;
        v.xout[r] = sum;
        l1 += pr * (sr * pr - a.d * sum);
        return;
    }
    const float base = kBaseVec ? a.basev[r] : a.base_scalar;
    const float scale = kRS ? a.rs[r] : 1.0f;
    float nv = base + a.d * (scale * sum);
    const float ov = v.xin[r];
    // The residual |J(x_k) - x_k| of the fixed-point equation: the change of
    // a plain Jacobi sweep, and the stopping rule of both iterations.
    const float dl = fabsf(nv - ov);
    // Chebyshev semi-iteration: x_{k+1} = omega (J(x_k) - x_{k-1}) + x_{k-1};
    // x_{k-1} is what the output buffer still holds.
    if (v.omega != 1.0f) {
        const float prev = v.xout[r];
        nv = v.omega * (nv - prev) + prev;
    }
    v.xout[r] = nv;
    if (kPS) v.gout[r] = nv * a.ps[r];
    l1 += dl;
    chg += dl > a.eps;
}

template <bool kEW>
__device__ __forceinline__ float edge_val(const SweepArgs &a, const SweepIter &v, int64_t e) {
    const float g = __ldca(v.gin + __ldg(a.nbr + e));
    return kEW ? g * __ldg(a.ew + e) : g;
}

// One sweep over every row with edges, by the whole grid; l1 and chg receive
// this thread's share of the residual.
template <bool kEW, bool kRS, bool kPS, bool kBaseVec, bool kCG = false>
__device__ __forceinline__ void sweep_rows(const SweepArgs &a, const PrPlanDev &plan, const SweepIter &it,
                                           float (*s_acc)[32], float &l1, int &chg) {
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    l1 = 0.f;
    chg = 0;
    const int total_items = plan.n_tasks + plan.n_long + plan.n_stream;

    for (int item = gwarp; item < total_items; item += nwarps) {
        if (item < plan.n_tasks) {
            // Chunk of a hub row.
            const int2 tk = plan.tasks[item];
            const HubInfo h = plan.hubs[tk.x];
            const int64_t rb = a.index[h.row], re = a.index[h.row + 1];
            const int64_t b = rb + (int64_t)tk.y * plan.chunk;
            const int64_t e = min(re, b + (int64_t)plan.chunk);
            // Four independent partial sums keep four gathers in flight.
            float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
            int64_t i = b + lane;
            for (; i + 96 < e; i += 128) {
                s0 += edge_val<kEW>(a, it, i);
                s1 += edge_val<kEW>(a, it, i + 32);
                s2 += edge_val<kEW>(a, it, i + 64);
                s3 += edge_val<kEW>(a, it, i + 96);
            }
            for (; i < e; i += 32) s0 += edge_val<kEW>(a, it, i);
            float s = warp_sum((s0 + s1) + (s2 + s3));
            int last = 0;
            if (lane == 0) {
                a.partials[h.first + tk.y] = s;
                __threadfence();
                last = atomicAdd(a.hub_count + tk.x, 1u) == (unsigned)(h.nchunks - 1);
            }
            last = __shfl_sync(kFull, last, 0);
            if (last) {
                __threadfence();
                float t = 0.f;
                for (int c = lane; c < h.nchunks; c += 32) t += __ldcg(a.partials + h.first + c);
                t = warp_sum(t);
                if (lane == 0) {
                    a.hub_count[tk.x] = 0;
                    finish_row<kEW, kRS, kPS, kBaseVec, kCG>(a, it, h.row, t, l1, chg);
                }
            }
        } else if (item < plan.n_tasks + plan.n_long) {
            const int32_t r = plan.longrows[item - plan.n_tasks];
            const int64_t b = a.index[r], e = a.index[r + 1];
            float s = 0.f;
            // Scalar head up to a 16-byte boundary, then 128-bit neighbour loads.
            const int64_t ab = min(e, (b + 3) & ~(int64_t)3);
            if (b + lane < ab) s += edge_val<kEW>(a, it, b + lane);
            for (int64_t i = ab + 4 * lane; i + 3 < e; i += 128) {
                const int4 v4 = __ldg(reinterpret_cast<const int4 *>(a.nbr + i));
                if (kEW) {
                    const float4 w4 = __ldg(reinterpret_cast<const float4 *>(a.ew + i));
                    s += __ldca(it.gin + v4.x) * w4.x + __ldca(it.gin + v4.y) * w4.y +
                         __ldca(it.gin + v4.z) * w4.z + __ldca(it.gin + v4.w) * w4.w;
                } else {
                    s += (__ldca(it.gin + v4.x) + __ldca(it.gin + v4.y)) + (__ldca(it.gin + v4.z) + __ldca(it.gin + v4.w));
                }
            }
            const int64_t tail = ab + ((e - ab) & ~(int64_t)3);
            if (tail + lane < e) s += edge_val<kEW>(a, it, tail + lane);
            s = warp_sum(s);
            if (lane == 0) finish_row<kEW, kRS, kPS, kBaseVec, kCG>(a, it, r, s, l1, chg);
        } else {
            // Stream group: rows r0 .. r0+31 (clipped to n_active).
            const int32_t r0 = plan.stream[item - plan.n_tasks - plan.n_long] * 32;
            const int32_t r = r0 + lane;
            const int32_t rc = min(r, a.n_active);
            const int64_t s0 = a.index[r0];
            const int32_t rel = (int32_t)(a.index[rc] - s0);  // start of this lane's row
            const int32_t gend = (int32_t)(a.index[min(r0 + 32, a.n_active)] - s0);
            s_acc[wib][lane] = 0.f;
            __syncwarp();
            // Four 32-edge chunks per pass: their loads and gathers are issued
            // together, then each chunk is summed by its segmented scan in the
            // same order as one chunk at a time.
            for (int k0 = 0; k0 < gend; k0 += 128) {
                float vals[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int k = k0 + 32 * j + lane;
                    vals[j] = k < gend ? edge_val<kEW>(a, it, s0 + k) : 0.f;
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const int kb = k0 + 32 * j;
                    if (kb >= gend) break;
                    const int k = kb + lane;
                    const bool act = k < gend;
                    int lo = 0;
#pragma unroll
                    for (int st = 16; st > 0; st >>= 1) {
                        const int c = __shfl_sync(kFull, rel, lo + st);
                        if (c <= k) lo += st;
                    }
                    int owner = act ? lo : 32;
                    float v = vals[j];
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const float y = __shfl_up_sync(kFull, v, o);
                        const int ow = __shfl_up_sync(kFull, owner, o);
                        if (lane >= o && ow == owner) v += y;
                    }
                    const int next_owner = __shfl_down_sync(kFull, owner, 1);
                    const bool tail = (lane == 31) || next_owner != owner;
                    if (act && tail) s_acc[wib][owner] += v;
                    __syncwarp();
                }
            }
            if (r < a.n_active) finish_row<kEW, kRS, kPS, kBaseVec, kCG>(a, it, r, s_acc[wib][lane], l1, chg);
            __syncwarp();
        }
    }

}

// Thread 0 of block 0, at the start of iteration `it`: once the launch has run for
// the run limit, it ends after this iteration.  Every block reads pause_after
// after the iteration's (first) barrier; by then block 0 may have moved on and
// named a later iteration, so the number is compared.  In shared memory, and
// before the sweep: the clock is slow to read, and a barrier's last arrival is
// what everybody waits for.
__device__ __forceinline__ void past_run_limit(IterState *st, int it, unsigned long long *s_start) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    const unsigned long long now = globaltimer_ns();
    if (*s_start == 0ull) *s_start = now;
    else if (now - *s_start > c_limits.run_ns) st->pause_after = it + 1;
}

// Adds the block's sums of l1 and chg to the iteration's slot (every thread calls it).
__device__ __forceinline__ void add_residual(IterSlot *slot, float l1, int chg) {
    __shared__ double s_l1[kPrThreads / 32];
    __shared__ int s_chg[kPrThreads / 32];
    const double dl1 = warp_sum((double)l1);
    const int dchg = __reduce_add_sync(kFull, chg);
    if ((threadIdx.x & 31) == 0) {
        s_l1[threadIdx.x >> 5] = dl1;
        s_chg[threadIdx.x >> 5] = dchg;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        int c = 0;
        for (int i = 0; i < kPrThreads / 32; i++) {
            t += s_l1[i];
            c += s_chg[i];
        }
        if (t != 0.0) atomicAdd(&slot->l1, t);
        if (c) atomicAdd(&slot->changed, c);
    }
}

// Sweeps until converged, in one cooperative launch: a grid barrier between
// sweeps, and every block evaluates the stopping rule from the iteration's
// sums.  (A launch per sweep and a host check per four took 340 us for any
// small graph; here a sweep of one costs its own few microseconds.)
// cheb_rho > 0: Chebyshev semi-iteration for a Jacobi operator whose spectrum
// lies in [-cheb_rho, cheb_rho] (a reversible walk scaled by d): weights
// omega_1 = 1, omega_2 = 1 / (1 - rho^2 / 2), omega_{k+1} = 1 / (1 - rho^2
// omega_k / 4) (Golub and Varga, 1961).
// A launch that has run for the run limit ends after its iteration, and the host
// launches the rest (run_solve): a solve may take longer, one launch may not.
template <bool kEW, bool kRS, bool kPS, bool kBaseVec>
__global__ void __launch_bounds__(kPrThreads, kPrBlocks) pr_solve(SweepArgs a, PrPlanDev plan) {
    __shared__ float s_acc[kPrThreads / 32][32];
    const double rho2 = (double)a.cheb_rho * a.cheb_rho;
    __shared__ unsigned long long s_start;
    __shared__ bool s_done, s_paused;
    if (threadIdx.x == 0) s_start = 0ull;
    double omega = a.first_omega;
    int it = a.first_iter, done = 0;
    bool ok = true, paused = false;
    while (it < a.max_iters && !done && !paused) {
        if (a.cheb_rho > 0.f)
            omega = it == 0 ? 1.0 : it == 1 ? 1.0 / (1.0 - rho2 / 2.0) : 1.0 / (1.0 - rho2 * omega / 4.0);
        const int cur = it & 1;
        const SweepIter v{kPS ? a.g[cur] : a.x[cur], a.x[cur], a.x[cur ^ 1], kPS ? a.g[cur ^ 1] : a.x[cur ^ 1],
                          (float)omega};
        float l1;
        int chg;
        past_run_limit(a.st, it, &s_start);
        sweep_rows<kEW, kRS, kPS, kBaseVec>(a, plan, v, s_acc, l1, chg);
        IterSlot *const slot = &a.st->slot[it % kMaxIterSlots];
        add_residual(slot, l1, chg);
        if (it + 2 >= kMaxIterSlots && blockIdx.x == 0 && threadIdx.x == 0)
            a.st->slot[(it + 2) % kMaxIterSlots] = IterSlot{0.0, 0.0, 0.0, 0, 0};
        if (!(ok = grid_barrier(&a.st->gs))) break;
        it++;
        if (threadIdx.x == 0) {  // one read a block: every warp's would queue at one L2 line
            const double sum = __ldcg(&slot->l1);
            const int moved = __ldcg(&slot->changed), pause_after = __ldcg(&a.st->pause_after);
            // eps >= 3e38 marks the per-vertex rule as unused.
            s_done = (a.tol_l1 > 0.f && sum < (double)a.tol_l1) || (a.eps < 3e38f && moved == 0);
            s_paused = pause_after == it;
        }
        __syncthreads();
        done = s_done;
        paused = s_paused;
    }
    paused = paused && !done && it < a.max_iters;
    if (ok && !paused && a.final_x) {
        const float *x = a.x[it & 1];
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) a.final_x[i] = x[i];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.out->err = *(volatile int *)&a.st->gs.err;
        a.out->iters = it;
        a.out->done = paused ? 0 : done ? 1 : 2;
        a.out->omega = omega;
        a.out->l1 = it > 0 ? __ldcg(&a.st->slot[(it - 1) % kMaxIterSlots].l1) : 0.0;
        a.out->changed = it > 0 ? __ldcg(&a.st->slot[(it - 1) % kMaxIterSlots].changed) : 0;
        __threadfence_system();
    }
}

// One sweep as its own launch (see launched_sweeps): the last block to finish
// decides convergence, and sweeps queued after it return at once.
template <bool kEW, bool kRS, bool kPS, bool kBaseVec>
__global__ void __launch_bounds__(kPrThreads) pr_step(SweepArgs a, PrPlanDev plan, SweepIter v, int it) {
    __shared__ float s_acc[kPrThreads / 32][32];
    if (*(volatile int *)&a.st->done) return;
    float l1;
    int chg;
    sweep_rows<kEW, kRS, kPS, kBaseVec>(a, plan, v, s_acc, l1, chg);
    IterSlot *const slot = &a.st->slot[it % kMaxIterSlots];
    add_residual(slot, l1, chg);
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(&a.st->blocks_done, 1) == (int)gridDim.x - 1) {
            __threadfence();
            const double tl1 = __ldcg(&slot->l1);
            const int tch = __ldcg(&slot->changed);
            a.st->blocks_done = 0;
            a.st->slot[(it + 1) % kMaxIterSlots] = IterSlot{0.0, 0.0, 0.0, 0, 0};
            const bool conv = (a.tol_l1 > 0.f && tl1 < (double)a.tol_l1) || (a.eps < 3e38f && tch == 0);
            if (conv || it + 1 >= a.max_iters) {
                a.st->done = 1;
                a.out->iters = it + 1;
                a.out->l1 = tl1;
                a.out->changed = tch;
                a.out->done = conv ? 1 : 2;
                __threadfence_system();
            }
        }
    }
}

// x <- (1-d) t (or (1-d)/N) for every vertex; gather vector g <- x * ps.
// Rows that may have edges start from x0_scale * (x0v or x0_scalar).
__global__ void pr_init(int32_t n, const float *basev, float base_scalar, float x0_scalar, const float *x0v,
                        float x0_scale, const float *ps, float *x, float *g, float *x2, float *g2, int32_t n_active) {
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const float base = basev ? basev[v] : base_scalar;
        // Vertices without edges sit at their base from the start; the rest
        // start from the initial guess.
        const float x0 = v >= n_active ? base : x0_scale * (x0v ? x0v[v] : x0_scalar);
        x[v] = x0;
        x2[v] = x0;
        if (g) {
            const float gv = ps ? x0 * ps[v] : x0;
            g[v] = gv;
            g2[v] = gv;
        }
    }
}

__global__ void sum_abs(const float *v, int32_t n, double *out) {
    __shared__ double s_red[32];
    double s = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) s += fabs((double)v[i]);
    s = block_sum(s, s_red);
    if (threadIdx.x == 0 && s != 0.0) atomicAdd(out, s);
}

__global__ void scale_vec(const float *in, float s, float *out, size_t n) {
    for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < n; v += (size_t)gridDim.x * blockDim.x)
        out[v] = s * in[v];
}

// dL/dw_uk = (d x_u / s_u) (lambda_k - sum_j W_uj lambda_j), slot order of
// row u, and at the fixed point sum_j W_uj lambda_j = (lambda_u - c_u) / d, so one pass:
// dL/dw_uk = (x_u / s_u) (d lambda_k - lambda_u + c_u).
// Work items are the row plan's: hub chunks and long rows (one warp, one row)
// and stream groups (32 rows, one warp walks their edges 32 at a time and
// each lane finds its edge's row among the group's offsets).
__global__ void __launch_bounds__(kPrThreads) pr_edge_grad(PrPlanDev plan, const int64_t *index, const int32_t *nbr,
                                                           const float *rs, const float *x, const float *lam,
                                                           const float *c, float d, int32_t n_active, float *grad) {
    const int lane = threadIdx.x & 31;
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const int total = plan.n_tasks + plan.n_long + plan.n_stream;
    for (int item = gwarp; item < total; item += nwarps) {
        if (item < plan.n_tasks + plan.n_long) {
            int32_t u;
            int64_t b, e;
            if (item < plan.n_tasks) {
                const int2 tk = plan.tasks[item];
                u = plan.hubs[tk.x].row;
                const int64_t rb = index[u], re = index[u + 1];
                b = rb + (int64_t)tk.y * plan.chunk;
                e = min(re, b + (int64_t)plan.chunk);
            } else {
                u = plan.longrows[item - plan.n_tasks];
                b = index[u];
                e = index[u + 1];
            }
            const float coef = x[u] * rs[u];
            const float off = lam[u] - c[u];
            for (int64_t i = b + lane; i < e; i += 32) grad[i] = coef * (d * __ldg(lam + nbr[i]) - off);
        } else {
            const int32_t r0 = plan.stream[item - plan.n_tasks - plan.n_long] * 32;
            const int32_t r = r0 + lane;
            const int32_t rc = min(r, n_active);
            const int64_t s0 = index[r0];
            const int32_t rel = (int32_t)(index[rc] - s0);
            const int32_t gend = (int32_t)(index[min(r0 + 32, n_active)] - s0);
            const float coef = r < n_active ? x[r] * rs[r] : 0.f;
            const float off = r < n_active ? lam[r] - c[r] : 0.f;
            for (int k0 = 0; k0 < gend; k0 += 32) {
                const int k = k0 + lane;
                int lo = 0;
#pragma unroll
                for (int st = 16; st > 0; st >>= 1) {
                    const int cc = __shfl_sync(kFull, rel, lo + st);
                    if (cc <= k) lo += st;
                }
                const float cf = __shfl_sync(kFull, coef, lo);
                const float of = __shfl_sync(kFull, off, lo);
                if (k < gend) grad[s0 + k] = cf * (d * __ldg(lam + nbr[s0 + k]) - of);
            }
        }
    }
}

// ---------------------------------------------------------------- SpMM form
// K columns per vertex, vertex-major [N][S], S = K rounded up to four (the
// added columns hold zeros).  Every gather is a float4: kLanes lanes hold one
// neighbour's row segment (kVec float4 each), so a warp has 32 / kLanes
// neighbours per load and kFlight loads in flight.  A hub chunk or long row is
// spread over the whole warp; shorter rows take 32 / kLanes at a time, one per
// kLanes lanes.  (One neighbour per round trip left a warp waiting on L2 for its
// whole row: Kronecker scale 18, 48 columns, 541 us a sweep; the gathers are 1.46
// GB through L2.)
struct SpmmArgs {
    const int64_t *index;
    const int32_t *nbr;
    const float *ew;
    const float *gin;        // [N][S], already divided by deg (unweighted)
    const float *xin;
    const float *basev;      // [N][S] dense base, or null with seeds
    const int32_t *seed_off; // sparse teleport: column c has seeds seed_idx[seed_off[c]..seed_off[c+1])
    const int32_t *seed_idx;
    float d;
    const float *ps;         // per-row gather scale
    float *xout, *gout;
    float *partials;         // [chunks][S]
    unsigned *hub_count;
    double *col_l1;          // [S] accumulators for this sweep
    const int32_t *col_map;  // packed column -> seed-list column (null: identity)
    int K, S;                // columns in the packed layout, and its row stride
    int32_t n_active;
};
__host__ __device__ constexpr int spmm_stride(int K) { return (K + 3) / 4 * 4; }

__device__ __forceinline__ float spmm_base(const SpmmArgs &a, int32_t r, int c, float one_minus_d) {
    if (a.basev) return a.basev[(size_t)r * a.S + c];
    if (c >= a.K) return 0.f;
    // Uniform over the seed set of column c.
    const int cc = a.col_map ? a.col_map[c] : c;
    const int32_t b = a.seed_off[cc], e = a.seed_off[cc + 1];
    for (int32_t i = b; i < e; i++)
        if (a.seed_idx[i] == r) return one_minus_d / (float)(e - b);
    return 0.f;
}

__device__ __forceinline__ void add4(float4 &x, const float4 &y) {
    x.x += y.x;
    x.y += y.y;
    x.z += y.z;
    x.w += y.w;
}
__device__ __forceinline__ void fma4(float4 &x, float w, const float4 &y) {
    x.x += w * y.x;
    x.y += w * y.y;
    x.z += w * y.z;
    x.w += w * y.w;
}

// Adds w * gin[nbr] over the edges i = b, b + step, ... below e to this lane's columns.
template <int kVec, int kLanes, bool kEW>
__device__ __forceinline__ void spmm_range(const SpmmArgs &a, int64_t b, int64_t e, int step, int q0,
                                           float4 (&acc)[kVec]) {
    constexpr int kFlight = kVec > 1 ? 4 : 8;
    for (int64_t i0 = b; i0 < e; i0 += (int64_t)step * kFlight) {
        float4 v[kFlight][kVec];
        float w[kFlight];
        int32_t u[kFlight];
#pragma unroll
        for (int f = 0; f < kFlight; f++) {
            const int64_t i = i0 + (int64_t)f * step;
            u[f] = i < e ? __ldg(a.nbr + i) : -1;
            w[f] = kEW && i < e ? __ldg(a.ew + i) : 0.f;
        }
#pragma unroll
        for (int f = 0; f < kFlight; f++)
#pragma unroll
            for (int j = 0; j < kVec; j++) {
                const int c = q0 + 4 * kLanes * j;
                v[f][j] = u[f] >= 0 && c < a.S ? __ldg(reinterpret_cast<const float4 *>(a.gin + (size_t)u[f] * a.S + c))
                                               : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
        for (int f = 0; f < kFlight; f++)
#pragma unroll
            for (int j = 0; j < kVec; j++) {
                if (kEW) fma4(acc[j], w[f], v[f][j]);
                else add4(acc[j], v[f][j]);
            }
    }
}

template <int kVec, int kLanes, bool kEW>
__global__ void __launch_bounds__(kPrThreads) spmm_sweep(SpmmArgs a, SpmmPlanDev plan, const uint8_t *is_seed) {
    constexpr int kSub = 32 / kLanes;  // rows (or neighbours of one row) at a time
    __shared__ float s_l1[kPrThreads / 32][4 * kLanes * kVec];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int sub = lane / kLanes, q0 = 4 * (lane % kLanes);
    const int gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    const float omd = 1.0f - a.d;
    float4 l1[kVec];
#pragma unroll
    for (int j = 0; j < kVec; j++) l1[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    auto clear = [](float4 (&x)[kVec]) {
#pragma unroll
        for (int j = 0; j < kVec; j++) x[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    };
    // The subs' sums of one row, in every sub.
    auto combine = [](float4 (&x)[kVec]) {
#pragma unroll
        for (int o = kLanes; o < 32; o <<= 1)
#pragma unroll
            for (int j = 0; j < kVec; j++) {
                float4 y;
                y.x = __shfl_xor_sync(kFull, x[j].x, o);
                y.y = __shfl_xor_sync(kFull, x[j].y, o);
                y.z = __shfl_xor_sync(kFull, x[j].z, o);
                y.w = __shfl_xor_sync(kFull, x[j].w, o);
                add4(x[j], y);
            }
    };
    auto finish = [&](int32_t r, const float4 (&acc)[kVec]) {
        const float ps = a.ps ? a.ps[r] : 1.0f;
        const bool seed = is_seed ? is_seed[r] != 0 : true;
#pragma unroll
        for (int j = 0; j < kVec; j++) {
            const int c = q0 + 4 * kLanes * j;
            if (c < a.S) {
                const size_t o = (size_t)r * a.S + c;
                const float4 ov = *reinterpret_cast<const float4 *>(a.xin + o);
                float4 nv = make_float4(0.f, 0.f, 0.f, 0.f);
                if (seed) nv = make_float4(spmm_base(a, r, c, omd), spmm_base(a, r, c + 1, omd),
                                           spmm_base(a, r, c + 2, omd), spmm_base(a, r, c + 3, omd));
                fma4(nv, a.d, acc[j]);
                *reinterpret_cast<float4 *>(a.xout + o) = nv;
                if (a.gout != a.xout)
                    *reinterpret_cast<float4 *>(a.gout + o) = make_float4(nv.x * ps, nv.y * ps, nv.z * ps, nv.w * ps);
                add4(l1[j], make_float4(fabsf(nv.x - ov.x), fabsf(nv.y - ov.y), fabsf(nv.z - ov.z), fabsf(nv.w - ov.w)));
            }
        }
    };
    const int total = plan.n_tasks + plan.n_long + (a.n_active + plan.rows - 1) / plan.rows;
    for (int item = gwarp; item < total; item += nwarps) {
        float4 acc[kVec];
        clear(acc);
        if (item < plan.n_tasks) {
            const int2 tk = plan.tasks[item];
            const HubInfo h = plan.hubs[tk.x];
            const int64_t rb = __ldg(a.index + h.row), re = __ldg(a.index + h.row + 1);
            const int64_t b = rb + (int64_t)tk.y * plan.chunk;
            spmm_range<kVec, kLanes, kEW>(a, b + sub, min(re, b + (int64_t)plan.chunk), kSub, q0, acc);
            combine(acc);
            if (sub == 0) {
#pragma unroll
                for (int j = 0; j < kVec; j++) {
                    const int c = q0 + 4 * kLanes * j;
                    if (c < a.S) *reinterpret_cast<float4 *>(a.partials + (size_t)(h.first + tk.y) * a.S + c) = acc[j];
                }
            }
            __syncwarp();
            int last = 0;
            if (lane == 0) {
                __threadfence();
                last = atomicAdd(a.hub_count + tk.x, 1u) == (unsigned)(h.nchunks - 1);
            }
            last = __shfl_sync(kFull, last, 0);
            if (!last) continue;
            __threadfence();
            clear(acc);
#pragma unroll 4
            for (int ch = sub; ch < h.nchunks; ch += kSub) {
#pragma unroll
                for (int j = 0; j < kVec; j++) {
                    const int c = q0 + 4 * kLanes * j;
                    if (c < a.S)
                        add4(acc[j], __ldcg(reinterpret_cast<const float4 *>(a.partials + (size_t)(h.first + ch) * a.S + c)));
                }
            }
            combine(acc);
            if (lane == 0) a.hub_count[tk.x] = 0;
            if (sub == 0) finish(h.row, acc);
        } else if (item < plan.n_tasks + plan.n_long) {
            const int32_t r = plan.longs[item - plan.n_tasks];
            spmm_range<kVec, kLanes, kEW>(a, __ldg(a.index + r) + sub, __ldg(a.index + r + 1), kSub, q0, acc);
            combine(acc);
            if (sub == 0) finish(r, acc);
        } else {
            const int32_t r0 = (item - plan.n_tasks - plan.n_long) * plan.rows;
            const int nr = min(plan.rows, a.n_active - r0);
            const int64_t start = __ldg(a.index + r0 + min(lane, nr));
            const int64_t deg = __shfl_down_sync(kFull, start, 1) - start;
            if (!__any_sync(kFull, lane < nr && deg <= kSpmmLong)) continue;
#pragma unroll 1
            for (int k0 = 0; k0 < nr; k0 += kSub) {
                const int k = k0 + sub;
                const int64_t b = __shfl_sync(kFull, start, min(k, 31)), e = __shfl_sync(kFull, start, min(k + 1, 31));
                if (k < nr && e - b <= kSpmmLong) {
                    clear(acc);
                    spmm_range<kVec, kLanes, kEW>(a, b, e, 1, q0, acc);
                    finish(r0 + k, acc);
                }
            }
        }
    }
    // Column sums: the subs', then the block's warps', then one atomic per column.
    combine(l1);
    if (sub == 0) {
#pragma unroll
        for (int j = 0; j < kVec; j++) *reinterpret_cast<float4 *>(&s_l1[wib][q0 + 4 * kLanes * j]) = l1[j];
    }
    __syncthreads();
    for (int c = threadIdx.x; c < a.K; c += blockDim.x) {
        double t = 0.0;
        for (int w = 0; w < kPrThreads / 32; w++) t += (double)s_l1[w][c];
        if (t != 0.0) atomicAdd(a.col_l1 + c, t);
    }
}

// A dense teleport matrix t ([n][K]) as the base (1-d) t at the padded stride.
__global__ void spmm_pad_base(int32_t n, int K, const float *t, float one_minus_d, float *base) {
    const int S = spmm_stride(K);
    const size_t total = (size_t)n * S;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % S);
        base[i] = c < K ? one_minus_d * t[i / S * K + c] : 0.f;
    }
}
// The scores without the padding ([n][K]).
__global__ void spmm_unpad(int32_t n, int K, const float *x, float *out) {
    const int S = spmm_stride(K);
    const size_t total = (size_t)n * K;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x)
        out[i] = x[i / K * S + i % K];
}

// Start: each column's teleport t (base / (1-d)), which has the fixed
// point's mass; vertices without edges sit at their base (1-d) t from the start.
__global__ void spmm_init(int32_t n, int K, const float *basev, const int32_t *seed_off, const int32_t *seed_idx,
                          const uint8_t *is_seed, float d, const float *ps, float *x, float *g, float *x2, float *g2,
                          int32_t n_active) {
    const int S = spmm_stride(K);
    const size_t total = (size_t)n * S;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int32_t v = (int32_t)(i / S);
        const int c = (int)(i % S);
        float base = 0.f;
        if (basev) {
            base = basev[i];
        } else if (c < K && is_seed[v]) {
            const int32_t b = seed_off[c], e = seed_off[c + 1];
            for (int32_t j = b; j < e; j++)
                if (seed_idx[j] == v) base = (1.0f - d) / (float)(e - b);
        }
        const float t = v < n_active ? base / (1.0f - d) : base;
        x[i] = t;
        x2[i] = t;
        const float gv = ps ? t * ps[v] : t;
        g[i] = gv;
        g2[i] = gv;
    }
}

// Repacks the live columns of x (kw columns) into xo (nkw columns, gather copy
// go = xo * ps when go is set), both at their padded strides; a column with
// newpos < 0 has converged and goes to its place col_map[c] in out ([n][K0]).
// Padding columns stay zero.
__global__ void spmm_repack(int32_t n, int kw, const float *x, const int32_t *newpos, const int32_t *col_map,
                            int K0, float *out, int nkw, float *xo, float *go, const float *ps) {
    const size_t total = (size_t)n * kw;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int32_t v = (int32_t)(i / kw);
        const int c = (int)(i % kw);
        const float val = x[(size_t)v * spmm_stride(kw) + c];
        const int np = newpos[c];
        const int so = spmm_stride(nkw);
        if (np < 0) {
            out[(size_t)v * K0 + col_map[c]] = val;
        } else {
            xo[(size_t)v * so + np] = val;
            if (go) go[(size_t)v * so + np] = ps ? val * ps[v] : val;
        }
        if (c == 0)
            for (int z = nkw; z < so; z++) {
                xo[(size_t)v * so + z] = 0.f;
                if (go) go[(size_t)v * so + z] = 0.f;
            }
    }
}

// One packed column c (width kw) as a plain vector (and its gather copy).
__global__ void spmm_take_column(int32_t n, int kw, int c, const float *x, const float *ps, float *x0, float *x1,
                                 float *g0, float *g1) {
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const float val = x[(size_t)v * spmm_stride(kw) + c];
        x0[v] = val;
        x1[v] = val;
        if (g0) {
            const float gv = ps ? val * ps[v] : val;
            g0[v] = gv;
            g1[v] = gv;
        }
    }
}

// base[v] = (1-d) / |seeds| on the seeds of one column (base zeroed before).
__global__ void spmm_column_base(const int32_t *seed_idx, int32_t b, int32_t e, float one_minus_d, float *base) {
    for (int i = b + blockIdx.x * blockDim.x + threadIdx.x; i < e; i += gridDim.x * blockDim.x)
        base[seed_idx[i]] = one_minus_d / (float)(e - b);
}

__global__ void spmm_put_column(int32_t n, const float *x, int K0, int oc, float *out) {
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        out[(size_t)v * K0 + oc] = x[v];
}

__global__ void mark_seeds(const int32_t *seed_idx, int32_t nseeds, uint8_t *is_seed) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nseeds; i += gridDim.x * blockDim.x)
        is_seed[seed_idx[i]] = 1;
}

__global__ void spmm_residual(const double *col_l1, int K, float tol, int *done_cols) {
    int c = 0;
    for (int i = threadIdx.x; i < K; i += blockDim.x) c += col_l1[i] < (double)tol;
    c = warp_sum(c);
    __shared__ int s[32];
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        int t = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += s[i];
        *done_cols = t;
    }
}

}  // namespace

// ------------------------------------------------------------------- plan

namespace {
// m / per rounded down to a power of two, in [kMinChunk, kMaxChunk].
int64_t plan_size(int64_t m, int64_t per) {
    int64_t x = kMinChunk;
    while (x < kMaxChunk && x * 2 * per <= m) x *= 2;
    return x;
}

// A plan's device arrays go up in one copy.
struct PlanPack {
    std::vector<char> host;
    template <class T>
    size_t add(const std::vector<T> &v) {
        const size_t at = host.size(), bytes = v.size() * sizeof(T);
        host.resize(at + (bytes + 255) / 256 * 256);
        if (bytes) std::memcpy(host.data() + at, v.data(), bytes);
        return at;
    }
    hc_status upload(DevBuf *buf) const {
        HC_TRY(buf->ensure(host.size() + 256));
        if (!host.empty()) HC_CUDA_TRY(cudaMemcpy(buf->ptr, host.data(), host.size(), cudaMemcpyHostToDevice));
        return HC_OK;
    }
};

// Rows longer than `least` edges in chunks: (hub index, chunk) tasks and the hubs' partial sums.
struct HubTasks {
    std::vector<int2> tasks;
    std::vector<HubInfo> hubs;
    int32_t slots = 0;
    void add(int32_t r, int64_t deg, int64_t chunk) {
        HubInfo h{r, slots, (int32_t)((deg + chunk - 1) / chunk), 0};
        for (int c = 0; c < h.nchunks; c++) tasks.push_back(make_int2((int)hubs.size(), c));
        slots += h.nchunks;
        hubs.push_back(h);
    }
};

hc_status build_plan(const int64_t *idx, int32_t na, int64_t stream_edges, int64_t chunk, DevBuf *buf,
                     PrPlanDev *view, int32_t *slots) {
    std::vector<int32_t> stream, longrows;
    HubTasks hub;
    const int32_t ngroups = (na + 31) / 32;
    // Rows that the limit would make single, in groups of up to 1024 and of up to 2048 edges.
    int64_t rows1 = 0, rows2 = 0;
    for (int32_t gid = 0; stream_edges < kMaxChunk && gid < ngroups; gid++) {
        const int32_t r0 = gid * 32, r1 = std::min(r0 + 32, na);
        const int64_t tot = idx[r1] - idx[r0];
        if (tot > stream_edges && tot <= kMaxChunk) (tot <= kMaxChunk / 2 ? rows1 : rows2) += r1 - r0;
    }
    if (rows1 > kMaxSingle1) stream_edges = std::max<int64_t>(stream_edges, kMaxChunk / 2);
    if (rows2 > kMaxSingle2) stream_edges = kMaxChunk;
    for (int32_t gid = 0; gid < ngroups; gid++) {
        const int32_t r0 = gid * 32, r1 = std::min(r0 + 32, na);
        if (idx[r1] - idx[r0] <= stream_edges) {
            stream.push_back(gid);
            continue;
        }
        for (int32_t r = r0; r < r1; r++) {
            const int64_t d = idx[r + 1] - idx[r];
            if (d > 2 * chunk) hub.add(r, d, chunk);
            else longrows.push_back(r);
        }
    }
    PlanPack pack;
    const size_t at_stream = pack.add(stream), at_long = pack.add(longrows);
    const size_t at_tasks = pack.add(hub.tasks), at_hubs = pack.add(hub.hubs);
    HC_TRY(pack.upload(buf));
    const char *p = buf->as<char>();
    *view = PrPlanDev{(const int32_t *)(p + at_stream), (const int32_t *)(p + at_long), (const int2 *)(p + at_tasks),
                      (const HubInfo *)(p + at_hubs), (int)stream.size(), (int)longrows.size(),
                      (int)hub.tasks.size(), (int)hub.hubs.size(), (int)chunk};
    *slots = hub.slots;
    return HC_OK;
}

// The multi-column sweeps' row plan.  A chunk is M / 65536 edges rounded down to
// a power of two, in [512, 2048]: a chunk is a serial chain of its warp, and its
// partial sums take a row of columns each.
hc_status build_spmm_plan(hc_graph *g, const int64_t *idx) {
    const int32_t na = g->n_active;
    int64_t chunk = 512;
    while (chunk < 2048 && chunk * 2 * 65536 <= g->M) chunk *= 2;
    std::vector<int32_t> longs;
    HubTasks hub;
    for (int32_t r = 0; r < na; r++) {
        const int64_t d = idx[r + 1] - idx[r];
        if (d > chunk) hub.add(r, d, chunk);
        else if (d > kSpmmLong) longs.push_back(r);
        else if (g->degree_sorted) break;  // every later row is short too
    }
    // Eight warps a block, eight blocks an SM (launch_spmm_cols).  On a small graph a
    // sweep is the longest warp's chain, and eight rows one after the other are most
    // of it (uniform, 2^11 vertices, three seeds a column: 200 columns 1350 us a solve, 410
    // us so, 64 columns 493 and 356).
    const int rows = (int)std::max<int64_t>(1, std::min<int64_t>(kSpmmRows, na / ((int64_t)g->sm_count * 64)));
    PlanPack pack;
    const size_t at_long = pack.add(longs), at_tasks = pack.add(hub.tasks), at_hubs = pack.add(hub.hubs);
    HC_TRY(pack.upload(&g->spmm_plan));
    const char *p = g->spmm_plan.as<char>();
    g->spmm_view = SpmmPlanDev{(const int32_t *)(p + at_long), (const int2 *)(p + at_tasks),
                               (const HubInfo *)(p + at_hubs), (int)longs.size(), (int)hub.tasks.size(),
                               (int)hub.hubs.size(), (int)chunk, rows};
    g->spmm_partial_slots = hub.slots;
    return HC_OK;
}
}  // namespace

// One read of the offsets serves every plan that a call lacks.
hc_status ensure_plans(hc_graph *g, unsigned which) {
    const int64_t stream_edges = plan_size(g->M, 8192), chunk = plan_size(g->M, 4096);
    // From 2^24 edges on the two plans are one.
    const bool same = stream_edges == kMaxChunk && chunk == kMaxChunk;
    if ((which & kPlanPr) && same) which = (which & ~kPlanPr) | kPlanBase;
    if (g->pr_plan.ptr) which &= ~kPlanPr;
    if (g->base_plan.ptr) which &= ~kPlanBase;
    if (g->spmm_plan.ptr) which &= ~kPlanSpmm;
    if (!which) return HC_OK;
    const int32_t na = g->n_active;
    // Not a vector: clearing it first takes as long as the copy.
    std::unique_ptr<int64_t[]> idx(new (std::nothrow) int64_t[(size_t)na + 1]);
    if (!idx) return fail(HC_ERR_OOM, "row plans: no host memory for %d offsets", na + 1);
    HC_CUDA_TRY(cudaMemcpy(idx.get(), g->index.as<int64_t>(), sizeof(int64_t) * ((size_t)na + 1),
                           cudaMemcpyDeviceToHost));
    if (which & kPlanPr)
        HC_TRY(build_plan(idx.get(), na, stream_edges, chunk, &g->pr_plan, &g->pr_view, &g->pr_partial_slots));
    if (which & kPlanBase) {
        HC_TRY(build_plan(idx.get(), na, kMaxChunk, kMaxChunk, &g->base_plan, &g->base_view, &g->base_partial_slots));
        if (same) {
            g->pr_view = g->base_view;
            g->pr_partial_slots = g->base_partial_slots;
        }
    }
    if (which & kPlanSpmm) HC_TRY(build_spmm_plan(g, idx.get()));
    return HC_OK;
}

namespace {

template <bool kEW>
void launch_spmm_cols(hc_graph *g, const SpmmArgs &a, const uint8_t *is_seed) {
    const int grid = g->sm_count * 8;
    const SpmmPlanDev &plan = g->spmm_view;
    if (a.S <= 8) spmm_sweep<1, 2, kEW><<<grid, kPrThreads, 0, g->stream>>>(a, plan, is_seed);
    else if (a.S <= 16) spmm_sweep<1, 4, kEW><<<grid, kPrThreads, 0, g->stream>>>(a, plan, is_seed);
    else if (a.S <= 32) spmm_sweep<1, 8, kEW><<<grid, kPrThreads, 0, g->stream>>>(a, plan, is_seed);
    else if (a.S <= 64) spmm_sweep<1, 16, kEW><<<grid, kPrThreads, 0, g->stream>>>(a, plan, is_seed);
    else if (a.S <= 128) spmm_sweep<1, 32, kEW><<<grid, kPrThreads, 0, g->stream>>>(a, plan, is_seed);
    else spmm_sweep<2, 32, kEW><<<grid, kPrThreads, 0, g->stream>>>(a, plan, is_seed);
    ::hc::count_launch();
}

void launch_spmm(hc_graph *g, const SpmmArgs &a, const uint8_t *is_seed) {
    if (a.ew) launch_spmm_cols<true>(g, a, is_seed);
    else launch_spmm_cols<false>(g, a, is_seed);
}

// A cooperative launch of `fn` over the row plan's items: no more blocks than a
// warp each needs (a barrier costs by the block), or all that fit (`all`).
hc_status launch_solve(hc_graph *g, const void *fn, int *blocks_per_sm, SweepArgs &a, const PrPlanDev &plan, bool all,
                       void *extra) {
    if (*blocks_per_sm == 0) {
        int b = 0;
        HC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, fn, kPrThreads, 0));
        if (b < 1) return fail(HC_ERR_CUDA, "PageRank kernel cannot be resident");
        *blocks_per_sm = b;
    }
    const int64_t warps = (int64_t)plan.n_tasks + plan.n_long + plan.n_stream;
    const int64_t want = std::max<int64_t>(1, (warps + kPrThreads / 32 - 1) / (kPrThreads / 32));
    const int64_t fit = (int64_t)*blocks_per_sm * g->sm_count;
    const int grid = (int)(all ? fit : std::min(want, fit));
    PrPlanDev p = plan;
    void *params[] = {&a, &p, extra};
    ::hc::count_launch();
    HC_CUDA_TRY(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(kPrThreads), params, 0, g->stream));
    return HC_OK;
}

// Whether a solve's sweeps are launched one by one: on a graph of at least 2^24
// edges without hub rows, whose sweeps miss L1 throughout (uniform, 33M edges: 1.19
// ms so, 1.33 ms in one launch; at 8M edges both 0.48 ms).  With hubs one launch is
// the faster at every size (Kronecker scale 22: 2.99 and 2.87 ms, scale 20: 0.94 and
// 0.85 ms, scale 12: 0.35 and 0.09 ms).  Where nearly every
// row is in a stream group, from 3 x 2^20 edges (uniform, 2^18 vertices, rows of 16:
// 0.32 and 0.38 ms; 2^19: 0.47 and 0.55, rows of 32: 0.65 and 0.78; but 2^17, rows of
// 16: 0.26 and 0.22, and 2^18, rows of 24, a quarter of them single: 0.38 and 0.35);
// from 2^18 vertices and 8 million edges whatever the rows (2^18, rows of 32: 0.42 and
// 0.44 ms, Chebyshev weights 1.51 and 1.61; but 2^17, rows of 64: 0.31 and 0.27).
bool launched_sweeps(const hc_graph *g, const PrPlanDev &plan) {
    return plan.n_tasks == 0 && (g->M >= (1ll << 24) || (plan.n_long <= plan.n_stream && g->M >= (3ll << 20)) ||
                                 (g->n_active >= (1 << 18) && g->M >= 8000000));
}

using SolveFn = hc_status (*)(hc_graph *, SweepArgs &, const PrPlanDev &, volatile SolveOut *);

// The Chebyshev weight of sweep `it` (the recurrence of pr_solve).
double next_omega(double omega, int it, float rho) {
    if (rho <= 0.f) return 1.0;
    const double rho2 = (double)rho * rho;
    return it == 0 ? 1.0 : it == 1 ? 1.0 / (1.0 - rho2 / 2.0) : 1.0 / (1.0 - rho2 * omega / 4.0);
}

template <bool kEW, bool kRS, bool kPS, bool kBaseVec>
hc_status launch_pr_solve(hc_graph *g, SweepArgs &a, const PrPlanDev &plan, volatile SolveOut *out) {
    if (launched_sweeps(g, plan)) {
        static int step_bps = 0;
        if (step_bps == 0) {
            HC_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&step_bps, pr_step<kEW, kRS, kPS, kBaseVec>,
                                                                      kPrThreads, 0));
            step_bps = std::max(step_bps, 1);
        }
        // Launches are queued in rounds, the host looking once per round.
        constexpr int kRound = 4;
        double omega = 1.0;
        for (int it = 0; it < a.max_iters && !out->done;) {
            for (int k = 0; k < kRound && it < a.max_iters; k++, it++) {
                omega = next_omega(omega, it, a.cheb_rho);
                const int cur = it & 1;
                const SweepIter v{kPS ? a.g[cur] : a.x[cur], a.x[cur], a.x[cur ^ 1], kPS ? a.g[cur ^ 1] : a.x[cur ^ 1],
                                  (float)omega};
                { pr_step<kEW, kRS, kPS, kBaseVec><<<g->sm_count * step_bps, kPrThreads, 0, g->stream>>>(a, plan, v, it); ::hc::count_launch(); }
            }
            HC_CUDA_TRY(cudaGetLastError());
            HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
        }
        if (a.final_x)
            HC_CUDA_TRY(cudaMemcpyAsync(a.final_x, a.x[out->iters & 1], (size_t)a.n * 4, cudaMemcpyDeviceToDevice,
                                        g->stream));
        return HC_OK;
    }
    static int bps = 0;
    return launch_solve(g, (const void *)pr_solve<kEW, kRS, kPS, kBaseVec>, &bps, a, plan, false, nullptr);
}

SolveFn pick_solve(bool ew, bool rs, bool ps, bool basev) {
    const int key = (ew ? 8 : 0) | (rs ? 4 : 0) | (ps ? 2 : 0) | (basev ? 1 : 0);
    switch (key) {
        case 2: return launch_pr_solve<false, false, true, false>;
        case 3: return launch_pr_solve<false, false, true, true>;
        case 5: return launch_pr_solve<false, true, false, true>;
        case 8: return launch_pr_solve<true, false, false, false>;
        case 9: return launch_pr_solve<true, false, false, true>;
        case 13: return launch_pr_solve<true, true, false, true>;
        default: return nullptr;
    }
}

struct SolveResult {
    int iters;
    int done;
    double l1;
    int changed;
    float ms;
};

// The solve's state for max_iters iterations, zeroed, and its report's mapped slot.
hc_status solve_begin(hc_graph *g, SweepArgs &a, SolveOut **out) {
    HC_TRY(g->ws_ctl.ensure(sizeof(IterState) + 4096));
    a.st = reinterpret_cast<IterState *>(g->ws_ctl.ptr);
    const size_t slots = std::min<size_t>((size_t)a.max_iters + 1, kMaxIterSlots);
    HC_CUDA_TRY(cudaMemsetAsync(a.st, 0, offsetof(IterState, slot) + sizeof(IterSlot) * slots, g->stream));
    HC_TRY(ctl_slot(g, 0, (void **)out, (void **)&a.out));
    **out = SolveOut{0, 0, 0, 0, 0.0, 1.0};
    a.first_iter = 0;
    a.first_omega = 1.0;
    HC_CUDA_TRY(cudaEventRecord(g->ev_start, g->stream));
    return HC_OK;
}
hc_status solve_end(hc_graph *g, const SolveOut *out, SolveResult *res) {
    HC_CUDA_TRY(cudaEventRecord(g->ev_stop, g->stream));
    HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
    if (out->err) return fail((hc_status)out->err, "PageRank: device run ended with status %d", out->err);
    res->iters = out->iters;
    res->done = out->done;
    res->l1 = out->l1;
    res->changed = out->changed;
    HC_CUDA_TRY(cudaEventElapsedTime(&res->ms, g->ev_start, g->ev_stop));
    return HC_OK;
}

hc_status run_solve(hc_graph *g, SweepArgs a, const PrPlanDev &plan, SolveFn fn, float *x[2], float *gv[2],
                    SolveResult *res, float cheb_rho = 0.f, float *final_x = nullptr) {
    for (int k = 0; k < 2; k++) {
        a.x[k] = x[k];
        a.g[k] = gv ? gv[k] : x[k];
    }
    a.cheb_rho = cheb_rho;
    a.final_x = final_x;
    SolveOut *out = nullptr;
    HC_TRY(solve_begin(g, a, &out));
    do {
        HC_TRY(fn(g, a, plan, out));
        HC_TRY(solve_end(g, out, res));
        a.first_iter = out->iters;
        a.first_omega = out->omega;
    } while (!res->done);
    return HC_OK;
}

// ------------------------------------------------- adjoint by conjugate gradients
// For a reversible walk (symmetric weights S, weighted degrees s, D = diag(s))
// the adjoint equation lambda = c + d D^-1 S lambda is, multiplied by D, the
// symmetric positive definite system (D - d S) lambda = D c, solved here by
// conjugate gradients with the diagonal preconditioner D (Hestenes and
// Stiefel, 1952).  The preconditioned residual z = D^-1 r equals the Jacobi
// residual c + d A^T lambda - lambda, so the stopping rule is the same as the
// sweeps'.  Rows without weight (s = 0) keep lambda = c.  Vectors are fp32,
// dot products fp64; alpha, beta and the stop decision stay on the device.
// From this many edges on an iteration's phases are launches of their own: the
// vector passes then run with as many threads as suit them and the sweep without
// the loop around it (adjoint solve, Kronecker scale 20: 2.66 ms so, 3.09 ms in one
// launch; scale 18: 1.18 and 1.00 ms).
constexpr int64_t kCgLaunchEdges = 1ll << 23;
// Without hub rows and with rows of up to 40 edges on average, from this many
// (uniform, rows of 32: 2^16 vertices 0.56 ms so, 0.62 in one launch; 2^18 0.89 and
// 1.02; rows of 16: 2^18 0.72 and 0.77, 2^17 0.58 and 0.56; but rows of 48: 2^17 0.62
// and 0.55, 2^18 1.01 and 0.94).
constexpr int64_t kCgFlatEdges = 2000000;
constexpr int64_t kCgFlatRow = 40;

struct CgArgs {
    const float *c;
    float *lam, *r, *p, *sp;
    float rel_tol;  // stop at |z|_1 < rel_tol * |c|_1
    int first_iter;  // pr_cg: 0, or the iteration that this launch goes on with
};

__device__ __forceinline__ float row_weight(const float *rs, int32_t v) {
    const float r = rs[v];
    return r > 0.f ? 1.0f / r : 0.f;
}

// Adds the block's sums of rz and z1 to the iteration's slot (every thread calls it).
__device__ __forceinline__ void add_dots(IterSlot *slot, double rz, double z1) {
    __shared__ double s0[32], s1[32];
    rz = block_sum(rz, s0);
    z1 = block_sum(z1, s1);
    if (threadIdx.x == 0) {
        if (rz != 0.0) atomicAdd(&slot->rz, rz);
        if (z1 != 0.0) atomicAdd(&slot->z1, z1);
    }
}

// This thread's share of the vector passes.
// r = s (c - lambda) + d S lambda, z = r / s, p = z.
__device__ __forceinline__ void cg_start_rows(const SweepArgs &a, const CgArgs &q, int gtid, int nthreads, double &rz,
                                              double &z1, double &c1) {
    for (int v = gtid; v < a.n; v += nthreads) {
        const float sv = row_weight(a.rs, v);
        c1 += fabs((double)q.c[v]);
        if (sv == 0.f) {
            q.lam[v] = q.c[v];
            q.r[v] = 0.f;
            q.p[v] = 0.f;
            continue;
        }
        const float rv = sv * (q.c[v] - q.lam[v]) + a.d * q.sp[v];
        const float zv = rv * a.rs[v];
        q.r[v] = rv;
        q.p[v] = zv;
        rz += (double)rv * zv;
        z1 += fabs((double)zv);
    }
}
// lambda += alpha p, r -= alpha q.
__device__ __forceinline__ void cg_update_rows(const SweepArgs &a, const CgArgs &q, int gtid, int nthreads, float alpha,
                                               double &rz, double &z1) {
    for (int v = gtid; v < a.n; v += nthreads) {
        const float pv = q.p[v];
        const float qv = row_weight(a.rs, v) * pv - a.d * q.sp[v];
        q.lam[v] += alpha * pv;
        const float rv = q.r[v] - alpha * qv;
        q.r[v] = rv;
        const float zv = rv * a.rs[v];
        rz += (double)rv * zv;
        z1 += fabs((double)zv);
    }
}
// p = z + beta p.
__device__ __forceinline__ void cg_direction_rows(const SweepArgs &a, const CgArgs &q, int gtid, int nthreads,
                                                  float beta) {
    for (int v = gtid; v < a.n; v += nthreads) q.p[v] = q.r[v] * a.rs[v] + beta * q.p[v];
}
__device__ __forceinline__ double cg_tol(const SweepArgs &a, const CgArgs &q) {
    return (double)(float)(q.rel_tol * __ldcg(&a.st->slot[0].l1));
}

// The whole solve in one cooperative launch, a grid barrier after each sweep and
// each vector pass (three an iteration).  Paused at the run limit as pr_solve.
template <bool kEW>
__global__ void __launch_bounds__(kPrThreads, kPrBlocks) pr_cg(SweepArgs a, PrPlanDev plan, CgArgs q) {
    __shared__ float s_acc[kPrThreads / 32][32];
    __shared__ double s_c[32];
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
    GridSync *const gs = &a.st->gs;
    float l1;
    int chg;
    __shared__ unsigned long long s_start;
    if (threadIdx.x == 0) s_start = 0ull;
    // The scalars of iteration it stay in slot it (as registers they would spill)
    // and one thread a block reads them: every warp's reads would queue at one L2 line.
    __shared__ float s_coef;  // alpha, then beta
    __shared__ bool s_stop, s_paused;
    int iters = 0, converged = 0;
    bool ok = true, paused = false;
    if (q.first_iter == 0) {
        // S x by the pull sweep with each row's own weights; its residual is p . q.
        sweep_rows<kEW, false, false, false, true>(a, plan, SweepIter{q.lam, q.lam, q.sp, q.sp, 1.f}, s_acc, l1, chg);
        ok = grid_barrier(gs);
        if (ok) {
            double rz = 0.0, z1 = 0.0, c1 = 0.0;
            cg_start_rows(a, q, gtid, nthreads, rz, z1, c1);
            add_dots(&a.st->slot[0], rz, z1);
            __syncthreads();
            c1 = block_sum(c1, s_c);
            if (threadIdx.x == 0 && c1 != 0.0) atomicAdd(&a.st->slot[0].l1, c1);
            ok = grid_barrier(gs);
            converged = ok && (__ldcg(&a.st->slot[0].z1) < cg_tol(a, q) || __ldcg(&a.st->slot[0].rz) <= 0.0);
        }
    } else {
        iters = q.first_iter - 1;
    }
    while (ok && !converged && !paused && iters < a.max_iters) {
        IterSlot *const slot = &a.st->slot[iters + 1];
        past_run_limit(a.st, iters + 1, &s_start);
        sweep_rows<kEW, false, false, false, true>(a, plan, SweepIter{q.p, q.p, q.sp, q.sp, 1.f}, s_acc, l1, chg);
        add_residual(slot, l1, 0);
        if (!(ok = grid_barrier(gs))) break;
        if (threadIdx.x == 0) {
            const double pq = __ldcg(&slot->l1), rz = __ldcg(&slot[-1].rz);
            s_stop = !(pq > 0.0);  // p = 0 (already exact) or a breakdown
            s_coef = (float)(rz / pq);
        }
        __syncthreads();
        if (s_stop) break;
        double nrz = 0.0, nz1 = 0.0;
        cg_update_rows(a, q, gtid, nthreads, s_coef, nrz, nz1);
        add_dots(slot, nrz, nz1);
        if (!(ok = grid_barrier(gs))) break;
        iters++;
        if (threadIdx.x == 0) {
            const double rz = __ldcg(&slot[-1].rz), next = __ldcg(&slot->rz);
            s_coef = (float)(rz > 0.0 ? next / rz : 0.0);
            s_stop = __ldcg(&slot->z1) < cg_tol(a, q);
            s_paused = __ldcg(&a.st->pause_after) == iters + 1;
        }
        __syncthreads();
        converged = s_stop;
        paused = s_paused;
        if (converged || iters == a.max_iters) break;
        // The same thread's entries as above.
        cg_direction_rows(a, q, gtid, nthreads, s_coef);
        ok = grid_barrier(gs);
    }
    paused = paused && !converged && iters < a.max_iters;
    if (gtid == 0) {
        a.out->err = *(volatile int *)&gs->err;
        a.out->iters = iters;
        a.out->done = paused ? 0 : converged ? 1 : 2;
        a.out->l1 = __ldcg(&a.st->slot[iters].z1);
        a.out->changed = 0;
        __threadfence_system();
    }
}

// The same phases as launches of their own (see run_cg).  Iteration it's sums are
// in slot it; launches queued after the end return at once.
template <bool kEW>
__global__ void __launch_bounds__(kPrThreads, kPrBlocks) cg_sweep(SweepArgs a, PrPlanDev plan, CgArgs q, int it) {
    __shared__ float s_acc[kPrThreads / 32][32];
    if (*(volatile int *)&a.st->done) return;
    float l1;
    int chg;
    const float *x = it == 0 ? q.lam : q.p;
    sweep_rows<kEW, false, false, false, true>(a, plan, SweepIter{x, x, q.sp, q.sp, 1.f}, s_acc, l1, chg);
    if (it > 0) add_residual(&a.st->slot[it], l1, 0);
}
__device__ __forceinline__ void cg_report(const SweepArgs &a, int iters, bool converged, double z1) {
    a.st->done = 1;
    a.out->iters = iters;
    a.out->l1 = z1;
    a.out->changed = 0;
    a.out->done = converged ? 1 : 2;
    __threadfence_system();
}
__global__ void cg_start(SweepArgs a, CgArgs q) {
    __shared__ double s_c[32];
    double rz = 0.0, z1 = 0.0, c1 = 0.0;
    cg_start_rows(a, q, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, rz, z1, c1);
    add_dots(&a.st->slot[0], rz, z1);
    __syncthreads();
    c1 = block_sum(c1, s_c);
    if (threadIdx.x == 0 && c1 != 0.0) atomicAdd(&a.st->slot[0].l1, c1);
}
__global__ void cg_update(SweepArgs a, CgArgs q, int it) {
    if (*(volatile int *)&a.st->done) return;
    const double rz = __ldcg(&a.st->slot[it - 1].rz), pq = __ldcg(&a.st->slot[it].l1);
    if (!(pq > 0.0)) return;  // cg_direction stops
    double nrz = 0.0, nz1 = 0.0;
    cg_update_rows(a, q, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x, (float)(rz / pq), nrz, nz1);
    add_dots(&a.st->slot[it], nrz, nz1);
}
// it 0: only the test after the start.
__global__ void cg_direction(SweepArgs a, CgArgs q, int it) {
    if (*(volatile int *)&a.st->done) return;
    const bool first = blockIdx.x == 0 && threadIdx.x == 0;
    const double nrz = __ldcg(&a.st->slot[it].rz), z1 = __ldcg(&a.st->slot[it].z1), tol = cg_tol(a, q);
    if (it == 0) {
        if (first && (z1 < tol || nrz <= 0.0)) cg_report(a, 0, true, z1);
        return;
    }
    if (!(__ldcg(&a.st->slot[it].l1) > 0.0)) {  // p = 0 (already exact) or a breakdown
        if (first) cg_report(a, it - 1, false, __ldcg(&a.st->slot[it - 1].z1));
        return;
    }
    if (z1 < tol || it >= a.max_iters) {
        if (first) cg_report(a, it, z1 < tol, z1);
        return;
    }
    const double rz = __ldcg(&a.st->slot[it - 1].rz);
    cg_direction_rows(a, q, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x,
                      (float)(rz > 0.0 ? nrz / rz : 0.0));
}

template <bool kEW>
hc_status launch_cg(hc_graph *g, SweepArgs &a, const PrPlanDev &plan, CgArgs &q, volatile SolveOut *out) {
    const bool flat = plan.n_tasks == 0 && g->M >= kCgFlatEdges && g->M <= kCgFlatRow * g->n_active;
    if (flat || g->M >= kCgLaunchEdges) {
        const int grid = g->sm_count * 4, sweep_grid = g->sm_count * kPrBlocks;
        auto sweep = [&](int it) { cg_sweep<kEW><<<sweep_grid, kPrThreads, 0, g->stream>>>(a, plan, q, it); ::hc::count_launch(); };
        auto direction = [&](int it) { cg_direction<<<grid, kPrThreads, 0, g->stream>>>(a, q, it); ::hc::count_launch(); };
        sweep(0);
        { cg_start<<<grid, kPrThreads, 0, g->stream>>>(a, q); ::hc::count_launch(); }
        direction(0);
        // Launches are queued in rounds, the host looking once per round.
        constexpr int kRound = 4;
        for (int it = 1; it <= a.max_iters && !out->done;) {
            for (int k = 0; k < kRound && it <= a.max_iters; k++, it++) {
                sweep(it);
                { cg_update<<<grid, kPrThreads, 0, g->stream>>>(a, q, it); ::hc::count_launch(); }
                direction(it);
            }
            HC_CUDA_TRY(cudaGetLastError());
            HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
        }
        return HC_OK;
    }
    static int bps = 0;
    // Each thread sums its rows' share of p . q, so the grid is part of the
    // rounding: one size for every graph (see the row plans).
    return launch_solve(g, (const void *)pr_cg<kEW>, &bps, a, plan, true, &q);
}

// Solves the adjoint into lam (which holds the start) with the row plan's
// sweep for S x.  `work` holds 3 vectors of n floats.
hc_status run_cg(hc_graph *g, const PrPlanDev &plan, bool weighted, const float *c, float *lam, float d, float rel_tol,
                 int max_iters, float *work, float *partials, unsigned *hub_count, SolveResult *res) {
    const int64_t n = g->N;
    CgArgs q{c, lam, work, work + n, work + 2 * n, rel_tol, 0};
    SweepArgs a{};
    a.index = g->index.as<int64_t>();
    a.nbr = g->nbr.as<int32_t>();
    a.ew = weighted ? pr_weights(g) : nullptr;
    a.d = d;
    a.rs = weighted ? g->inv_wsum.as<float>() : g->inv_deg.as<float>();
    a.partials = partials;
    a.hub_count = hub_count;
    a.max_iters = max_iters;
    a.n = g->N;
    a.n_active = g->n_active;
    SolveOut *out = nullptr;
    HC_TRY(solve_begin(g, a, &out));
    do {
        HC_TRY(weighted ? launch_cg<true>(g, a, plan, q, out) : launch_cg<false>(g, a, plan, q, out));
        HC_TRY(solve_end(g, out, res));
        q.first_iter = out->iters + 1;
    } while (!res->done);
    res->done = res->done == 1;
    return HC_OK;
}

// A multi-column call whose workspace cannot be had (columns are padded to a
// multiple of four, five matrices of them): its columns in two halves, each a call
// of its own into a matrix on the device, from where they go to their places.
template <class F>
hc_status columns_in_halves(hc_graph *g, int K, float *scores, hc_pr_stats *stats, F solve) {
    const int64_t n = g->N;
    g->ws_pr.release();
    hc_pr_stats all{};
    all.converged = 1;
    for (int c0 = 0, h = 0; h < 2; h++) {
        const int k = h == 0 ? (K + 1) / 2 : K - c0;
        DevBuf out;
        HC_TRY(out.ensure((size_t)n * k * 4));
        hc_pr_stats st{};
        HC_TRY(solve(c0, k, out.as<float>(), &st));
        HC_CUDA_TRY(cudaMemcpy2DAsync(scores + c0, (size_t)K * 4, out.ptr, (size_t)k * 4, (size_t)k * 4, n,
                                      cudaMemcpyDefault, g->stream));
        HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
        all.iterations = std::max(all.iterations, st.iterations);
        all.converged = all.converged && st.converged;
        all.residual_l1 = std::max(all.residual_l1, st.residual_l1);
        all.ms += st.ms;
        all.bytes_model += st.bytes_model;
        c0 += k;
    }
    if (stats) *stats = all;
    return HC_OK;
}

void fill_opts(const hc_pr_opts *opts, hc_pr_opts *o) {
    hc_pr_opts d{};
    if (opts) d = *opts;
    if (d.damping <= 0.f) d.damping = 0.85f;
    if (d.max_iters <= 0) d.max_iters = 50;
    if (d.tol_l1 < 0.f) d.tol_l1 = 0.f;
    if (d.eps_vertex < 0.f) d.eps_vertex = 0.f;
    if (d.tol_l1 == 0.f && d.eps_vertex == 0.f) d.tol_l1 = 1e-4f;
    *o = d;
}

}  // namespace
}  // namespace hc

using namespace hc;

extern "C" hc_status hc_pr_forward(hc_graph *g, const float *teleport, int32_t ncols, float *scores_out,
                                   const hc_pr_opts *opts, hc_pr_stats *stats) {
    clear_error();
    HC_TRY(activate(g));
    ReclaimScope reclaim_scope(g, kKeepPrWeighted);
    if (ncols < 1 || !scores_out) return fail(HC_ERR_INVALID_ARG, "hc_pr_forward: bad ncols / output");
    if (ncols > 1 && !teleport) return fail(HC_ERR_INVALID_ARG, "hc_pr_forward: ncols > 1 needs a teleport matrix");
    hc_pr_opts o;
    fill_opts(opts, &o);
    if (o.max_iters > kMaxIterSlots - 1) o.max_iters = kMaxIterSlots - 1;
    if (stats) std::memset(stats, 0, sizeof(*stats));
    HC_TRY(after_default_stream(g));
    const bool weighted = o.weighted != 0;
    HC_TRY(ensure_pr_derived(g, weighted));
    // A single-column call builds the adjoint's plan too: a training step wants both,
    // and the offsets are read once.
    HC_TRY(ensure_plans(g, ncols > 1 ? kPlanSpmm : kPlanPr | kPlanBase));
    const int partial_slots = g->pr_partial_slots;
    const PrPlanDev plan = g->pr_view;
    const int64_t n = g->N;
    HC_TRY(g->ws_ctl.ensure(sizeof(IterState) + 4096));

    if (ncols > 1) {
        // Dense multi-column form.
        const int K = ncols;
        if (K > 256) return fail(HC_ERR_UNSUPPORTED, "hc_pr_forward: at most 256 columns per call");
        const int S = spmm_stride(K);
        const size_t nk = (size_t)n * S;
        const size_t slots = (size_t)g->spmm_partial_slots + 1;
        const size_t bytes = 5 * nk * sizeof(float) + slots * S * sizeof(float) +
                             (size_t)(g->spmm_view.n_hub + 1) * 4 + (size_t)S * 8 + 4096;
        const hc_status room = g->ws_pr.ensure(bytes);
        if (room == HC_ERR_OOM) {
            clear_error();
            return columns_in_halves(g, K, scores_out, stats, [&](int c0, int k, float *out, hc_pr_stats *st) {
                DevBuf t;
                HC_TRY(t.ensure((size_t)n * k * 4));
                HC_CUDA_TRY(cudaMemcpy2DAsync(t.ptr, (size_t)k * 4, teleport + c0, (size_t)K * 4, (size_t)k * 4, n,
                                              cudaMemcpyDefault, g->stream));
                return hc_pr_forward(g, t.as<float>(), k, out, opts, st);
            });
        }
        HC_TRY(room);
        char *p = g->ws_pr.as<char>();
        auto take = [&](size_t b) {
            char *r = p;
            p += (b + 255) / 256 * 256;
            return r;
        };
        float *basev = (float *)take(nk * 4);
        float *x[2] = {(float *)take(nk * 4), (float *)take(nk * 4)};
        float *gv[2] = {(float *)take(nk * 4), (float *)take(nk * 4)};
        float *partials = (float *)take(slots * S * 4);
        unsigned *hub_count = (unsigned *)take((size_t)(g->spmm_view.n_hub + 1) * 4);
        double *col_l1 = (double *)take((size_t)S * 8);
        // Host matrices cross PCIe whole and are padded or packed on the device: a 2-D
        // copy of rows of a few floats goes row by row (uniform, 2^17 vertices, 33
        // columns, both matrices in host memory: 14.6 ms a call, 1.8 ms so).
        const float *t = teleport;
        if (!is_device_pointer(teleport)) {
            HC_TRY(copy_in(x[1], teleport, (size_t)n * K * 4, g->stream));
            t = x[1];
        }
        { spmm_pad_base<<<g->sm_count * 8, 256, 0, g->stream>>>(g->N, K, t, 1.0f - o.damping, basev); ::hc::count_launch(); }
        HC_CUDA_TRY(cudaMemsetAsync(hub_count, 0, (size_t)(g->spmm_view.n_hub + 1) * 4, g->stream));
        const float *ps = weighted ? nullptr : g->inv_deg.as<float>();
        { spmm_init<<<g->sm_count * 8, 256, 0, g->stream>>>(g->N, K, basev, nullptr, nullptr, nullptr, o.damping, ps,
                                                          x[0], gv[0], x[1], gv[1], g->n_active); ::hc::count_launch(); }
        HC_CUDA_TRY(cudaGetLastError());
        SpmmArgs a{};
        a.index = g->index.as<int64_t>();
        a.nbr = g->nbr.as<int32_t>();
        a.ew = weighted ? g->wtn.as<float>() : nullptr;
        a.basev = basev;
        a.d = o.damping;
        a.ps = ps;
        a.partials = partials;
        a.hub_count = hub_count;
        a.col_l1 = col_l1;
        a.K = K;
        a.S = S;
        a.n_active = g->n_active;
        HC_CUDA_TRY(cudaEventRecord(g->ev_start, g->stream));
        int it = 0;
        std::vector<double> hl1(K);
        bool conv = false;
        for (; it < o.max_iters && !conv; it++) {
            a.gin = weighted ? x[it & 1] : gv[it & 1];
            a.xin = x[it & 1];
            a.xout = x[(it + 1) & 1];
            a.gout = weighted ? a.xout : gv[(it + 1) & 1];
            HC_CUDA_TRY(cudaMemsetAsync(col_l1, 0, (size_t)K * 8, g->stream));
            launch_spmm(g, a, nullptr);
            HC_CUDA_TRY(cudaGetLastError());
            HC_CUDA_TRY(cudaMemcpyAsync(hl1.data(), col_l1, (size_t)K * 8, cudaMemcpyDeviceToHost, g->stream));
            HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
            double mx = 0;
            for (double v : hl1) mx = std::max(mx, v);
            conv = o.tol_l1 > 0.f && mx < (double)o.tol_l1;
        }
        HC_CUDA_TRY(cudaEventRecord(g->ev_stop, g->stream));
        const bool dev_out = is_device_pointer(scores_out);
        float *dense = dev_out ? scores_out : basev;
        { spmm_unpad<<<g->sm_count * 8, 256, 0, g->stream>>>(g->N, K, x[it & 1], dense); ::hc::count_launch(); }
        HC_CUDA_TRY(cudaGetLastError());
        if (!dev_out) HC_TRY(copy_out(scores_out, dense, (size_t)n * K * 4, g->stream));
        HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
        float ms = 0;
        HC_CUDA_TRY(cudaEventElapsedTime(&ms, g->ev_start, g->ev_stop));
        if (stats) {
            stats->iterations = it;
            stats->converged = conv;
            double mx = 0;
            for (double v : hl1) mx = std::max(mx, v);
            stats->residual_l1 = (float)mx;
            stats->ms = ms;
            stats->bytes_model = (double)it * (8.0 * (n + 1) + 4.0 * g->M * (weighted ? 2 : 1) +
                                               12.0 * (double)n * K);
        }
        return HC_OK;
    }

    const size_t bytes = 5 * (size_t)n * 4 + (size_t)(partial_slots + 1) * 4 + (size_t)(plan.n_hub + 1) * 4 + 4096;
    HC_TRY(g->ws_pr.ensure(bytes));
    char *p = g->ws_pr.as<char>();
    auto take = [&](size_t b) {
        char *r = p;
        p += (b + 255) / 256 * 256;
        return r;
    };
    float *basev = (float *)take(n * 4);
    float *x[2] = {(float *)take(n * 4), (float *)take(n * 4)};
    float *gv[2] = {(float *)take(n * 4), (float *)take(n * 4)};
    float *partials = (float *)take((size_t)(partial_slots + 1) * 4);
    unsigned *hub_count = (unsigned *)take((size_t)(plan.n_hub + 1) * 4);
    HC_CUDA_TRY(cudaMemsetAsync(hub_count, 0, (size_t)(plan.n_hub + 1) * 4, g->stream));
    bool cheb = false;
    if (o.accel == 1) HC_TRY(ensure_pr_symmetry(g, weighted, &cheb));
    const bool basevec = teleport != nullptr;
    if (basevec) {
        HC_TRY(copy_in(basev, teleport, n * 4, g->stream));
        { scale_vec<<<g->sm_count * 8, 256, 0, g->stream>>>(basev, 1.0f - o.damping, basev, (size_t)g->N); ::hc::count_launch(); }
    }
    // Uniform teleport: base (1-d)/N as the reference computes it
    // (src/kernels/gpu/pr.cuh:152), start from 1/N (src/kernels/cpu/pr.cuh:39).
    // A teleport vector t starts from t itself (base / (1-d)), which has the
    // fixed point's mass, so the error has no part in the slowest mode.
    const float base_scalar = (1.0f - o.damping) / (float)g->N;
    const float *ps = weighted ? nullptr : g->inv_deg.as<float>();
    { pr_init<<<g->sm_count * 8, 256, 0, g->stream>>>(g->N, basevec ? basev : nullptr, base_scalar,
                                                    basevec ? 0.f : 1.0f / (float)g->N, basevec ? basev : nullptr,
                                                    basevec ? 1.0f / (1.0f - o.damping) : 1.0f, ps, x[0], weighted ? nullptr : gv[0], x[1],
                                                    weighted ? nullptr : gv[1], g->n_active); ::hc::count_launch(); }
    HC_CUDA_TRY(cudaGetLastError());
    SweepArgs a{};
    a.index = g->index.as<int64_t>();
    a.nbr = g->nbr.as<int32_t>();
    a.ew = weighted ? g->wtn.as<float>() : nullptr;
    a.basev = basev;
    a.base_scalar = base_scalar;
    a.d = o.damping;
    a.rs = nullptr;
    a.ps = ps;
    a.partials = partials;
    a.hub_count = hub_count;
    a.tol_l1 = o.tol_l1;
    a.eps = o.eps_vertex > 0.f ? o.eps_vertex : 3.4e38f;
    a.max_iters = o.max_iters;
    a.n = g->N;
    a.n_active = g->n_active;
    SolveFn fn = pick_solve(weighted, false, !weighted, basevec);
    if (!fn) return fail(HC_ERR_UNSUPPORTED, "hc_pr_forward: no sweep for this option set");
    if (o.eps_vertex <= 0.f) a.eps = 3.4e38f;
    SolveResult r;
    // Device scores are written by the solve itself.
    const bool dev_out = is_device_pointer(scores_out);
    HC_TRY(run_solve(g, a, plan, fn, x, weighted ? nullptr : gv, &r, cheb ? o.damping : 0.f,
                     dev_out ? scores_out : nullptr));
    if (!dev_out) {
        HC_TRY(copy_out(scores_out, x[r.iters & 1], n * 4, g->stream));
        HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
    }
    if (stats) {
        stats->iterations = r.iters;
        stats->converged = r.done == 1;
        stats->residual_l1 = (float)r.l1;
        stats->changed = r.changed;
        stats->ms = r.ms;
        stats->bytes_model = (double)r.iters * (8.0 * (n + 1) + 4.0 * g->M * (weighted ? 2 : 1) + 12.0 * n);
    }
    return HC_OK;
}

extern "C" hc_status hc_pr_backward(hc_graph *g, const float *scores, const float *dL_dscores, float *dL_dteleport,
                                    float *dL_dweights, const hc_pr_opts *opts, hc_pr_stats *stats) {
    clear_error();
    HC_TRY(activate(g));
    ReclaimScope reclaim_scope(g, kKeepPrWeighted);
    if (!scores || !dL_dscores) return fail(HC_ERR_INVALID_ARG, "hc_pr_backward: scores and dL/dscores required");
    hc_pr_opts o;
    fill_opts(opts, &o);
    if (o.max_iters > kMaxIterSlots - 1) o.max_iters = kMaxIterSlots - 1;
    if (stats) std::memset(stats, 0, sizeof(*stats));
    HC_TRY(after_default_stream(g));
    const bool weighted = o.weighted != 0;
    HC_TRY(ensure_pr_derived(g, weighted));
    HC_TRY(ensure_plans(g, kPlanBase));
    const int partial_slots = g->base_partial_slots;
    const PrPlanDev plan = g->base_view;
    const int64_t n = g->N;
    // cvec, lam[2], xs, spare and the three vectors of the CG solve.
    const size_t bytes = 8 * (size_t)n * 4 + (size_t)(partial_slots + 1) * 4 + (size_t)(plan.n_hub + 1) * 4 + 8192;
    HC_TRY(g->ws_pr.ensure(bytes));
    char *p = g->ws_pr.as<char>();
    auto take = [&](size_t b) {
        char *r = p;
        p += (b + 255) / 256 * 256;
        return r;
    };
    float *cvec = (float *)take(n * 4);
    float *lam[2] = {(float *)take(n * 4), (float *)take(n * 4)};
    float *xs = (float *)take(n * 4);
    float *spare = (float *)take(n * 4);
    float *cg_work = (float *)take(3 * n * 4);  // r, p and S p of the conjugate-gradient solve
    float *partials = (float *)take((size_t)(partial_slots + 1) * 4);
    unsigned *hub_count = (unsigned *)take((size_t)(plan.n_hub + 1) * 4);
    HC_CUDA_TRY(cudaMemsetAsync(hub_count, 0, (size_t)(plan.n_hub + 1) * 4, g->stream));
    HC_TRY(copy_in(cvec, dL_dscores, n * 4, g->stream));
    HC_TRY(copy_in(xs, scores, n * 4, g->stream));
    // lambda_0 = c / (1-d); isolated vertices keep lambda = c.  With
    // symmetric weights the walk's stationary vector is the weighted degree
    // s, and the fixed point has s.lambda = s.c / (1-d) on every connected
    // component: this start already carries that, so the mode that decays
    // only at rate d (eigenvalue 1 of the walk) is absent from the start.
    // Any start converges to the same fixed point; this one converges fastest.
    { pr_init<<<g->sm_count * 8, 256, 0, g->stream>>>(g->N, cvec, 0.f, 0.f, cvec, 1.0f / (1.0f - o.damping), nullptr,
                                                    lam[0], nullptr, lam[1], nullptr, g->n_active); ::hc::count_launch(); }
    HC_CUDA_TRY(cudaGetLastError());
    SweepArgs a{};
    a.index = g->index.as<int64_t>();
    a.nbr = g->nbr.as<int32_t>();
    a.ew = weighted ? pr_weights(g) : nullptr;
    a.basev = cvec;
    a.d = o.damping;
    a.rs = weighted ? g->inv_wsum.as<float>() : g->inv_deg.as<float>();
    a.ps = nullptr;
    a.partials = partials;
    a.hub_count = hub_count;
    a.eps = o.eps_vertex > 0.f ? o.eps_vertex : 3.4e38f;
    a.max_iters = o.max_iters;
    a.n = g->N;
    a.n_active = g->n_active;
    SolveFn fn = pick_solve(weighted, true, false, true);
    // lambda = c + d A^T lambda.  For a reversible walk (symmetric weights)
    // A^T = D^-1 S is similar to a symmetric matrix with spectrum in [-1, 1]:
    // conjugate gradients on (D - d S) lambda = D c (accel 0 / 1), or Chebyshev
    // weights on the Jacobi sweeps, whose operator's spectrum lies in [-d, d]
    // (accel 2).  Otherwise, and with accel -1, plain Jacobi sweeps.
    bool sym = false;
    if (o.accel >= 0) HC_TRY(ensure_pr_symmetry(g, weighted, &sym));
    SolveResult r;
    float *lfin;
    if (sym && o.accel != 2) {
        HC_CUDA_TRY(cudaMemsetAsync(cg_work + 2 * n, 0, n * 4, g->stream));  // S p rows without edges stay 0
        HC_TRY(run_cg(g, plan, weighted, cvec, lam[0], o.damping, o.tol_l1, o.max_iters, cg_work, partials,
                      hub_count, &r));
        lfin = lam[0];
    } else {
        // The L1 rule is relative to sum |dL/dx| (lambda scales with it).
        HC_TRY(g->pinned.ensure(64));
        double *hacc = g->pinned.as<double>();
        double *dacc = reinterpret_cast<double *>(spare);  // scratch until the solve ends
        HC_CUDA_TRY(cudaMemsetAsync(dacc, 0, sizeof(double), g->stream));
        { sum_abs<<<g->sm_count * 4, 256, 0, g->stream>>>(cvec, g->N, dacc); ::hc::count_launch(); }
        HC_CUDA_TRY(cudaMemcpyAsync(hacc, dacc, sizeof(double), cudaMemcpyDeviceToHost, g->stream));
        HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
        a.tol_l1 = (float)(o.tol_l1 * *hacc);
        HC_TRY(run_solve(g, a, plan, fn, lam, nullptr, &r, sym ? o.damping : 0.f));
        lfin = lam[r.iters & 1];
    }
    HC_CUDA_TRY(cudaEventRecord(g->ev_start, g->stream));
    if (dL_dteleport) {
        const bool dev = is_device_pointer(dL_dteleport);
        float *dst = dev ? dL_dteleport : spare;
        { scale_vec<<<g->sm_count * 8, 256, 0, g->stream>>>(lfin, 1.0f - o.damping, dst, (size_t)g->N); ::hc::count_launch(); }
        HC_CUDA_TRY(cudaGetLastError());
        if (!dev) HC_TRY(copy_out(dL_dteleport, spare, n * 4, g->stream));
    }
    if (dL_dweights) {
        const bool dev = is_device_pointer(dL_dweights);
        float *dst = dL_dweights;
        if (!dev) {
            HC_TRY(g->ws_out0.ensure(sizeof(float) * (size_t)std::max<int64_t>(g->M, 1)));
            dst = g->ws_out0.as<float>();
        }
        const float *rsv = weighted ? g->inv_wsum.as<float>() : g->inv_deg.as<float>();
        { pr_edge_grad<<<g->sm_count * 8, kPrThreads, 0, g->stream>>>(plan, a.index, a.nbr, rsv, xs, lfin, cvec,
                                                                      o.damping, g->n_active, dst); ::hc::count_launch(); }
        HC_CUDA_TRY(cudaGetLastError());
        if (!dev) HC_TRY(copy_out(dL_dweights, dst, sizeof(float) * (size_t)g->M, g->stream));
    }
    HC_CUDA_TRY(cudaEventRecord(g->ev_stop, g->stream));
    HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
    float ms2 = 0;
    HC_CUDA_TRY(cudaEventElapsedTime(&ms2, g->ev_start, g->ev_stop));
    if (stats) {
        stats->iterations = r.iters;
        stats->converged = r.done == 1;
        stats->residual_l1 = (float)r.l1;
        stats->changed = r.changed;
        stats->ms = r.ms + ms2;
        stats->bytes_model = (double)r.iters * (8.0 * (n + 1) + 4.0 * g->M * (weighted ? 2 : 1) + 12.0 * n) +
                             (dL_dweights ? (8.0 * (n + 1) + 4.0 * g->M * (weighted ? 3 : 2) + 8.0 * n) : 0.0);
    }
    return HC_OK;
}

extern "C" hc_status hc_ppr_batched(hc_graph *g, const int32_t *seed_offsets, const int32_t *seeds, int32_t ncols,
                                    float *scores_out, const hc_pr_opts *opts, hc_pr_stats *stats) {
    clear_error();
    HC_TRY(activate(g));
    ReclaimScope reclaim_scope(g, kKeepPrWeighted | kKeepBatch);
    if (ncols < 1 || ncols > 256 || !seed_offsets || !seeds || !scores_out)
        return fail(HC_ERR_INVALID_ARG, "hc_ppr_batched: bad arguments (1 <= ncols <= 256)");
    hc_pr_opts o;
    fill_opts(opts, &o);
    if (stats) std::memset(stats, 0, sizeof(*stats));
    const bool weighted = o.weighted != 0;
    HC_TRY(ensure_pr_derived(g, weighted));
    HC_TRY(ensure_plans(g, kPlanPr | kPlanSpmm));
    const int partial_slots = g->pr_partial_slots;
    const PrPlanDev plan = g->pr_view;
    std::vector<int32_t> off(ncols + 1);
    HC_CUDA_TRY(cudaMemcpy(off.data(), seed_offsets, sizeof(int32_t) * (ncols + 1), cudaMemcpyDefault));
    if (off[0] != 0) return fail(HC_ERR_INVALID_ARG, "hc_ppr_batched: seed_offsets[0] must be 0");
    for (int c = 0; c < ncols; c++)
        if (off[c + 1] <= off[c]) return fail(HC_ERR_INVALID_ARG, "hc_ppr_batched: column %d has no seed", c);
    const int32_t nseeds = off[ncols];
    std::vector<int32_t> sd(nseeds);
    HC_CUDA_TRY(cudaMemcpy(sd.data(), seeds, sizeof(int32_t) * nseeds, cudaMemcpyDefault));
    for (int32_t s : sd)
        if (s < 0 || s >= g->N) return fail(HC_ERR_INVALID_ARG, "hc_ppr_batched: seed %d out of range", s);
    const int K = ncols;
    const int64_t n = g->N;
    const int S = spmm_stride(K);
    const size_t nk = (size_t)n * K, ns = (size_t)n * S;
    // One column's partial sums and counters (the tail's sweeps) fit these too.
    const size_t slots = std::max((size_t)g->spmm_partial_slots * S, (size_t)partial_slots) + S;
    const size_t counters = (size_t)std::max(g->spmm_view.n_hub, plan.n_hub) + 1;
    const size_t bytes = 4 * ns * sizeof(float) + slots * 4 + counters * 4 + (size_t)S * 8 + (size_t)n + (size_t)(nseeds + ncols + 1) * 4 + 5 * (size_t)n * 4 + 16384;
    const hc_status room = g->ws_pr.ensure(bytes);
    if (room == HC_ERR_OOM && K == 1) {  // one column: the solve of one column takes less
        clear_error();
        DevBuf t, idx;
        HC_TRY(t.ensure((size_t)n * 4));
        HC_TRY(idx.ensure((size_t)nseeds * 4));
        HC_CUDA_TRY(cudaMemsetAsync(t.ptr, 0, (size_t)n * 4, g->stream));
        HC_CUDA_TRY(cudaMemcpyAsync(idx.ptr, sd.data(), (size_t)nseeds * 4, cudaMemcpyHostToDevice, g->stream));
        { spmm_column_base<<<4, 256, 0, g->stream>>>(idx.as<int32_t>(), 0, nseeds, 1.0f, t.as<float>()); ::hc::count_launch(); }
        HC_CUDA_TRY(cudaGetLastError());
        hc_pr_opts one = o;
        one.eps_vertex = 0.f;
        one.accel = 0;
        return hc_pr_forward(g, t.as<float>(), 1, scores_out, &one, stats);
    }
    if (room == HC_ERR_OOM) {
        clear_error();
        return columns_in_halves(g, K, scores_out, stats, [&](int c0, int k, float *out, hc_pr_stats *st) {
            std::vector<int32_t> part(k + 1);
            for (int c = 0; c <= k; c++) part[c] = off[c0 + c] - off[c0];
            return hc_ppr_batched(g, part.data(), sd.data() + off[c0], k, out, opts, st);
        });
    }
    HC_TRY(room);
    char *p = g->ws_pr.as<char>();
    auto take = [&](size_t b) {
        char *r = p;
        p += (b + 255) / 256 * 256;
        return r;
    };
    float *x[2] = {(float *)take(ns * 4), (float *)take(ns * 4)};
    float *gv[2] = {(float *)take(ns * 4), (float *)take(ns * 4)};
    float *partials = (float *)take(slots * 4);
    unsigned *hub_count = (unsigned *)take(counters * 4);
    double *col_l1 = (double *)take((size_t)S * 8);
    uint8_t *is_seed = (uint8_t *)take((size_t)n);
    int32_t *d_off = (int32_t *)take((size_t)(ncols + 1) * 4);
    int32_t *d_seeds = (int32_t *)take((size_t)nseeds * 4);
    float *col_x[2] = {(float *)take((size_t)n * 4), (float *)take((size_t)n * 4)};
    float *col_g[2] = {(float *)take((size_t)n * 4), (float *)take((size_t)n * 4)};
    float *col_base = (float *)take((size_t)n * 4);
    HC_CUDA_TRY(cudaMemcpyAsync(d_off, off.data(), (ncols + 1) * 4, cudaMemcpyHostToDevice, g->stream));
    HC_CUDA_TRY(cudaMemcpyAsync(d_seeds, sd.data(), (size_t)nseeds * 4, cudaMemcpyHostToDevice, g->stream));
    HC_CUDA_TRY(cudaMemsetAsync(is_seed, 0, (size_t)n, g->stream));
    HC_CUDA_TRY(cudaMemsetAsync(hub_count, 0, counters * 4, g->stream));
    { mark_seeds<<<64, 256, 0, g->stream>>>(d_seeds, nseeds, is_seed); ::hc::count_launch(); }
    const float *ps = weighted ? nullptr : g->inv_deg.as<float>();
    { spmm_init<<<g->sm_count * 8, 256, 0, g->stream>>>(g->N, K, nullptr, d_off, d_seeds, is_seed, o.damping, ps,
                                                      x[0], gv[0], x[1], gv[1], g->n_active); ::hc::count_launch(); }
    HC_CUDA_TRY(cudaGetLastError());
    SpmmArgs a{};
    a.index = g->index.as<int64_t>();
    a.nbr = g->nbr.as<int32_t>();
    a.ew = weighted ? g->wtn.as<float>() : nullptr;
    a.basev = nullptr;
    a.seed_off = d_off;
    a.seed_idx = d_seeds;
    a.d = o.damping;
    a.ps = ps;
    a.partials = partials;
    a.hub_count = hub_count;
    a.col_l1 = col_l1;
    a.K = K;
    a.n_active = g->n_active;
    // Columns converge at their own pace (personalised teleports differ):
    // a column whose L1 change falls below tol is final.  Whenever the live
    // columns fit fewer 32-column chunks, one pass writes the final ones to
    // the output and packs the live ones tighter, so later sweeps gather only
    // live columns.
    const bool dev_out = is_device_pointer(scores_out);
    float *out = scores_out;
    if (!dev_out) {
        HC_TRY(g->ws_out0.ensure(nk * 4));
        out = g->ws_out0.as<float>();
    }
    HC_TRY(g->ws_src.ensure((size_t)2 * K * 4));
    int32_t *d_map = g->ws_src.as<int32_t>();
    int32_t *d_newpos = d_map + K;
    std::vector<int32_t> hmap(K), hpos(K);
    for (int c = 0; c < K; c++) hmap[c] = c;
    HC_CUDA_TRY(cudaMemcpyAsync(d_map, hmap.data(), (size_t)K * 4, cudaMemcpyHostToDevice, g->stream));
    a.col_map = d_map;
    auto repack = [&](int cur, int kw, int nkw) -> hc_status {
        HC_CUDA_TRY(cudaMemcpyAsync(d_newpos, hpos.data(), (size_t)kw * 4, cudaMemcpyHostToDevice, g->stream));
        {
            spmm_repack<<<g->sm_count * 8, 256, 0, g->stream>>>(g->N, kw, x[cur], d_newpos, d_map, K, out, nkw,
                                                                x[cur ^ 1], weighted ? nullptr : gv[cur ^ 1], ps);
            ::hc::count_launch();
        }
        HC_CUDA_TRY(cudaGetLastError());
        // Rows without edges (past n_active) are never written by a sweep:
        // give the buffer the next sweep writes their values in the new layout.
        if (nkw > 0 && g->n_active < g->N)
            HC_CUDA_TRY(cudaMemcpyAsync(x[cur] + (size_t)g->n_active * spmm_stride(nkw),
                                        x[cur ^ 1] + (size_t)g->n_active * spmm_stride(nkw),
                                        (size_t)(g->N - g->n_active) * spmm_stride(nkw) * 4, cudaMemcpyDeviceToDevice,
                                        g->stream));
        return HC_OK;
    };
    // The single-column solver's run_solve records g's events: this call
    // times itself with its own pair.
    cudaEvent_t ev0, ev1;
    HC_CUDA_TRY(cudaEventCreate(&ev0));
    HC_CUDA_TRY(cudaEventCreate(&ev1));
    struct EvGuard {
        cudaEvent_t a, b;
        ~EvGuard() {
            cudaEventDestroy(a);
            cudaEventDestroy(b);
        }
    } ev_guard{ev0, ev1};
    HC_CUDA_TRY(cudaEventRecord(ev0, g->stream));
    int it = 0, cur = 0, kw = K;
    std::vector<double> hl1(K);
    double bytes_model = 0, mx = 0;
    bool conv = false;
    // A few slow columns (a seed set in a small bipartite component converges
    // at rate d) finish on the single-column sweeps, which gather 4 bytes per
    // edge instead of a 32-column row segment.
    constexpr int kSingleCols = 4;
    for (; it < o.max_iters && kw > (K > kSingleCols ? kSingleCols : 0); it++) {
        a.K = kw;
        a.S = spmm_stride(kw);
        a.gin = weighted ? x[cur] : gv[cur];
        a.xin = x[cur];
        a.xout = x[cur ^ 1];
        a.gout = weighted ? a.xout : gv[cur ^ 1];
        HC_CUDA_TRY(cudaMemsetAsync(col_l1, 0, (size_t)kw * 8, g->stream));
        launch_spmm(g, a, is_seed);
        HC_CUDA_TRY(cudaGetLastError());
        bytes_model += 8.0 * (n + 1) + 4.0 * g->M * (weighted ? 2 : 1) + 12.0 * (double)n * kw;
        cur ^= 1;
        HC_CUDA_TRY(cudaMemcpyAsync(hl1.data(), col_l1, (size_t)kw * 8, cudaMemcpyDeviceToHost, g->stream));
        HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
        int live = 0;
        mx = 0;
        for (int c = 0; c < kw; c++) {
            mx = std::max(mx, hl1[c]);
            const bool done = o.tol_l1 > 0.f && hl1[c] < (double)o.tol_l1;
            hpos[c] = done ? -1 : live++;
        }
        if (live == 0) {
            conv = true;
            HC_TRY(repack(cur, kw, 0));  // every column is final
            kw = 0;
        } else if ((live + 31) / 32 < (kw + 31) / 32 || (live <= kSingleCols && kw > kSingleCols)) {
            HC_TRY(repack(cur, kw, live));
            std::vector<int32_t> nmap(live);
            for (int c = 0; c < kw; c++)
                if (hpos[c] >= 0) nmap[hpos[c]] = hmap[c];
            HC_CUDA_TRY(cudaStreamSynchronize(g->stream));  // d_map is read by the repack
            hmap = nmap;
            HC_CUDA_TRY(cudaMemcpyAsync(d_map, hmap.data(), (size_t)live * 4, cudaMemcpyHostToDevice, g->stream));
            cur ^= 1;
            kw = live;
        }
    }
    int tail_iters = 0;
    if (kw > 0 && it < o.max_iters) {
        // Each remaining column continues from its packed values on the
        // single-column sweeps (teleport vector, same stopping rule).
        SweepArgs sa{};
        sa.index = g->index.as<int64_t>();
        sa.nbr = g->nbr.as<int32_t>();
        sa.ew = weighted ? g->wtn.as<float>() : nullptr;
        sa.basev = col_base;
        sa.d = o.damping;
        sa.ps = ps;
        sa.partials = partials;
        sa.hub_count = hub_count;
        sa.tol_l1 = o.tol_l1;
        sa.eps = 3.4e38f;
        sa.max_iters = o.max_iters - it;
        sa.n = g->N;
        sa.n_active = g->n_active;
        SolveFn fn = pick_solve(weighted, false, !weighted, true);
        bool all_conv = true;
        for (int c = 0; c < kw; c++) {
            const int oc = hmap[c];
            HC_CUDA_TRY(cudaMemsetAsync(col_base, 0, (size_t)n * 4, g->stream));
            { spmm_column_base<<<4, 256, 0, g->stream>>>(d_seeds, off[oc], off[oc + 1], 1.0f - o.damping, col_base); ::hc::count_launch(); }
            {
                spmm_take_column<<<g->sm_count * 4, 256, 0, g->stream>>>(g->N, kw, c, x[cur], ps, col_x[0], col_x[1],
                                                                         weighted ? nullptr : col_g[0],
                                                                         weighted ? nullptr : col_g[1]);
                ::hc::count_launch();
            }
            HC_CUDA_TRY(cudaGetLastError());
            SolveResult r;
            HC_TRY(run_solve(g, sa, plan, fn, col_x, weighted ? nullptr : col_g, &r));
            { spmm_put_column<<<g->sm_count * 4, 256, 0, g->stream>>>(g->N, col_x[r.iters & 1], K, oc, out); ::hc::count_launch(); }
            HC_CUDA_TRY(cudaGetLastError());
            tail_iters = std::max(tail_iters, r.iters);
            all_conv = all_conv && r.done == 1;
            mx = std::max(mx, r.l1);
            bytes_model += (double)r.iters * (8.0 * (n + 1) + 4.0 * g->M * (weighted ? 2 : 1) + 12.0 * (double)n);
        }
        conv = all_conv;
        kw = 0;
    }
    if (kw > 0) {  // iteration cap: the live columns as they stand
        for (int c = 0; c < kw; c++) hpos[c] = -1;
        HC_TRY(repack(cur, kw, 0));
    }
    HC_CUDA_TRY(cudaEventRecord(ev1, g->stream));
    if (!dev_out) HC_TRY(copy_out(scores_out, out, nk * 4, g->stream));
    HC_CUDA_TRY(cudaStreamSynchronize(g->stream));
    float ms = 0;
    HC_CUDA_TRY(cudaEventElapsedTime(&ms, ev0, ev1));
    if (stats) {
        stats->iterations = it + tail_iters;
        stats->converged = conv;
        stats->residual_l1 = (float)mx;
        stats->ms = ms;
        stats->bytes_model = bytes_model;
    }
    return HC_OK;
}
