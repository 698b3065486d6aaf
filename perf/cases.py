"""The calls whose speed counts, through the public entry points (hc.Graph).

Graphs are made here with torch from a seed alone: Kronecker (R-MAT, the
construction of hc.gen_kronecker: A=.57 B=C=.19, random permutation,
symmetrised, self loops and duplicates dropped, relabelled by descending
degree), uniform (Erdos-Renyi, the same build) and 4-neighbour grids (road-like:
no hubs, a diameter of rows + cols).  Vertex counts need not be powers of two.
Integer weights are uniform in [1, 255], float weights in (0, 1], both symmetric.
Sources are vertices with at least one edge.

BFS parents are any valid tree (which frontier neighbour claims a vertex first
is not fixed), so every BFS call computes them as a user's does, and the
depths, which are fixed, are what is returned.  BFS depths and SSSP distances
are whole numbers: they have one right value and `exact` leaves them out.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hetero-compute_b200"))

import hc  # noqa: E402

DAMPING = 0.85

_BFS_OPS = ("bfs", "bfs_host", "bfs_batched")
_SSSP_OPS = ("sssp", "sssp_batched")


def listed():
    return [
        # One query on a graph that a service answers while somebody waits: latency and launches.
        dict(name="bfs_kron10_one", op="bfs", graph="kron", nodes=1 << 10, degree=16, count=1),
        # A handful of queries on a mid-sized graph without hubs, odd vertex count.
        dict(name="bfs_uniform18_16", op="bfs", graph="uniform", nodes=250_007, degree=16, count=16),
        # The benchmark's BFS phase: 64 sources on the scale-22 Kronecker graph.
        dict(name="bfs_kron22_64", op="bfs", graph="kron", nodes=1 << 22, degree=16, count=64),
        # One BFS on a road-like graph: two thousand thin levels.
        dict(name="bfs_grid_1023x1025", op="bfs", graph="grid", nodes=1023, degree=1025, count=1),
        # One shortest-path query on a small graph.
        dict(name="sssp_kron12_one", op="sssp", graph="kron", nodes=1 << 12, degree=16, count=1),
        # The benchmark's SSSP phase: 64 sources on the scale-22 Kronecker graph.
        dict(name="sssp_kron22_64", op="sssp", graph="kron", nodes=1 << 22, degree=16, count=64),
        # One shortest-path query on a road-like graph (the grid suite, smaller).
        dict(name="sssp_grid_701x517", op="sssp", graph="grid", nodes=701, degree=517, count=1),
        # The benchmark's PageRank phase.
        dict(name="pagerank_kron22", op="pagerank", graph="kron", nodes=1 << 22, degree=16, count=1),
        # A training step through the weighted PageRank: scores, and the gradients of teleport and weights.
        dict(name="pagerank_grad_kron18", op="pagerank_grad", graph="kron", nodes=260_101, degree=16, count=1),
        # Personalised PageRank for a batch of users (three seeds each).
        dict(name="ppr_kron18_48", op="ppr", graph="kron", nodes=1 << 18, degree=16, count=48),
        # All sources of an offline job in one batched call each.
        dict(name="bfs_batched_kron20_512", op="bfs_batched", graph="kron", nodes=1 << 20, degree=16, count=512),
        dict(name="sssp_batched_kron20_200", op="sssp_batched", graph="kron", nodes=1 << 20, degree=16, count=200),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(("bfs", "bfs", "bfs_host", "sssp", "sssp", "pagerank", "pagerank_grad", "ppr", "bfs_batched",
                     "sssp_batched"))
    kinds = {"bfs": ("kron", "kron", "uniform", "grid"), "sssp": ("kron", "kron", "uniform", "grid")}
    graph = rng.choice(kinds.get(op, ("kron", "kron", "uniform")))
    if graph == "grid":
        side = 700 if op == "sssp" else 1024
        return dict(op=op, graph=graph, nodes=_log_uniform(rng, 24, side), degree=_log_uniform(rng, 24, side),
                    count=rng.choice((1, 1, 2, 3)))
    degree = rng.choice((8, 16, 16, 24))
    top = {"bfs": 21.5, "bfs_host": 19, "sssp": 21, "pagerank": 22, "pagerank_grad": 20, "ppr": 18.5,
           "bfs_batched": 20, "sssp_batched": 19.5}[op]
    nodes = _log_uniform(rng, 2 ** 10, 2 ** top) | (1 if rng.random() < 0.7 else 0)
    count = 1
    if op in ("bfs", "bfs_host", "sssp"):
        count = rng.choice((1, 2, 7, 16, 33, 64))
        while nodes * degree * count > 1 << 31:
            count = max(1, count // 2)
    elif op == "ppr":
        count = _log_uniform(rng, 2, 64)
    elif op in ("bfs_batched", "sssp_batched"):
        count = _log_uniform(rng, 33, 512 if op == "bfs_batched" else 256)
    return dict(op=op, graph=graph, nodes=nodes, degree=degree, count=count)


# ------------------------------------------------------------------ inputs

def _mix(x, seed):
    """A 64-bit mixer (the finaliser of SplitMix64, on int64 with wrap-around)."""
    x = x + (seed * 0x1E3779B97F4A7C15 + 0x632BE59BD9B4E019 & 0x7FFFFFFFFFFFFFFF)
    x = (x ^ (x >> 30 & 0x3FFFFFFFF)) * -0x40A7B892E31B1A47
    x = (x ^ (x >> 27 & 0x1FFFFFFFFF)) * -0x6B2FB644ECCEEE15
    return x ^ (x >> 31 & 0x1FFFFFFFF)


def _grid(rows, cols):
    ids = torch.arange(rows * cols, device="cuda", dtype=torch.int64).view(rows, cols)
    pairs = [(ids[:, :-1].reshape(-1), ids[:, 1:].reshape(-1)), (ids[:-1].reshape(-1), ids[1:].reshape(-1))]
    return torch.cat([p[0] for p in pairs]), torch.cat([p[1] for p in pairs])


def _random_pairs(kind, n, degree, gen):
    m = n * degree
    if kind == "uniform":
        return (torch.randint(n, (m,), generator=gen, device="cuda"),
                torch.randint(n, (m,), generator=gen, device="cuda"))
    u = torch.zeros(m, dtype=torch.int64, device="cuda")
    v = torch.zeros(m, dtype=torch.int64, device="cuda")
    for _ in range(max(1, (n - 1).bit_length())):
        r = torch.rand(m, generator=gen, device="cuda")
        u = u * 2 + (r >= 0.76)
        v = v * 2 + ((r >= 0.57) & (r < 0.76) | (r >= 0.95))
    perm = torch.randperm(n, generator=gen, device="cuda")
    return perm[u % n], perm[v % n]


def _csr(case, seed):
    """(index int64[N+1], neighbors int32[M], hash int64[M]) on the GPU; the hash is the same both ways along an edge."""
    gen = torch.Generator(device="cuda")
    # Training runs stay on one graph and change its weights (the gradients then have one shape).
    gen.manual_seed(1 if case["op"] == "pagerank_grad" else seed)
    if case["graph"] == "grid":
        n = case["nodes"] * case["degree"]
        u, v = _grid(case["nodes"], case["degree"])
    else:
        n = case["nodes"]
        u, v = _random_pairs(case["graph"], n, case["degree"], gen)
        keep = u != v
        u, v = u[keep], v[keep]
    key = torch.cat([u * n + v, v * n + u])
    del u, v
    key = torch.sort(key)[0]
    if case["graph"] != "grid":
        first = torch.ones_like(key, dtype=torch.bool)
        torch.ne(key[1:], key[:-1], out=first[1:])
        key = key[first]
        deg = torch.bincount(key // n, minlength=n)
        new = torch.empty(n, dtype=torch.int64, device="cuda")
        new[torch.sort(deg, descending=True, stable=True)[1]] = torch.arange(n, device="cuda")
        key = torch.sort(new[key // n] * n + new[key % n])[0]
    row, col = key // n, key % n
    index = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(torch.bincount(row, minlength=n), 0, out=index[1:])
    h = _mix(torch.minimum(row, col) * n + torch.maximum(row, col), seed)
    return index, col.to(torch.int32), h


def _inputs(case, seed):
    index, nbr, h = _csr(case, seed)
    w = None
    if case["op"] in _SSSP_OPS:
        w = (1 + (h & 0x7FFFFFFF) % 255).to(torch.int32)
    elif case["op"] == "pagerank_grad":
        w = (1 + (h & 0xFFFFF)).to(torch.float32) / float(1 << 20)
    n, k = index.numel() - 1, case["count"]
    rng = np.random.default_rng(seed)
    linked = int((index[1:] > index[:-1]).sum())  # a prefix: vertices are sorted by degree (every vertex on a grid)
    more = {}
    if case["op"] == "pagerank_grad":
        more["dx"] = torch.from_numpy(rng.standard_normal(n).astype(np.float32)).cuda()
    elif case["op"] == "ppr":
        more["off"] = np.arange(k + 1, dtype=np.int32) * 3
        more["seeds"] = rng.integers(0, linked, 3 * k).astype(np.int32)
        for c in range(k):  # three different ones
            while len(set(more["seeds"][3 * c:3 * c + 3])) < 3:
                more["seeds"][3 * c:3 * c + 3] = rng.integers(0, linked, 3)
    else:
        more["src"] = rng.integers(0, linked, k).astype(np.int32)
    return index, nbr, w, more


def prepare(case, seed):
    index, nbr, w, state = _inputs(case, seed)
    op, n, m, k = case["op"], index.numel() - 1, nbr.numel(), case["count"]
    state["op"] = op
    state["g"] = hc.Graph(index, nbr, w)
    torch.cuda.synchronize()

    def dev(*shape, dtype=torch.int32):
        return torch.empty(shape, dtype=dtype, device="cuda")

    if op == "bfs":
        state["depth"], state["parent"] = dev(k, n), dev(k, n)
    elif op == "bfs_host":
        state["depth"], state["parent"] = (torch.empty((k, n), dtype=torch.int32).pin_memory().numpy()
                                           for _ in range(2))
    elif op == "bfs_batched":
        state["depth"] = dev(k, n)
    elif op in _SSSP_OPS:
        state["dist"] = dev(k, n)
    elif op == "pagerank":
        state["scores"] = dev(n, dtype=torch.float32)
    elif op == "pagerank_grad":
        state["scores"], state["dt"], state["dw"] = (dev(s, dtype=torch.float32) for s in (n, n, m))
    elif op == "ppr":
        state["scores"] = dev(n, k, dtype=torch.float32)
    return state


def run(state):
    g, op = state["g"], state["op"]
    if op in ("bfs", "bfs_host"):
        depth, _, _ = g.bfs(state["src"], state["depth"], state["parent"])
        return depth
    if op == "bfs_batched":
        return g.bfs_batched(state["src"], state["depth"])[0]
    if op == "sssp":
        return g.sssp(state["src"], state["dist"])[0]
    if op == "sssp_batched":
        return g.sssp_batched(state["src"], state["dist"])[0]
    if op == "pagerank":
        return g.pagerank(None, state["scores"], tol_l1=1e-4, max_iters=50)[0]
    if op == "pagerank_grad":
        opts = dict(tol_l1=1e-6, max_iters=200, weighted=True)
        x, _ = g.pagerank(None, state["scores"], **opts)
        dt, dw, _ = g.pagerank_backward(x, state["dx"], dteleport=state["dt"], dweights=state["dw"], **opts)
        return {"scores": x, "dteleport": dt, "dweights": dw}
    return g.ppr_batched(state["off"], state["seeds"], state["scores"], tol_l1=1e-4, max_iters=50)[0]


def work(case):
    """The graph read once and the outputs written once; one addition or comparison per edge and result vector."""
    if case["graph"] == "grid":
        n = case["nodes"] * case["degree"]
        m = 4 * n - 2 * (case["nodes"] + case["degree"])
    else:
        n, m = case["nodes"], 2 * case["nodes"] * case["degree"]
    op, k = case["op"], case["count"]
    graph = 8 * (n + 1) + 4 * m
    if op in ("bfs", "bfs_host"):
        return {"bytes": graph + 8 * n * k, "flops": 0}
    if op == "bfs_batched":
        return {"bytes": graph + 4 * n * k, "flops": 0}
    if op in _SSSP_OPS:
        return {"bytes": graph + 4 * m + 4 * n * k, "flops": m * k}
    if op == "pagerank":
        return {"bytes": graph + 4 * n, "flops": m}
    if op == "pagerank_grad":
        return {"bytes": graph + 4 * m + 4 * m + 12 * n, "flops": 4 * m}
    return {"bytes": graph + 4 * n * k, "flops": m * k}


# ------------------------------------------------------------------ 64 bits

def _spmm(index, nbr, vals, x):
    a = torch.sparse_csr_tensor(index, nbr.to(torch.int64), vals, size=(x.shape[0], x.shape[0]))
    return a @ x


def _iterate(index, nbr, vals, base, x, tol, most):
    """x <- base + d A x until the largest column's L1 change is below tol."""
    for _ in range(most):
        y = base + DAMPING * _spmm(index, nbr, vals, x)
        change = float((y - x).abs().sum(0).max())
        x = y
        if change < tol:
            break
    return x


def exact(case, seed):
    op = case["op"]
    if op in _BFS_OPS or op in _SSSP_OPS:
        return None
    index, nbr, w, more = _inputs(case, seed)
    n, k = index.numel() - 1, case["count"]
    deg = index[1:] - index[:-1]
    col = nbr.to(torch.int64)
    f64 = dict(dtype=torch.float64, device="cuda")
    base = torch.full((n, 1), (1 - DAMPING) / n, **f64)
    if op in ("pagerank", "ppr"):
        vals = (1.0 / deg.clamp(min=1).to(torch.float64))[col]
    else:
        row = torch.repeat_interleave(torch.arange(n, device="cuda"), deg)
        w = w.to(torch.float64)
        s = torch.zeros(n, **f64).index_add_(0, row, w)
        vals = w / s[col]  # symmetric: w(u->v) stands in v's row, divided by u's sum
    if op == "ppr":
        base.zero_()
        t = torch.zeros((n, k), **f64)
        seeds = torch.from_numpy(more["seeds"]).cuda().long()
        t[seeds, torch.arange(k, device="cuda").repeat_interleave(3)] = 1.0 / 3.0
        return _iterate(index, nbr, vals, (1 - DAMPING) * t, t, 1e-13, 300)
    start = torch.where(deg > 0, 1.0 / n, (1 - DAMPING) / n).to(torch.float64)[:, None]
    if op == "pagerank":
        return _iterate(index, nbr, vals, base, start, 1e-4, 50)[:, 0]
    x = _iterate(index, nbr, vals, base, start, 1e-6, 200)[:, 0]
    # The adjoint: lambda = dL/dx + d A^T lambda, A^T holding w / (the row's own sum).
    c = more["dx"].to(torch.float64)[:, None]
    lam = _iterate(index, nbr, w / s[row], c, c / (1 - DAMPING), 1e-11 * float(c.abs().sum()), 400)[:, 0]
    dw = (x / s)[row] * (DAMPING * lam[col] - (lam - c[:, 0])[row])
    return {"scores": x, "dteleport": (1 - DAMPING) * lam, "dweights": dw}
