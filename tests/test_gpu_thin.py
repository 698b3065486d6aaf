"""Thin frontiers: levels and epochs that one block runs alone, at the sizes where they start and stop."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def csr(n, u, v):
    """Symmetric CSR of the pairs (u, v)."""
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    index = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(src, minlength=n), out=index[1:])
    return index, dst[order].astype(np.int32)


def path(n):
    return csr(n, np.arange(n - 1), np.arange(1, n))


def fan(width, tail):
    """A root, `width` vertices next to it through hubs of 100 edges, and `tail` more levels of that width."""
    hubs = (width + 99) // 100
    first = 1 + hubs
    lane = np.arange(width)
    u = [np.zeros(hubs, np.int64), 1 + lane // 100]
    v = [1 + np.arange(hubs), first + lane]
    for t in range(tail):
        u.append(first + t * width + lane)
        v.append(first + (t + 1) * width + lane)
    return csr(first + (tail + 1) * width, np.concatenate(u), np.concatenate(v))


def star_chain(deg, links):
    """A chain of stars: each centre has `deg` edges in all."""
    c = np.arange(links) * deg
    leaves = [c[i] + 1 + np.arange(deg - 2) for i in range(links)]
    u = np.concatenate([np.repeat(c, deg - 2), c[:-1]])
    v = np.concatenate(leaves + [c[1:]])
    return csr(links * deg, u, v)


GRAPHS = {
    "path_3000": lambda: path(3000),            # more levels than one turn of the block
    "path_2": lambda: path(2),
    "fan_1919": lambda: fan(1919, 40),          # around the block's queue capacity
    "fan_1920": lambda: fan(1920, 40),
    "fan_1921": lambda: fan(1921, 40),
    "fan_600": lambda: fan(600, 9),
    "star_127": lambda: star_chain(127, 30),    # around the longest row it takes
    "star_128": lambda: star_chain(128, 30),
    "star_129": lambda: star_chain(129, 30),
    "star_300": lambda: star_chain(300, 12),
}


@pytest.mark.parametrize("direction", [0, 1, 2])
@pytest.mark.parametrize("name", sorted(GRAPHS))
def test_bfs_thin_levels(name, direction):
    import hc
    index, nbr = GRAPHS[name]()
    n = len(index) - 1
    g = hc.Graph(index, nbr)
    sources = [0, n - 1, n // 2]
    for stats in (False, True):
        depth, parent, _ = g.bfs(sources, direction=direction, stats=stats)
        for i, s in enumerate(sources):
            want = oracle.bfs_depth(index, nbr, s)
            assert np.array_equal(depth[i], want)
            assert oracle.verify_bfs_parents(index, nbr, want, parent[i], s)[0] == 0
    g.close()


@pytest.mark.parametrize("scale,count", [(6, 1), (6, 300), (10, 7), (13, 65), (17, 18)])
@pytest.mark.parametrize("host", [False, True])
def test_bfs_sources_at_a_time(scale, count, host):
    """Sources run several at a time, in one launch or (more than one launch takes, host outputs) several."""
    import torch

    import hc
    host_g = hc.gen_kronecker(scale, 16, 3)
    n = host_g.num_nodes
    g = hc.Graph.from_host(host_g)
    picks = np.random.default_rng(scale).integers(0, n, count).astype(np.int32)  # isolated and repeated ones too
    if host:
        depth, parent, _ = g.bfs(picks)
        only = g.bfs(picks, want_depth=False)[1]
    else:
        out = [torch.full((count, n), 7, dtype=torch.int32, device="cuda") for _ in range(3)]
        depth, parent, _ = g.bfs(picks, out[0], out[1])
        only = g.bfs(picks, None, out[2], want_depth=False)[1].cpu().numpy()
        depth, parent = depth.cpu().numpy(), parent.cpu().numpy()
    for i in sorted({0, count // 2, count - 1, *range(0, count, 17)}):
        want = oracle.bfs_depth(host_g.index, host_g.neighbors, picks[i])
        assert np.array_equal(depth[i], want)
        for p in (parent[i], only[i]):
            assert oracle.verify_bfs_parents(host_g.index, host_g.neighbors, want, p, picks[i])[0] == 0
    g.close()


def weights(index, nbr, top):
    """Symmetric integer weights in [0, top]: a hash of the unordered pair."""
    row = np.repeat(np.arange(len(index) - 1, dtype=np.int64), np.diff(index))
    lo, hi = np.minimum(row, nbr), np.maximum(row, nbr)
    h = (lo * 2654435761 + hi * 40503 + 12345) & 0x7FFFFFFF
    return ((h >> 7) % (top + 1)).astype(np.int32)


def shuffled(index, nbr, seed):
    """The same graph under a random relabelling: rows of all lengths side by side."""
    n = len(index) - 1
    perm = np.random.default_rng(seed).permutation(n)
    row = np.repeat(np.arange(n), np.diff(index))
    u, v = perm[row], perm[nbr]
    keep = u < v
    return csr(n, u[keep], v[keep])


@pytest.mark.parametrize("top", [1, 255, 70000])
@pytest.mark.parametrize("name", sorted(GRAPHS) + ["mixed"])
def test_sssp_thin_epochs(name, top):
    import hc
    if name == "mixed":  # unsorted: long rows inside groups of short ones
        k = hc.gen_kronecker(12, 16, 5)
        index, nbr = shuffled(k.index, k.neighbors, 1)
    else:
        index, nbr = GRAPHS[name]()
    w = weights(index, nbr, top)
    n = len(index) - 1
    g = hc.Graph(index, nbr, w)
    sources = [0, n - 1, n // 2]
    want = [oracle.sssp_dijkstra(index, nbr, w, s) for s in sources]
    for kw in ({}, {"delta": -1}, {"delta": 1 + top // 8, "pull_alpha": -1}, {"pull_alpha": 1 << 20}, {"stats": True}):
        dist, parent, _ = g.sssp(sources, want_parent=True, **kw)
        for i, s in enumerate(sources):
            assert np.array_equal(dist[i], want[i]), (kw, s)
            v = np.flatnonzero((dist[i] != hc.INF_DIST) & (np.arange(n) != s))
            assert (parent[i][v] >= 0).all() and (parent[i][dist[i] == hc.INF_DIST] == -1).all()
            assert (dist[i][parent[i][v]] <= dist[i][v]).all()
    g.close()


@pytest.mark.parametrize("scale,count", [(6, 1), (6, 300), (10, 7), (13, 65), (16, 18)])
@pytest.mark.parametrize("out", ["host", "device", "parents"])
def test_sssp_sources_at_a_time(scale, count, out):
    import torch

    import hc
    h = hc.gen_kronecker(scale, 16, 3, wtype=hc.W_I32)
    n = h.num_nodes
    g = hc.Graph.from_host(h)
    picks = np.random.default_rng(scale).integers(0, n, count).astype(np.int32)  # isolated and repeated ones too
    if out == "host":
        dist = g.sssp(picks)[0]
    else:
        dist = torch.full((count, n), 7, dtype=torch.int32, device="cuda")
        parent = torch.full((count, n), 7, dtype=torch.int32, device="cuda") if out == "parents" else None
        g.sssp(picks, dist, parent)
        dist = dist.cpu().numpy()
    for i in sorted({0, count // 2, count - 1, *range(0, count, 17)}):
        assert np.array_equal(dist[i], oracle.sssp_dijkstra(h.index, h.neighbors, h.weights, picks[i]))
        if out == "parents":
            p = parent[i].cpu().numpy()
            v = np.flatnonzero((dist[i] != hc.INF_DIST) & (np.arange(n) != picks[i]))
            assert p[picks[i]] == picks[i] and (p[v] >= 0).all() and (dist[i][p[v]] < dist[i][v]).all()
    g.close()


@pytest.mark.parametrize("bits", [0, 32])
@pytest.mark.parametrize("top", [1, 255, 3000])
@pytest.mark.parametrize("name", ["path_3000", "fan_600", "star_129", "star_300", "mixed"])
def test_sssp_batched_gaps(name, top, bits):
    """Batched pulls pass over edges heavier than a row's widest gap: zero weights, heavy ones, unreached rows."""
    import hc
    if name == "mixed":
        k = hc.gen_kronecker(11, 16, 5)
        index, nbr = shuffled(k.index, k.neighbors, 1)
    else:
        index, nbr = GRAPHS[name]()
    w = weights(index, nbr, top)
    n = len(index) - 1
    g = hc.Graph(index, nbr, w)
    sources = np.random.default_rng(top).integers(0, n, 70).astype(np.int32)
    for alpha in (0, -1, 1 << 20):  # default switch, pushes only, pulls wherever edges are queued
        for use_graph in (hc.GRAPH_AUTO, hc.GRAPH_ON, hc.GRAPH_OFF):
            dist, _ = g.sssp_batched(sources, switch_alpha=alpha, dist_bits=bits, use_graph=use_graph)
            for i in (0, 33, 69):
                assert np.array_equal(dist[i], oracle.sssp_dijkstra(index, nbr, w, sources[i])), (alpha, use_graph)
    for use_graph in (hc.GRAPH_AUTO, hc.GRAPH_ON, hc.GRAPH_OFF):
        depth, _ = g.bfs_batched(sources, use_graph=use_graph)
        for i in (0, 33, 69):
            assert np.array_equal(depth[i], oracle.bfs_depth(index, nbr, sources[i])), use_graph
    g.close()


@pytest.mark.parametrize("name,delta", [("kron16", 1), ("kron16", 3), ("kron18", 2), ("grid", 1), ("grid", 40)])
def test_sssp_pile_handover(name, delta):
    """Teams of many blocks and small buckets: whole-team epochs end again and again with an empty near queue and
    a short pile, which one block takes over and hands back.  Every source, run several times."""
    import hc
    if name == "grid":
        h = hc.gen_grid(211, 190, 3, wtype=hc.W_I32)
    else:
        h = hc.gen_kronecker(int(name[4:]), 16, 3, wtype=hc.W_I32)
    g = hc.Graph.from_host(h)
    sources = hc.pick_sources(h, 6)
    want = np.stack([oracle.sssp_dijkstra(h.index, h.neighbors, h.weights, s) for s in sources])
    for alpha in (-1, 0):  # pushes only (phases to the end), and with pulls
        for count in (1, 2, 6):  # one team of every block, several teams
            for _ in range(4):
                dist, _, _ = g.sssp(sources[:count], delta=delta, pull_alpha=alpha)
                assert np.array_equal(dist, want[:count]), (alpha, count)
    g.close()


def scanned(index, nbr, n_active, src, alpha=15, beta=18):
    """(vertices, edges) that a run of the direction rule scans: every frontier edge in top-down levels, and in
    bottom-up ones each unvisited row up to its first neighbour in the frontier."""
    n = len(index) - 1
    deg = np.diff(index)
    depth = oracle.bfs_depth(index, nbr, src)
    push, to_check, edges = True, int(index[-1]), int(deg[src])
    vertices = probes = 0
    for level in range(depth.max() + 1):
        front = np.flatnonzero(depth == level)
        if push and edges > to_check // alpha:
            push = False
        if push:
            to_check -= edges
            vertices += len(front)
            probes += int(deg[front].sum())
            edges = int(deg[depth == level + 1].sum())
        else:
            open_ = np.flatnonzero((depth[:n_active] > level) | (depth[:n_active] < 0))
            vertices += len(open_)
            for v in open_:
                hit = np.flatnonzero(depth[nbr[index[v]:index[v + 1]]] == level)
                probes += int(hit[0]) + 1 if len(hit) else int(deg[v])
            grown = int((depth == level + 1).sum())
            if not (grown > len(front) or grown > n // beta):
                push, edges = True, 1
    return vertices, probes


@pytest.mark.parametrize("tail", [0, 1, 3, 40])
@pytest.mark.parametrize("width", [1, 20, 700])
def test_bfs_scanned_edges(width, tail):
    """Statistics of runs whose bottom-up levels are followed by thin top-down ones: a Kronecker core with a strip
    of `tail` levels, `width` vertices each, hanging on its vertices of highest degree."""
    import hc
    k = hc.gen_kronecker(11, 16, 3)
    core = k.num_nodes
    row = np.repeat(np.arange(core), k.degrees())
    u, v = [row[row < k.neighbors]], [k.neighbors[row < k.neighbors]]
    for t in range(tail):
        lane = np.arange(width)
        u.append(lane if t == 0 else core + (t - 1) * width + lane)
        v.append(core + t * width + lane)
    index, nbr = csr(core + tail * width, np.concatenate(u), np.concatenate(v))
    g = hc.Graph(index, nbr)
    for src in (1, int(hc.pick_sources(k, 3)[2]), len(index) - 2):
        _, _, st = g.bfs([src], stats=True)
        assert (st.vertices_scanned, st.edges_scanned) == scanned(index, nbr, g.info().num_active, src), src
    g.close()


@pytest.mark.parametrize("kind,scale,counts", [("kronecker", 17, (17, 18, 19, 70)), ("uniform", 17, (15, 17, 33)),
                                               ("kronecker", 19, (12, 13, 14, 33))])
def test_many_sources_on_a_large_graph(kind, scale, counts):
    """On both sides of the work from which three blocks an SM run: every source's rows equal those of its own call."""
    import torch

    import hc
    g = hc.Graph.generate(hc.GEN_KRONECKER if kind == "kronecker" else hc.GEN_UNIFORM, scale, 16, 5, hc.W_I32)
    n, m = g.num_nodes, g.num_edges
    line = 1 << 26 if scale == 17 else 3 << 26
    assert any(k * m < line for k in counts) and any(k * m >= line for k in counts)
    src = g.pick_sources(max(counts))

    def rows(k):
        return [torch.full((k, n), 7, dtype=torch.int32, device="cuda") for _ in range(3)]

    one = rows(len(src))
    for i, s in enumerate(src):
        g.bfs([s], one[0][i:i + 1], one[1][i:i + 1])
        g.sssp([s], one[2][i:i + 1])
    index, nbr, w = g.csr()
    assert np.array_equal(one[0][0].cpu().numpy(), oracle.bfs_depth(index, nbr, src[0]))
    assert np.array_equal(one[2][0].cpu().numpy(), oracle.sssp_dijkstra(index, nbr, w, src[0]))
    for k in counts:
        depth, parent, dist = rows(k)
        g.bfs(src[:k], depth, parent)
        g.sssp(src[:k], dist)
        assert torch.equal(depth, one[0][:k]) and torch.equal(dist, one[2][:k])
        for i in (0, k - 1):
            assert oracle.verify_bfs_parents(index, nbr, depth[i].cpu().numpy(), parent[i].cpu().numpy(), src[i])[0] == 0
    g.close()


@pytest.mark.parametrize("rows,cols", [(3, 5), (40, 41)])
@pytest.mark.parametrize("alpha", [0, -1, 3, 1 << 20])
def test_batched_loops_on_short_rows(rows, cols, alpha):
    """Road-like graphs: the batched loops are a graph from the start, most pushes note no minima, and a pull may
    follow one that did not."""
    import hc
    h = hc.gen_grid(rows, cols, 3, wtype=hc.W_I32)
    g = hc.Graph.from_host(h)
    sources = np.random.default_rng(rows).integers(0, h.num_nodes, 70).astype(np.int32)
    for bits in (0, 32):
        for use_graph in (hc.GRAPH_AUTO, hc.GRAPH_OFF):
            dist, _ = g.sssp_batched(sources, switch_alpha=alpha, dist_bits=bits, use_graph=use_graph)
            for i in (0, 33, 69):
                assert np.array_equal(dist[i], oracle.sssp_dijkstra(h.index, h.neighbors, h.weights, sources[i]))
    depth, _ = g.bfs_batched(sources)
    for i in (0, 33, 69):
        assert np.array_equal(depth[i], oracle.bfs_depth(h.index, h.neighbors, sources[i]))
    g.close()
