"""Device memory pressure: a call whose allocation fails releases the rebuildable derived arrays it does not
need (the SSSP pull sweeps' pair array here) and tries once more, and a later call builds them again."""
import numpy as np
import pytest

import hc
import oracle

pytestmark = pytest.mark.gpu


def test_weighted_pagerank_reclaims_the_sssp_pair_array():
    torch = pytest.importorskip("torch")
    host = hc.gen_kronecker(20, 16, 7, wtype=hc.W_I32)
    n, m = host.num_nodes, host.num_edges
    src = hc.pick_sources(host, 2)
    ref = hc.Graph.from_host(host)
    x_ref, st_ref = ref.pagerank(weighted=True, tol_l1=1e-6)
    ref.close()

    g = hc.Graph.from_host(host)
    d0, _, _ = g.sssp(src)  # builds the pair array: 8 (M + 64) bytes
    held_adj = g.info().device_bytes
    adj_bytes = 8 * (m + 64)
    weighted_bytes = 8 * (m + 64) + 4 * n  # fp32 weights, normalised weights, 1 / row sums
    free, _ = torch.cuda.mem_get_info()
    # Leave less than the weighted arrays need, and more than they need once the pair array is gone.
    leave = weighted_bytes - adj_bytes // 2
    filler = torch.empty(max(free - leave, 0), dtype=torch.uint8, device="cuda")
    try:
        x, st = g.pagerank(weighted=True, tol_l1=1e-6)
        held_after = g.info().device_bytes
    finally:
        del filler
        torch.cuda.empty_cache()
    assert held_after < held_adj - adj_bytes + weighted_bytes + adj_bytes // 2  # the pair array went
    assert st.iterations == st_ref.iterations
    assert np.allclose(x, x_ref, rtol=0, atol=1e-7)
    # SSSP builds the pair array again and stays exact.
    d1, _, _ = g.sssp(src)
    assert np.array_equal(d1, d0)
    for i, s in enumerate(src):
        assert np.array_equal(d1[i], oracle.sssp_dijkstra(host.index, host.neighbors, host.weights, s))
    g.close()


@pytest.fixture(scope="module")
def weighted20():
    host = hc.gen_kronecker(20, 16, 7, wtype=hc.W_I32)
    src = hc.pick_sources(host, 64)
    ref = hc.Graph.from_host(host)
    depth, dist = ref.bfs(src, want_parent=False)[0], ref.sssp(src)[0]
    ref.close()
    for i in (0, 63):
        assert np.array_equal(depth[i], oracle.bfs_depth(host.index, host.neighbors, src[i]))
        assert np.array_equal(dist[i], oracle.sssp_dijkstra(host.index, host.neighbors, host.weights, src[i]))
    return host, src, depth, dist


def _fill(torch, leave):
    """Takes all but `leave` bytes of the device's free memory."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(max(free - leave, 0), dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("host_out", [False, True])
def test_bfs_beside_the_sssp_workspace(weighted20, host_out):
    """After hc_sssp with many sources, whose workspaces stay, hc_bfs fits where one source of each does."""
    torch = pytest.importorskip("torch")
    host, src, depth, _ = weighted20
    g = hc.Graph.from_host(host)
    out = torch.empty((64, host.num_nodes), dtype=torch.int32, device="cuda")
    g.sssp(src, out)
    got = np.empty((64, host.num_nodes), np.int32) if host_out else out
    filler = _fill(torch, 12 << 20)  # a BFS workspace of one source takes more
    try:
        g.bfs(src, got, want_parent=False)
    finally:
        del filler
        torch.cuda.empty_cache()
    assert np.array_equal(got if host_out else got.cpu().numpy(), depth)
    g.close()


@pytest.mark.parametrize("room", [1.15, 2.0, 3.5])
def test_sssp_pair_array_before_many_workspaces(weighted20, room):
    """The first call with pulls on a nearly full device: the pair array is built, and the workspaces of several
    sources shrink to one where both do not fit."""
    torch = pytest.importorskip("torch")
    host, src, _, dist = weighted20
    g = hc.Graph.from_host(host)
    out = torch.empty((64, host.num_nodes), dtype=torch.int32, device="cuda")
    g.sssp(src[:1], out[:1], pull_alpha=-1)  # weight statistics, row plan, one workspace
    filler = _fill(torch, int(room * 8 * host.num_edges) + (8 << 20))
    try:
        g.sssp(src, out)
    finally:
        del filler
        torch.cuda.empty_cache()
    assert np.array_equal(out.cpu().numpy(), dist)
    g.close()


@pytest.mark.parametrize("room_mb", [60, 150, 400, 700])
@pytest.mark.parametrize("op", ["bfs", "sssp"])
def test_host_outputs_when_staging_does_not_fit(weighted20, op, room_mb):
    """Workspaces and staging of several sources are given back when only a part of them can be had."""
    torch = pytest.importorskip("torch")
    host, src, depth, dist = weighted20
    g = hc.Graph.from_host(host)
    g.sssp(src[:1])
    g.bfs(src[:1])
    filler = _fill(torch, room_mb << 20)
    try:
        got = g.bfs(src, want_parent=False)[0] if op == "bfs" else g.sssp(src)[0]
    finally:
        del filler
        torch.cuda.empty_cache()
    assert np.array_equal(got, depth if op == "bfs" else dist)
    g.close()


@pytest.mark.parametrize("form,k", [("dense", 33), ("dense_host", 33), ("seeds", 33), ("seeds_weighted", 33),
                                    ("seeds", 1)])
def test_columns_when_the_workspace_does_not_fit(weighted20, form, k):
    """Columns are padded to a multiple of four: a call whose padded matrices do not fit runs its columns in parts."""
    torch = pytest.importorskip("torch")
    host = weighted20[0]
    n = host.num_nodes
    g = hc.Graph.from_host(host)
    opts = dict(tol_l1=1e-6, max_iters=100)
    gen = torch.Generator("cuda").manual_seed(1)
    if form.startswith("dense"):
        t = torch.rand((n, k), generator=gen, device="cuda")
        t /= t.sum(0)
        out = torch.empty((n, k), device="cuda")
        if form == "dense_host":
            t, out = t.cpu().numpy(), np.empty((n, k), np.float32)

        def call():
            return g.pagerank(t, out, **opts)
    else:
        out = torch.empty((n, k), device="cuda")
        seeds = weighted20[1][np.arange(3 * k) % 64].astype(np.int32)

        def call():
            return g.ppr_batched(np.arange(k + 1) * 3, seeds, out, weighted=form == "seeds_weighted", **opts)

    want, st = call()
    want = torch.as_tensor(want).clone().cpu()
    assert st.converged
    g.close()
    g = hc.Graph.from_host(host)
    g.pagerank(weighted=form == "seeds_weighted", max_iters=2)  # derived arrays
    # All matrices of k columns but one (of half the columns they fit), or what one column's solve takes.
    filler = _fill(torch, 4 * 4 * n * k if k > 1 else 4 * 13 * n)
    try:
        got, st = call()
    finally:
        del filler
        torch.cuda.empty_cache()
    assert st.converged
    # Each run stops within tol d / (1 - d) of the fixed point in L1, per column.
    assert float((torch.as_tensor(got).cpu() - want).abs().double().sum(0).max()) <= 2 * 1e-6 * 0.85 / 0.15 + 1e-5
    g.close()
