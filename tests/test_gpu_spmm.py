"""Multi-column PageRank at the widths and row lengths where its sweep changes form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DAMPING, TOL = 0.85, 1e-6
# The stop leaves at most TOL * d / (1 - d) in any entry; fp32 sums of at most 2000 terms of total <= 1 add 2000 * 2^-24.
BOUND = TOL * DAMPING / (1 - DAMPING) + 2000 * 2.0 ** -24


def stars(degrees):
    """Star centres of these degrees on a common ring of leaves, leaves linked in a path: every row length side by side."""
    leaves = max(degrees)
    u, v = [], []
    for i, d in enumerate(degrees):
        u.append(np.full(d, leaves + i))
        v.append((np.arange(d) + 7 * i) % leaves)
    u.append(np.arange(leaves - 1))
    v.append(np.arange(1, leaves))
    u, v = np.concatenate(u), np.concatenate(v)
    n = leaves + len(degrees)
    src, dst = np.concatenate([u, v]), np.concatenate([v, u])
    order = np.lexsort((dst, src))
    index = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(src, minlength=n), out=index[1:])
    return index, dst[order].astype(np.int32)


def fixed_point(index, nbr, w, t):
    """x = (1-d) t + d A x in 64 bits, A[v,u] = w(u->v) / sum of u's weights (symmetric weights)."""
    n = len(index) - 1
    row = np.repeat(np.arange(n), np.diff(index))
    s = np.bincount(row, weights=w, minlength=n)
    vals = (w / s[nbr])[:, None]
    x = t.copy()
    for _ in range(400):
        y = np.zeros_like(x)
        np.add.at(y, row, vals * x[nbr])
        x = (1 - DAMPING) * t + DAMPING * y
    return x


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("k", [2, 4, 5, 8, 9, 16, 17, 31, 33, 64, 65, 129, 256])
def test_columns(k, weighted):
    import hc
    index, nbr = stars([1, 63, 64, 65, 127, 511, 512, 513, 1025, 1537])
    n = len(index) - 1
    row = np.repeat(np.arange(n), np.diff(index))
    w = (1 + (row + nbr) % 7).astype(np.float32) if weighted else None
    g = hc.Graph(index, nbr, w)
    rng = np.random.default_rng(k)
    # Dense teleports of two distinct columns, repeated: a column's place must not matter.
    two = rng.random((n, 2)).astype(np.float32)
    two /= two.sum(0)
    t = np.ascontiguousarray(two[:, np.arange(k) % 2])
    x, st = g.pagerank(t, tol_l1=TOL, max_iters=300, weighted=weighted)
    want = fixed_point(index, nbr, np.ones(len(nbr)) if w is None else w.astype(np.float64), two.astype(np.float64))
    assert st.converged and np.abs(x - want[:, np.arange(k) % 2]).max() <= BOUND
    # Seeds: two per column.
    seeds = np.stack([np.arange(k) % n, (np.arange(k) * 37 + 5) % n], 1).astype(np.int32)
    seeds[seeds[:, 0] == seeds[:, 1], 1] += 1
    x, st = g.ppr_batched(np.arange(k + 1) * 2, seeds.ravel(), tol_l1=TOL, max_iters=300, weighted=weighted)
    cols = sorted({0, 1, k // 2, k - 1})
    t = np.zeros((n, len(cols)))
    for i, c in enumerate(cols):
        t[seeds[c], i] = 0.5
    want = fixed_point(index, nbr, np.ones(len(nbr)) if w is None else w.astype(np.float64), t)
    assert st.converged and np.abs(x[:, cols] - want).max() <= BOUND
    g.close()


@pytest.mark.parametrize("kind,scale", [("uniform", 20), ("kronecker", 18), ("kronecker", 8), ("uniform", 6)])
def test_single_column_against_two(kind, scale):
    """The single-column solve (one launch, or a launch per sweep on a large graph without hubs) against the
    multi-column sweeps: each stops within TOL * d / (1 - d) of the fixed point in L1, and fp32 rounding adds at
    most 100 sweeps of 2^-23 of the total."""
    import torch

    import hc
    g = hc.Graph.generate(hc.GEN_UNIFORM if kind == "uniform" else hc.GEN_KRONECKER, scale, 16, 1)
    n = g.num_nodes
    t = torch.full((n, 2), 1.0 / n, device="cuda")
    two = torch.empty((n, 2), device="cuda")
    g.pagerank(t, two, tol_l1=TOL, max_iters=100)
    for accel in (0, 1):
        one = torch.empty(n, device="cuda")
        _, st = g.pagerank(None, one, tol_l1=TOL, max_iters=100, accel=accel)
        host, _ = g.pagerank(None, tol_l1=TOL, max_iters=100, accel=accel)
        assert st.converged and np.abs(one.cpu().numpy() - host).sum() <= 1e-4 * TOL + 100 * 2.0 ** -23
        assert (one - two[:, 0]).abs().double().sum().item() <= 2 * TOL * DAMPING / (1 - DAMPING) + 100 * 2.0 ** -23
    capped, st = g.pagerank(None, tol_l1=TOL, max_iters=2)
    assert st.iterations == 2 and not st.converged
    g.close()


@pytest.mark.parametrize("k", [2, 3, 4, 7, 33, 130, 255])
def test_host_and_device_matrices(k):
    """Teleport and scores in host or device memory, and one matrix for both: the same scores."""
    import torch

    import hc
    h = hc.gen_kronecker(9, 16, 3)
    g = hc.Graph.from_host(h)
    t = np.random.default_rng(k).random((h.num_nodes, k)).astype(np.float32)
    t /= t.sum(0)
    opts = dict(tol_l1=1e-6, max_iters=100)
    want, st = g.pagerank(t, **opts)
    for tele_dev in (False, True):
        for out_dev in (False, True):
            tele = torch.from_numpy(t).cuda() if tele_dev else t
            out = torch.full((h.num_nodes, k), 7.0, device="cuda") if out_dev else np.full_like(t, 7.0)
            got, st1 = g.pagerank(tele, out, **opts)
            got = got.cpu().numpy() if out_dev else got
            assert st1.iterations == st.iterations and np.array_equal(got, want)
    both = torch.from_numpy(t).cuda()
    g.pagerank(both, both, **opts)
    assert np.array_equal(both.cpu().numpy(), want)
    both = t.copy()
    g.pagerank(both, both, **opts)
    assert np.array_equal(both, want)
    g.close()


@pytest.mark.parametrize("n", [9471, 18943, 18944, 28417, 47363, 66304, 75775, 75776])
def test_rows_per_warp(n):
    """Vertex counts at which a warp takes another number of short rows, against the single-column solve (bounds as
    above)."""
    import hc
    rng = np.random.default_rng(n)
    u, v = rng.integers(0, n, 4 * n), rng.integers(0, n, 4 * n)
    key = np.unique(np.concatenate([u * n + v, v * n + u])[np.concatenate([u != v, u != v])])
    index = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(key // n, minlength=n), out=index[1:])
    g = hc.Graph(index, (key % n).astype(np.int32))
    t = rng.random((n, 2)).astype(np.float32)
    t /= t.sum(0)
    opts = dict(tol_l1=TOL, max_iters=200)
    one = [g.pagerank(np.ascontiguousarray(t[:, i]), **opts)[0] for i in (0, 1)]
    for k in (2, 6, 19, 67, 140):
        x = g.pagerank(np.ascontiguousarray(t[:, np.arange(k) % 2]), **opts)[0]
        for c in {0, 1, k // 2, k - 1}:
            assert np.abs(x[:, c] - one[c % 2]).sum() <= 2 * TOL * DAMPING / (1 - DAMPING) + 100 * 2.0 ** -23
    g.close()
