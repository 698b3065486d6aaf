"""Row plans: built when first wanted, in whatever order the calls come; from 2^24 edges on two of them are one."""
import itertools

import numpy as np
import pytest

import hc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [11, 20])
def test_row_plans_in_any_order(scale):
    import torch
    first = hc.Graph.generate(hc.GEN_KRONECKER, scale, 16, 3, hc.W_I32)
    n = first.num_nodes
    assert (first.num_edges >= 1 << 24) == (scale == 20)
    csr = [torch.from_numpy(a).cuda() for a in first.csr()]
    src = first.pick_sources(2)
    first.close()
    f32 = dict(dtype=torch.float32, device="cuda")
    c = torch.from_numpy(np.random.default_rng(1).standard_normal(n).astype(np.float32)).cuda()
    x = torch.full((n,), 1.0 / n, **f32)
    opts = dict(tol_l1=1e-6, max_iters=100)

    def forward(g):
        return g.pagerank(None, torch.empty(n, **f32), **opts)[0]

    def adjoint(g):
        return g.pagerank_backward(x, c, dteleport=torch.empty(n, **f32), want_dw=False, **opts)[0]

    def columns(g):
        return g.ppr_batched(np.arange(6), src[[0, 1, 0, 1, 0]], torch.empty((n, 5), **f32), **opts)[0]

    def paths(g):
        return g.sssp(src, torch.empty((2, n), dtype=torch.int32, device="cuda"))[0]

    calls = (forward, adjoint, columns, paths)
    want = {}
    for f in calls:
        g = hc.Graph(*csr)
        want[f] = f(g)
        g.close()
    for order in itertools.permutations(calls) if scale == 11 else itertools.permutations(calls[:2] + calls[3:]):
        g = hc.Graph(*csr)
        for f in order:
            got = f(g)
            if f is paths:
                assert torch.equal(got, want[f])
            else:  # sums of residuals and dot products meet in any order: the last digits
                assert float((got - want[f]).abs().max()) <= 1e-5 * float(want[f].abs().max())
        g.close()
