"""Outputs on memory that the legacy default stream still uses: a call's writes come after what was queued there."""
import numpy as np
import pytest

import hc
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graphs():
    h = hc.gen_kronecker(10, 16, 3, wtype=hc.W_I32)
    f = hc.gen_kronecker(10, 16, 3, wtype=hc.W_F32)
    return h, hc.Graph.from_host(h), f, hc.Graph.from_host(f)


def _calls(h, g, gf, out, aux):
    src = [int(hc.pick_sources(h, 1)[0])]
    return {
        "bfs": lambda: g.bfs(src, out["i"], aux["i"]),
        "bfs_parents": lambda: g.bfs(src, None, out["i"], want_depth=False),
        "sssp": lambda: g.sssp(src, out["i"]),
        "pagerank": lambda: g.pagerank(None, out["f"]),
        "pagerank_teleport": lambda: g.pagerank(aux["t"], out["f"]),
        "pagerank_columns": lambda: g.pagerank(aux["t2"], out["f2"]),
        "backward": lambda: gf.pagerank_backward(aux["t"], aux["t"], dteleport=out["f"], want_dw=False, weighted=True),
        "ppr": lambda: g.ppr_batched([0, 1, 2], src * 2, out["f2"]),
        "bfs_batched": lambda: g.bfs_batched(src, out["i"]),
        "sssp_batched": lambda: g.sssp_batched(src, out["i"]),
    }


@pytest.mark.parametrize("name", ["bfs", "bfs_parents", "sssp", "pagerank", "pagerank_teleport", "pagerank_columns",
                                  "backward", "ppr", "bfs_batched", "sssp_batched"])
def test_outputs_after_the_default_stream(graphs, name):
    import torch
    h, g, _, gf = graphs
    n = h.num_nodes
    i32 = dict(dtype=torch.int32, device="cuda")
    f32 = dict(dtype=torch.float32, device="cuda")
    out = {"i": torch.empty((1, n), **i32), "f": torch.empty(n, **f32), "f2": torch.empty((n, 2), **f32)}
    t = torch.rand(n, generator=torch.Generator("cpu").manual_seed(1)).cuda()
    aux = {"i": torch.empty((1, n), **i32), "t": t / t.sum(), "t2": torch.stack([t, t.flip(0)], 1) / t.sum()}
    call = _calls(h, g, gf, out, aux)[name]
    call()  # plans and workspaces
    torch.cuda.synchronize()
    want = {k: v.clone() for k, v in out.items()}
    torch.cuda.synchronize()
    # The previous user of the outputs, still running on the default stream when the call is made.
    torch.cuda._sleep(40_000_000)
    for v in out.values():
        v.fill_(7)
    call()
    torch.cuda.synchronize()
    key = {"bfs": "i", "bfs_parents": "i", "sssp": "i", "bfs_batched": "i", "sssp_batched": "i",
           "pagerank_columns": "f2", "ppr": "f2"}.get(name, "f")
    got = out[key]
    if name == "bfs_parents":  # any valid tree
        src = int(hc.pick_sources(h, 1)[0])
        depth = oracle.bfs_depth(h.index, h.neighbors, src)
        assert oracle.verify_bfs_parents(h.index, h.neighbors, depth, got[0].cpu().numpy(), src)[0] == 0
    elif key == "i":
        assert np.array_equal(got.cpu().numpy(), want[key].cpu().numpy())
    else:
        assert torch.allclose(got, want[key], rtol=1e-5, atol=1e-9)
