"""Output rows longer than the pitch limit of a 2-D copy (2^31 - 1 bytes)."""
import numpy as np
import pytest

import hc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph():
    import torch
    n = (1 << 29) + 9
    # A path of three vertices at the start, an edge at the end, nothing between (so not sorted by degree).
    deg = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    deg[torch.tensor([1, 3, n - 1, n])] = 1
    deg[2] = 2
    index = torch.cumsum(deg, 0)
    del deg
    nbr = torch.tensor([1, 0, 2, 1, n - 1, n - 2], dtype=torch.int32, device="cuda")
    w = torch.tensor([5, 5, 7, 7, 3, 3], dtype=torch.int32, device="cuda")
    g = hc.Graph(index, nbr, w)
    del index
    torch.cuda.empty_cache()
    yield g
    g.close()


@pytest.mark.parametrize("op", ["bfs", "sssp"])
def test_host_rows_above_the_pitch_limit(graph, op):
    n = graph.num_nodes
    sources = [1, n - 1]
    far = -1 if op == "bfs" else hc.INF_DIST
    out = np.full((len(sources), n), 9, np.int32)
    if op == "bfs":
        graph.bfs(sources, out, want_parent=False)
    else:
        graph.sssp(sources, out)
    heads = {"bfs": {1: [1, 0, 1]}, "sssp": {1: [5, 0, 7]}}[op]
    for row, s in zip(out, sources):
        head = heads.get(s, [far] * 3)
        tail = [far, far] if s == 1 else [1 if op == "bfs" else 3, 0]
        assert row[:3].tolist() == head and row[-2:].tolist() == tail
        assert (row[3:-2] == far).all()
