"""Single-source shortest paths at the edges of what a pass stages and cuts:
rows of 4 to 5, 32, 64 and 65, 128 and 129 entries, rows of many chunks (and
those that the relabelling gives a block each, from 2,048 entries on), and
queues that overflow a warp's buffer of 128 vertices within one pass.
Distances are compared exactly with the oracle."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [3, 4, 5, 31, 32, 33, 64, 65, 127, 128, 129, 257, 700, 2047, 2048, 2049, 20000])
@pytest.mark.parametrize("directed", [False, True])
def test_rows(rows, directed):
    import graphhet_b200 as G
    rng = np.random.default_rng(rows)
    n = 30000
    hubs = 40 if rows < 3000 else 3
    # A chain through the hubs, their rows, and a sparse rest.
    src = [np.arange(hubs), rng.integers(0, n, n)] + [np.full(rows, h) for h in range(hubs)]
    dst = [np.arange(1, hubs + 1), rng.integers(0, n, n)] + [rng.choice(n, rows, replace=False) for h in range(hubs)]
    og = O.make_graph(n, np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32), directed,
                      weight_mode=1, weight_seed=rows)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    kw = dict(n=og.n, rowptr=t(og.rowptr), col=t(og.col), w=t(og.w), directed=directed)
    if directed:
        kw.update(in_rowptr=t(og.in_rowptr), in_col=t(og.in_col), in_w=t(og.in_w))
    g = G.CSRGraph(**kw)
    rg = G.ResidentGraph(g)
    for s in (0, 1, n - 1):
        want = O.sssp(og, s)
        for delta in (0.0, 0.02, 8.0):
            assert np.array_equal(rg.sssp(s, delta=delta)[0].cpu().numpy(), want), (s, delta)
            assert np.array_equal(G.sssp(g, s, delta=delta)[0].cpu().numpy(), want), (s, delta)
    rg.close()
