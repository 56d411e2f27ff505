"""Multi-source SSSP on a graph of 2.2M entries, where rows are cut at 64 entries
for up to eight sources and at 32 for more: rows at the edges of both.
Distances are compared exactly with one-source runs of the oracle."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def graph():
    rng = np.random.default_rng(5)
    n, first = 60000, 20000
    src, dst = [rng.integers(first, n, 1100000)], [rng.integers(first, n, 1100000)]
    # Rows of known length: hubs of their own leaves, the leaves on into the rest.
    leaf = 200
    for hub, d in enumerate((31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 191, 192, 193, 4096, 4097, 9000)):
        leaves = np.arange(leaf, leaf + d) if leaf + d < first else rng.choice(np.arange(leaf, first), d, replace=False)
        leaf = min(leaf + d, first - 9001)
        src += [np.full(d, hub), leaves]
        dst += [leaves, rng.integers(first, n, d)]
    og = O.make_graph(n, np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32), False,
                      weight_mode=1, weight_seed=2)
    assert 8 << 18 <= og.m < 9 << 18
    return og


@pytest.mark.parametrize("k", [1, 2, 3, 4, 8, 9, 33])
def test_cut(graph, k):
    import graphhet_b200 as G
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    g = G.CSRGraph(n=graph.n, rowptr=t(graph.rowptr), col=t(graph.col), w=t(graph.w), directed=False)
    rg = G.ResidentGraph(g)
    ws = G.Workspace()
    sources = (np.arange(k) * 7) % 18
    for log2 in (2, -4):
        G.tune_set("mssp_width_log2", log2, ws=ws)
        dist = rg.mssssp(sources, ws=ws)[0].cpu().numpy()
        for i in sorted({0, k // 2, k - 1}):
            assert np.array_equal(dist[i], O.sssp(graph, int(sources[i]))), (log2, i)
    rg.close()
    ws.close()


@pytest.mark.parametrize("k", [1, 2, 3, 4])
def test_wide_rounds_of_short_rows(k):
    """Rounds of many vertices a warp (the bounds of 32 loaded together): stars
    whose leaves, 200,000 of them or some tens of thousands, have one entry or two."""
    import graphhet_b200 as G
    rng = np.random.default_rng(k)
    leaves, n = 200000, 200000 + 40
    leaf = np.arange(40, n)
    src = np.concatenate([rng.integers(0, 3, leaves), rng.integers(3, 40, leaves // 5)])
    dst = np.concatenate([leaf, leaf[rng.permutation(leaves)[:leaves // 5]]])
    og = O.make_graph(n, src.astype(np.int32), dst.astype(np.int32), False, weight_mode=1, weight_seed=k)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    rg = G.ResidentGraph(G.CSRGraph(n=og.n, rowptr=t(og.rowptr), col=t(og.col), w=t(og.w), directed=False))
    sources = [0, 50000, 7, 1][:k]
    dist = rg.mssssp(sources)[0].cpu().numpy()
    for i in range(k):
        assert np.array_equal(dist[i], O.sssp(og, sources[i])), i
    rg.close()
