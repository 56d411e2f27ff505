"""Multi-source SSSP at the edges of its source groups (32 lanes, 64 sources a
walk, fewer than four active sources) and of its row chunks (32 entries).
Distances are compared exactly with one-source runs of the oracle."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import graphhet_b200 as G
    G.lib()
    return G


@pytest.mark.parametrize("k", [1, 3, 4, 31, 32, 33, 64, 65, 96, 97, 130])
@pytest.mark.parametrize("persistent", [0, 1])
def test_groups(G, k, persistent):
    rng = np.random.default_rng(k)
    n = 3000
    src, dst = [rng.integers(0, n, 4000)], [rng.integers(0, n, 4000)]
    for hub, d in enumerate((31, 32, 33, 64, 65, 127, 1500)):
        src.append(np.full(d, hub))
        dst.append(rng.choice(n, d, replace=False))
    og = O.make_graph(n, np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32), False,
                      weight_mode=1, weight_seed=k)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    rg = G.ResidentGraph(G.CSRGraph(n=og.n, rowptr=t(og.rowptr), col=t(og.col), w=t(og.w), directed=False))
    ws = G.Workspace()
    G.tune_set("mssp_persistent", persistent, ws=ws)
    sources = rng.integers(0, n, k)
    for log2 in (2, -6):
        G.tune_set("mssp_width_log2", log2, ws=ws)
        dist = rg.mssssp(sources, ws=ws)[0].cpu().numpy()
        for i in sorted({0, k // 3, k // 2, k - 1}):
            assert np.array_equal(dist[i], O.sssp(og, int(sources[i]))), (log2, i)


@pytest.mark.parametrize("leaves", [63, 64, 65, 1000, 20000])
@pytest.mark.parametrize("persistent", [0, 1])
def test_queue(G, leaves, persistent):
    """Rounds that queue around and well past a warp's buffer of 64 vertices:
    stars whose leaves lead on to a second star."""
    n = 2 * leaves + 10
    hub = np.arange(3)
    leaf = np.arange(10, 10 + leaves)
    src = np.concatenate([np.repeat(hub, leaves), leaf, leaf])
    dst = np.concatenate([np.tile(leaf, 3), leaf + leaves, np.full(leaves, 5)])
    og = O.make_graph(n, src.astype(np.int32), dst.astype(np.int32), False, weight_mode=1, weight_seed=leaves)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    rg = G.ResidentGraph(G.CSRGraph(n=og.n, rowptr=t(og.rowptr), col=t(og.col), w=t(og.w), directed=False))
    ws = G.Workspace()
    G.tune_set("mssp_persistent", persistent, ws=ws)
    sources = np.array([0, 1, 2, 5, 12, n - 1] * 6)[:33]
    for log2 in (2, -4):
        G.tune_set("mssp_width_log2", log2, ws=ws)
        dist, st = rg.mssssp(sources, ws=ws)
        assert st["edges_examined"] > 0
        dist = dist.cpu().numpy()
        for i in (0, 3, 4, 5, 32):
            assert np.array_equal(dist[i], O.sssp(og, int(sources[i]))), (log2, i)
