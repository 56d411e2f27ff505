"""Traversals whose frontiers stay small, outgrow one block's queue and shrink
again: long paths, thin grids, fans wider than the queue in shared memory, hubs
whose rows are cut into more chunks than one block takes, and a barrier limit
that makes the one-block runs hand back to the grid again and again.  Depths and
distances are compared exactly."""
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


def path(n):
    return n, np.arange(n - 1), np.arange(1, n)


def broom(stem, fan):
    """A path into a hub with `fan` leaves, each of which starts a short path."""
    hub = stem
    leaves = np.arange(hub + 1, hub + 1 + fan)
    tails = leaves + fan
    src = np.concatenate([np.arange(stem), np.full(fan, hub), leaves])
    dst = np.concatenate([np.arange(1, stem + 1), leaves, tails])
    return int(tails[-1]) + 1, src, dst


def lattice(rows, cols):
    v = np.arange(rows * cols).reshape(rows, cols)
    return (rows * cols, np.concatenate([v[:, :-1].ravel(), v[:-1].ravel()]),
            np.concatenate([v[:, 1:].ravel(), v[1:].ravel()]))


SHAPES = {"path": path(3000), "two": path(2), "thin": lattice(5, 900), "wide": lattice(700, 800),
          "fan_2047": broom(40, 2047), "fan_2049": broom(40, 2049), "fan_9000": broom(3, 9000), "fan_200": broom(1, 200)}


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("mode", [1, 2])  # weights in (0, 1], whole numbers to 100
@pytest.mark.parametrize("directed", [False, True])
def test_narrow_frontiers(G, shape, mode, directed):
    n, src, dst = SHAPES[shape]
    og = O.make_graph(n, src.astype(np.int32), dst.astype(np.int32), directed, weight_mode=mode, weight_seed=3)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    g = G.CSRGraph(n=og.n, rowptr=t(og.rowptr), col=t(og.col), w=t(og.w), directed=directed)
    if directed:
        g.in_rowptr, g.in_col, g.in_w = t(og.in_rowptr), t(og.in_col), t(og.in_w)
    rg = G.ResidentGraph(g)
    ws = G.Workspace()
    for limit_us in (2000000, 4000):
        G.tune_set("barrier_limit_us", limit_us, ws=ws)
        for s in (0, n // 2):
            dist, depth = O.sssp(og, s), O.bfs(og, s)
            for delta in (0.0, 1e-3, 1e6):
                assert np.array_equal(G.sssp(g, s, delta=delta, ws=ws)[0].cpu().numpy(), dist), ("raw", s, delta)
                assert np.array_equal(rg.sssp(s, delta=delta, ws=ws)[0].cpu().numpy(), dist), ("resident", s, delta)
            for kw in ({}, {"max_depth": 7}, {"policy": G.POLICY_PUSH}):
                ref = O.bfs(og, s, kw.get("max_depth", 2**31 - 1))
                assert np.array_equal(G.bfs(g, s, ws=ws, **kw)[0].cpu().numpy(), ref), ("raw", s, kw)
                d, st = rg.bfs(s, ws=ws, **kw)
                assert np.array_equal(d.cpu().numpy(), ref), ("resident", s, kw)
                assert st["reached"] == int((ref != 2**31 - 1).sum())
            assert st["levels"] >= int(depth[depth != 2**31 - 1].max())
