"""CDLP on 2^17 vertices and more at the mean degree (6) from which changed labels
are kept as bits: meshes, trees, uniform and community graphs on both sides of
it, through iterations in which most, some and no labels move.  Against the CPU
path."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


def edges(kind):
    rng = np.random.default_rng(len(kind))
    if kind == "grid":
        return O.grid_edges(400, 500)
    if kind == "tree":
        a = np.arange(1, 150000)
        return (a - 1) // 3, a
    if kind == "star":
        a = np.arange(1, 140000)
        return np.zeros_like(a), a
    n, k = 150000, {"uniform 5": 5, "uniform 7": 7, "communities 5": 5, "communities 7": 7}[kind] * 75000
    if kind.startswith("u"):
        return rng.integers(0, n, k), rng.integers(0, n, k)
    base = rng.integers(0, n // 50, k) * 50
    return base + rng.integers(0, 50, k), base + rng.integers(0, 50, k)


@pytest.mark.parametrize("kind", ["grid", "tree", "star", "uniform 5", "uniform 7", "communities 5", "communities 7"])
def test_sparse(kind):
    import graphhet_b200 as G
    src, dst = (np.asarray(x).astype(np.int32) for x in edges(kind))
    n = int(max(src.max(), dst.max())) + 1
    og = O.make_graph(n, src, dst, False, weight_mode=0)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    g = G.CSRGraph(n=og.n, rowptr=t(og.rowptr), col=t(og.col), w=None, directed=False)
    rg = G.ResidentGraph(g)
    for it in (3, 4, 10, 25):
        want = O.cdlp(og, it)
        assert np.array_equal(G.cdlp(g, it).cpu().numpy(), want)
        assert np.array_equal(rg.cdlp(it).cpu().numpy(), want)
    rg.close()
