"""Label propagation on rows at the edges of its classes, with and without a
leading label, below and above the size from which unchanged neighbourhoods
are skipped (2^17 vertices).  Labels are whole numbers: exact comparison."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu
EDGES = (1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 255, 256, 257, 1024, 1025, 2048, 2049, 4096, 4097, 6144, 6145, 9000)


@pytest.fixture(scope="module")
def G():
    import graphhet_b200 as G
    G.lib()
    return G


def hub_graph(n, background, directed, seed):
    """Two hubs of every class-edge degree, over a sparse random background."""
    rng = np.random.default_rng(seed)
    src, dst = [], []
    for k, d in enumerate(EDGES * 2):
        src.append(np.full(d, k))
        dst.append(len(EDGES) * 2 + rng.choice(n - len(EDGES) * 2, d, replace=False))
    src.append(rng.integers(0, n, background))
    dst.append(rng.integers(0, n, background))
    s, d = np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32)
    return O.make_graph(n, s, d, directed, weight_mode=0)


@pytest.mark.parametrize("n,background", [(20000, 30000), (20000, 400000), ((1 << 17) - 1, 300000), (1 << 17, 100000),
                                          (150001, 1200000)])
@pytest.mark.parametrize("directed", [False, True])
def test_class_edges(G, n, background, directed):
    og = hub_graph(n, background, directed, n + background)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    g = G.CSRGraph(n=og.n, rowptr=t(og.rowptr), col=t(og.col), directed=directed)
    if directed:
        g.in_rowptr, g.in_col = t(og.in_rowptr), t(og.in_col)
    rg = G.ResidentGraph(g)
    for it in (1, 2, 3, 4, 9, 14):
        ref = O.cdlp(og, it)
        assert np.array_equal(G.cdlp(g, it).cpu().numpy(), ref), ("raw", it)
        assert np.array_equal(rg.cdlp(it).cpu().numpy(), ref), ("resident", it)
