"""CSR builder and relabelling at the edges of their tiles (2,048 entries):
entry counts around a tile, runs of equal pairs across a tile's end, lists
without a usable entry, and stretches of isolated vertices before, between and
after the rows, short and longer than a thread fills alone.  Compared exactly
with the CPU builder; the weight of a repeated pair is its last one's."""
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


def check(G, n, src, dst, symmetrize, drop):
    src, dst = np.asarray(src, np.int32), np.asarray(dst, np.int32)
    w = np.arange(1, len(src) + 1, dtype=np.float64)
    t = lambda a: torch.from_numpy(a).cuda()
    rp, col, wt = G.build_csr(n, t(src), t(dst), w=t(w), symmetrize=symmetrize, drop_self_loops=drop)
    orp, ocol, ow = O.build_csr(n, src, dst, w=w, symmetrize=symmetrize, drop_self_loops=drop)
    assert np.array_equal(rp.cpu().numpy(), orp)
    assert np.array_equal(col.cpu().numpy(), ocol)
    assert np.array_equal(wt.cpu().numpy(), ow)
    if not symmetrize or len(ocol) == 0:
        return
    g = G.CSRGraph(n=n, rowptr=rp, col=col, w=wt, directed=False)
    rg = G.ResidentGraph(g)
    assert rg.n_active == int((np.diff(orp) > 0).sum())
    og = O.Graph(n=n, rowptr=orp, col=ocol, w=ow, directed=False, in_rowptr=orp, in_col=ocol, in_w=ow)
    s = int(np.argmax(np.diff(orp)))
    assert np.array_equal(rg.sssp(s)[0].cpu().numpy(), O.sssp(og, s))
    assert np.array_equal(rg.cdlp(3).cpu().numpy(), O.cdlp(og, 3))


@pytest.mark.parametrize("count", [1, 2, 1023, 1024, 1025, 2047, 2048, 2049, 4096, 5000])
@pytest.mark.parametrize("symmetrize", [False, True])
def test_tile_edges(G, count, symmetrize):
    rng = np.random.default_rng(count)
    check(G, 40, rng.integers(0, 40, count), rng.integers(0, 40, count), symmetrize, True)   # long runs
    check(G, 900, rng.integers(0, 900, count), rng.integers(0, 900, count), symmetrize, False)


@pytest.mark.parametrize("n,ids", [(70, [0, 69]), (200000, [0, 1]), (200000, [199998, 199999]), (200000, [100, 100000, 100063, 100128]),
                                   (5, [4, 2]), (4096, [0, 63, 64, 65, 128, 4095])])
def test_isolated_stretches(G, n, ids):
    src = np.repeat(ids, len(ids))
    dst = np.tile(ids, len(ids))
    for symmetrize in (False, True):
        for drop in (False, True):
            check(G, n, src, dst, symmetrize, drop)


def test_nothing_usable(G):
    for sym in (False, True):
        check(G, 3000, np.arange(3000), np.arange(3000), sym, True)
