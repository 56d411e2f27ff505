"""Triangle counting through the hub bitmaps of a resident graph: sizes at the
edges of the hub range (4,096 ids), of a bitmap (32 hub neighbours), of a
slice (128 entries) and of the bitmap table (2^18 ids).  Counts are whole
numbers: every comparison is exact."""
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


def check(G, og):
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    g = G.CSRGraph(n=og.n, rowptr=t(og.rowptr), col=t(og.col), directed=False)
    c64, c32, total = G.ResidentGraph(g).tc()
    ref, ref_total = O.tc_oriented(og)
    assert np.array_equal(c64.cpu().numpy(), ref)
    assert np.array_equal(c32.cpu().numpy(), ref.astype(np.int32))
    assert total == ref_total


@pytest.mark.parametrize("n", [2, 3, 32, 33, 34, 128, 129, 130, 257, 258, 385])
def test_complete_graphs(G, n):
    iu = np.triu_indices(n, 1)
    check(G, O.make_graph(n, iu[0].astype(np.int32), iu[1].astype(np.int32), False, weight_mode=0))


@pytest.mark.parametrize("n", [4095, 4096, 4097, 4130, 9000])
def test_hub_range_edges(G, n):
    """Degrees fall with the id, so the low ids are hubs of every density and
    triangles lie inside the hub range, across its end and beyond it."""
    rng = np.random.default_rng(n)
    e = 40 * n
    src = (n * rng.random(e) ** 3).astype(np.int32)
    dst = (n * rng.random(e)).astype(np.int32)
    check(G, O.make_graph(n, src, dst, False, weight_mode=0))


def test_past_the_bitmap_table(G):
    """More than 2^18 vertices of 33 hub neighbours or more: those past the
    table are probed one by one."""
    rng = np.random.default_rng(7)
    n, hubs, per = (1 << 18) + 6000, 512, 40
    low = np.repeat(np.arange(hubs, n), per)
    src = np.concatenate([low, np.arange(hubs, n - 1)]).astype(np.int32)
    dst = np.concatenate([rng.integers(0, hubs, low.size), np.arange(hubs + 1, n)]).astype(np.int32)
    check(G, O.make_graph(n, src, dst, False, weight_mode=0))


@pytest.mark.parametrize("longest", [20, 32, 33, 128, 129, 1024, 1025, 4097])
@pytest.mark.parametrize("loops", [False, True])
def test_directed_rows(G, longest, loops):
    """Directed rows of every length class of the hash kernels, with and
    without self-loops, against the reference's merge over every entry."""
    rng = np.random.default_rng(longest)
    n = 6000
    hub = np.arange(40)
    src = np.concatenate([np.repeat(hub, longest), rng.integers(0, n, 3 * n), np.arange(0, n, 7) if loops else hub[:0]])
    dst = np.concatenate([np.concatenate([rng.choice(n, longest, replace=False) for _ in hub]),
                          np.concatenate([rng.integers(0, 200, n), rng.integers(0, n, 2 * n)]),
                          np.arange(0, n, 7) if loops else hub[:0]])
    rp, col, _ = O.build_csr(n, src.astype(np.int32), dst.astype(np.int32), drop_self_loops=not loops, weight_mode=0)
    irp, icol, _ = O.build_csr(n, dst.astype(np.int32), src.astype(np.int32), drop_self_loops=not loops, weight_mode=0)
    og = O.Graph(n=n, rowptr=rp, col=col, w=None, directed=True, in_rowptr=irp, in_col=icol, in_w=None)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    g = G.CSRGraph(n=n, rowptr=t(rp), col=t(col), directed=True)
    g.in_rowptr, g.in_col = t(irp), t(icol)
    ref = O.tc(og)
    for c64, c32, _ in (G.tc(g), G.ResidentGraph(g).tc()):
        assert np.array_equal(c32.cpu().numpy(), ref)
        assert np.array_equal(c64.cpu().numpy().astype(np.int32), ref)


@pytest.mark.parametrize("scale", [15, 16])  # below and above the entries from which raw rows are relabelled
def test_raw_rows_of_a_skewed_graph(G, scale):
    og = O.rmat_graph(scale, 16, 5, directed=False, weight_mode=0)
    assert (og.m >= 1 << 20) == (scale == 16)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    c64, c32, total = G.tc(G.CSRGraph(n=og.n, rowptr=t(og.rowptr), col=t(og.col), directed=False))
    ref, ref_total = O.tc_oriented(og)
    assert np.array_equal(c64.cpu().numpy(), ref) and total == ref_total
    assert np.array_equal(c32.cpu().numpy(), ref.astype(np.int32))
