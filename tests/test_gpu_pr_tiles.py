"""PageRank where its tiles (256 entries) meet rows: lengths around a lane's 32
values, a tile and several tiles, rows that end on a tile's edge, rows without
entries and isolated vertices, no entries at all; fixed iterations, the L1
history and a tolerance.  Against the CPU path; FP64 sums of up to 6,000 terms
differ by rounding alone (6,000 x 1.1e-16, tolerance 1e-12)."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu
LENGTHS = [1, 2, 31, 32, 33, 63, 64, 255, 256, 257, 511, 512, 513, 4096, 4097, 4352, 4609, 6000]


@pytest.fixture(scope="module")
def G():
    import graphhet_b200 as G
    G.lib()
    return G


def rows_graph(lengths, n, seed):
    rng = np.random.default_rng(seed)
    dst = np.concatenate([np.full(d, 3 * k, np.int64) for k, d in enumerate(lengths)])  # two bare ids between rows
    src = np.concatenate([rng.choice(np.arange(n // 4, n - 50), d, replace=False) for d in lengths])
    return O.make_graph(n, src.astype(np.int32), dst.astype(np.int32), True, weight_mode=0)


@pytest.mark.parametrize("case", ["all", "tiles", "reversed", "small", "one"])
def test_tiles(G, case):
    lengths = {"all": LENGTHS, "tiles": [256] * 8 + [512, 256], "reversed": LENGTHS[::-1], "small": [3, 0, 5, 1] * 40,
               "one": [1]}[case]
    og = rows_graph(lengths, 12000, len(lengths))
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    g = G.CSRGraph(n=og.n, rowptr=t(og.rowptr), col=t(og.col), directed=True)
    g.in_rowptr, g.in_col = t(og.in_rowptr), t(og.in_col)
    for h in (g, G.ResidentGraph(g)):
        run = (lambda **k: h.pagerank(**k)) if isinstance(h, G.ResidentGraph) else (lambda **k: G.pagerank(h, **k))
        for it in (0, 1, 2, 7):
            ref = O.pagerank(og, it, 0.85)
            for prec, tol in ((G.PR_FP64, 1e-12), (G.PR_FP32_KAHAN, 1e-6)):
                for kw in ({}, {"l1_history": True}):
                    rank, ran, hist = run(iterations=it, precision=prec, **kw)
                    assert ran == it
                    assert np.abs(rank.cpu().numpy() - ref).sum() <= tol * ref.sum()
                    if kw and it and prec == G.PR_FP64:
                        prev = O.pagerank(og, it - 1, 0.85)
                        assert abs(hist[-1] - np.abs(ref - prev).sum()) <= 1e-12
        rank, ran, _ = run(iterations=60, tolerance=1e-10)
        assert ran < 60
        assert np.abs(rank.cpu().numpy() - O.pagerank(og, ran, 0.85)).sum() <= 1e-12


def test_refuses_capture(G):
    """A call on a capturing stream is refused, and the workspace stays usable."""
    og = rows_graph([5, 300, 40], 2000, 4)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    rg = G.ResidentGraph(G.CSRGraph(n=og.n, rowptr=t(og.rowptr), col=t(og.col), w=None, directed=True,
                                    in_rowptr=t(og.in_rowptr), in_col=t(og.in_col), in_w=None))
    ws = G.Workspace()
    first = G_rank(rg.pagerank(iterations=3, ws=ws))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    out = torch.empty(og.n, dtype=torch.float64, device="cuda")
    with torch.cuda.stream(side), torch.cuda.graph(graph, stream=side):
        with pytest.raises(Exception, match="captur"):
            rg.pagerank(iterations=3, out=out, ws=ws)
        out.zero_()
    torch.cuda.synchronize()
    assert np.array_equal(G_rank(rg.pagerank(iterations=3, ws=ws)), first)
    rg.close()


def G_rank(result):
    r = result[0] if isinstance(result, tuple) else result
    return r.cpu().numpy()
