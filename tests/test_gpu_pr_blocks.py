"""PageRank at the entry counts where its blocks change shape (2^18 and 2^20) and
its hub cache sets in (2^20): ranks, the L1 history and a tolerance against the
CPU path.  Sums of a few thousand FP64 terms differ by rounding alone (1e-12); FP32
rows are Kahan sums (1e-6 relative L1)."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("entries", [2**18, 2**20])
@pytest.mark.parametrize("more", [-1, 0, 1])
def test_block_shapes(entries, more):
    import graphhet_b200 as G
    rng = np.random.default_rng(entries + more)
    n, m = 30011, entries + more
    # Distinct edges without loops: strides of a permuted id space, and a hub.
    flat = rng.choice((n - 3000) * n, m + 1000, replace=False)
    src, dst = flat // n, flat % n
    keep = src != dst
    src, dst = src[keep][:m].astype(np.int32), dst[keep][:m].astype(np.int32)
    og = O.make_graph(n, src, dst, True, weight_mode=0)
    assert og.col.size == m
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    g = G.CSRGraph(n=n, rowptr=t(og.rowptr), col=t(og.col), directed=True)
    g.in_rowptr, g.in_col = t(og.in_rowptr), t(og.in_col)
    rg = G.ResidentGraph(g)
    for call in (lambda *a, **k: G.pagerank(g, *a, **k), rg.pagerank):
        for it in (1, 7):
            want = O.pagerank(og, it, 0.85)
            got, ran, hist = call(it, 0.85, l1_history=True)
            assert ran == it and np.abs(got.cpu().numpy() - want).sum() <= 1e-12 * np.abs(want).sum()
            assert hist[-1] == pytest.approx(np.abs(want - O.pagerank(og, it - 1, 0.85)).sum(), rel=1e-9)
            got = call(it, 0.85, precision=G.PR_FP32_KAHAN)[0].cpu().numpy()
            assert np.abs(got - want).sum() <= 1e-6 * np.abs(want).sum()
        got, ran, _ = call(40, 0.85, tolerance=1e-7)
        assert 1 < ran < 40
        assert np.abs(got.cpu().numpy() - O.pagerank(og, ran, 0.85)).sum() <= 1e-12
    rg.close()
