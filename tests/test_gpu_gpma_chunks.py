"""Dynamic-graph batches on rows at the edges of a chunk (256 entries) and of
the rows that one warp rebuilds (256 for small batches, 512 for large ones):
updates before a row's first entry, at a chunk's first and last columns, between
chunks, past the end, and none at all in some chunks; and exports with and
without a cached snapshot.  Compared exactly with the oracle."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu
LENGTHS = (1, 2, 255, 256, 257, 300, 511, 512, 513, 767, 768, 769, 2000, 4100)


@pytest.fixture(scope="module")
def G():
    import graphhet_b200 as G
    G.lib()
    return G


@pytest.mark.parametrize("batch", ["edges", "sparse", "large", "insert_only", "delete_only"])
@pytest.mark.parametrize("snapshot", [False, True])
def test_chunk_edges(G, batch, snapshot):
    rng = np.random.default_rng(len(batch))
    n = 20000
    rows = np.concatenate([np.full(d, 3 * k) for k, d in enumerate(LENGTHS)])
    cols = np.concatenate([100 + 4 * np.arange(d) for d in LENGTHS])  # gaps of 4: room between entries
    keys = O.gpma_keys(rows, cols)
    vals = rng.uniform(0.1, 1.0, len(keys))
    rp, col, w = O.gpma_to_csr(n, keys, vals)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    dg = G.DynamicGraph.from_csr(t(rp), t(col), t(w))
    bk, bv = [], []
    for k, d in enumerate(LENGTHS):
        r = 3 * k
        at = sorted({0, 1, 254, 255, 256, 257, 510, 511, 512, 513, d // 2, d - 1})
        at = [j for j in at if j < d]
        ins = [5, 99] + [100 + 4 * j + o for j in at for o in (-1, 1)] + [100 + 4 * d, n - 1]
        dele = [100 + 4 * j for j in at]
        if batch == "sparse":
            ins, dele = ins[-1:], dele[:1] if k % 2 else []
        if batch in ("edges", "large", "sparse", "insert_only"):
            bk += [(r, c) for c in ins]
            bv += list(rng.uniform(0.1, 1.0, len(ins)))
        if batch in ("edges", "large", "sparse", "delete_only"):
            bk += [(r, c) for c in dele]
            bv += [0.0] * len(dele)
    if batch == "large":  # over the 32,768 updates of a small batch
        extra = rng.integers(0, n, (40000, 2))
        bk += [tuple(x) for x in extra.tolist()]
        bv += list(np.where(rng.random(40000) < 0.2, 0.0, 0.5))
    bk, bv = O.gpma_keys(*np.array(bk).T), np.array(bv)
    for _ in range(2):  # the second time most of the batch changes weights or nothing
        if snapshot:
            dg.csr_view(weights=True)
        got = dg.update(t(bk), t(bv))
        keys, vals, counts = O.gpma_update(keys, vals, bk, bv)
        assert (got["inserted"], got["deleted"], got["modified"], got["ignored"]) == counts
        if snapshot:
            dg.csr_view(weights=True)
        for weights in (True, False):
            cg = dg.csr_graph(weights=weights)
            rp, col, w = O.gpma_to_csr(n, keys, vals)
            assert np.array_equal(cg.rowptr.cpu().numpy(), rp)
            assert np.array_equal(cg.col.cpu().numpy(), col)
            if weights:
                assert np.array_equal(cg.w.cpu().numpy(), w)
