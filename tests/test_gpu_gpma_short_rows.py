"""Dynamic-graph batches on short rows: a lane an entry up to 32 entries, steps of
64 above, at their edges, with updates before, inside, at the ends of and behind
a row, on every second row, and rows that empty.  Compared exactly with the oracle."""
import numpy as np
import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu
LENGTHS = (1, 2, 3, 15, 16, 30, 31, 32, 33, 34, 62, 63, 64, 65, 95, 96, 97, 127, 128, 129, 191, 192, 193, 250)


@pytest.mark.parametrize("kind", ["mixed", "insert", "delete", "empty"])
@pytest.mark.parametrize("size", ["small", "large"])  # up to 32,768 updates, and above
def test_short_rows(kind, size):
    import graphhet_b200 as G
    rng = np.random.default_rng(len(kind) + len(size))
    n = 30000
    rows = np.concatenate([np.full(d, 2 * k) for k, d in enumerate(LENGTHS)])
    cols = np.concatenate([50 + 3 * np.arange(d) for d in LENGTHS])
    keys = O.gpma_keys(rows, cols)
    vals = rng.uniform(0.1, 1.0, len(keys))
    rp, col, w = O.gpma_to_csr(n, keys, vals)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    dg = G.DynamicGraph.from_csr(t(rp), t(col), t(w))
    bk, bv = [], []
    for k, d in enumerate(LENGTHS):
        at = sorted({j for j in (0, 1, 30, 31, 32, 33, 63, 64, 65, d // 2, d - 2, d - 1) if 0 <= j < d})
        if kind in ("mixed", "insert"):
            new = [7] + [50 + 3 * j + o for j in at for o in (-1, 1)] + [50 + 3 * d, n - 1]
            bk += [(2 * k, c) for c in new]
            bv += list(rng.uniform(0.1, 1.0, len(new)))
        if kind in ("mixed", "delete") and k % 2:
            bk += [(2 * k, 50 + 3 * j) for j in at]
            bv += [0.0] * len(at)
        if kind == "empty":
            bk += [(2 * k, 50 + 3 * j) for j in range(d)]
            bv += [0.0] * d
    if size == "large":
        extra = rng.integers(0, n, (40000, 2))
        bk += [tuple(x) for x in extra.tolist()]
        bv += list(np.where(rng.random(40000) < 0.3, 0.0, 0.5))
    bk, bv = O.gpma_keys(*np.array(bk).T), np.array(bv)
    for _ in range(2):
        got = dg.update(t(bk), t(bv))
        keys, vals, counts = O.gpma_update(keys, vals, bk, bv)
        assert (got["inserted"], got["deleted"], got["modified"], got["ignored"]) == counts
        cg = dg.csr_graph()
        for a, b in zip((cg.rowptr, cg.col, cg.w), O.gpma_to_csr(n, keys, vals)):
            assert np.array_equal(a.cpu().numpy(), b)
