"""Row classes of label propagation at the edges of the blocks that count and
fill them (256 and 1,024 rows) and of every class's length, against the
oracle."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [255, 256, 257, 1023, 1024, 1025, 3071, 140000])
def test_classes(n):
    import graphhet_b200 as G
    rng = np.random.default_rng(n)
    src, dst = [rng.integers(0, n, n)], [rng.integers(0, n, n)]
    for k, d in enumerate((1, 2, 3, 4, 5, 8, 9, 16, 17, 32, 33, 128, 129, 256, 1000, 3000, 5000)):
        d = min(d, n - 1)
        v = (k * 61) % n
        src.append(np.full(d, v))
        dst.append(rng.choice(n, d, replace=False))
    og = O.make_graph(n, np.concatenate(src).astype(np.int32), np.concatenate(dst).astype(np.int32), False,
                      weight_mode=0)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    g = G.CSRGraph(n=og.n, rowptr=t(og.rowptr), col=t(og.col), w=None, directed=False)
    rg = G.ResidentGraph(g)
    for it in (1, 2, 5):
        want = O.cdlp(og, it)
        assert np.array_equal(G.cdlp(g, it).cpu().numpy(), want)
        assert np.array_equal(rg.cdlp(it).cpu().numpy(), want)
    rg.close()
