"""The sample behind the bucket width, where it takes every weight (below 2^20)
and at the edges of a step of all its threads: the rule's width is 32 mean
weights over the mean degree, of which a float32 is kept."""
import numpy as np
import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

pytestmark = pytest.mark.gpu
STEP = 128 * 512


@pytest.mark.parametrize("m", [1, 31, 32, 511, 513, STEP - 1, STEP, STEP + 1, 8 * STEP - 1, 8 * STEP, 8 * STEP + 1,
                               2**20 - 1, 2**20, 2**20 + 1, 2**21 + 7])
def test_rule_width(m):
    import graphhet_b200 as G
    n = 9
    w = np.random.default_rng(m).uniform(0.1, 2.0, m)
    rp = np.full(n + 1, m, np.int32)
    rp[:3] = 0, 0, m // 3
    t = lambda a: torch.from_numpy(a).cuda()
    g = G.CSRGraph(n=n, rowptr=t(rp), col=t(np.arange(m, dtype=np.int32) % n), w=t(w), directed=True)
    g.in_rowptr, g.in_col, g.in_w = G.transpose_csr(n, g.rowptr, g.col, g.w)
    rg = G.ResidentGraph(g)
    row = rg.sssp(2, trace=True)[2]
    want = w.mean() * 32.0 / max(1.0, m / n)
    # All of the weights below 2^21 entries (summed in another order); from there on every second.
    assert row[14] == pytest.approx(want, rel=3e-7 if m < 2**21 else 5e-3)
    rg.close()
