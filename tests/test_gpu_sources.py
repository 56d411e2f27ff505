"""A resident call maps its sources to the graph's ids on the device, in the
one-launch kernels and in the host-driven loops: depths, distances and trees
from vertices at both ends of the degree ranking, isolated ones included, and
batches past one pass of 256 sources."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("persistent", [0, 1])
def test_sources(directed, persistent):
    import graphhet_b200 as G
    rng = np.random.default_rng(5)
    n = 1500
    src, dst = rng.integers(0, n - 20, 4000), rng.integers(0, n - 20, 4000)
    src[:300] = 7
    og = O.make_graph(n, src.astype(np.int32), dst.astype(np.int32), directed, weight_mode=1, weight_seed=3)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    kw = dict(n=og.n, rowptr=t(og.rowptr), col=t(og.col), w=t(og.w), directed=directed)
    if directed:
        kw.update(in_rowptr=t(og.in_rowptr), in_col=t(og.in_col), in_w=t(og.in_w))
    rg = G.ResidentGraph(G.CSRGraph(**kw))
    ws = G.Workspace()
    for name in ("sssp_persistent", "ms_persistent", "mssp_persistent"):
        G.tune_set(name, persistent, ws=ws)
    for s in (0, 7, 700, n - 1):
        want, far = O.bfs(og, s), O.sssp(og, s)
        d, st = rg.bfs(s, ws=ws, oracle_timing=not persistent)[:2]
        assert np.array_equal(d.cpu().numpy(), want)
        assert st["reached"] == int((want < np.iinfo(np.int32).max).sum())
        d, p = rg.bfs_pred(s, ws=ws)[:2]
        assert np.array_equal(d.cpu().numpy(), want)
        x, st = rg.sssp(s, ws=ws)
        assert np.array_equal(x.cpu().numpy(), far)
        assert st["reached"] == int((far < 1e300).sum())
        assert np.array_equal(rg.sssp(s, delta=0.25, ws=ws)[0].cpu().numpy(), far)
        x, p = rg.sssp_pred(s, ws=ws)
        assert np.array_equal(x.cpu().numpy(), far)
        p = p.cpu().numpy()
        assert p[s] < 0 and (p[(far < 1e300) & (np.arange(n) != s)] >= 0).all()
    many = rng.integers(0, n, 260)
    md, mx = rg.msbfs(many, ws=ws)[0].cpu().numpy(), rg.mssssp(many, ws=ws)[0].cpu().numpy()
    for i in (0, 255, 256, 259):
        assert np.array_equal(md[i], O.bfs(og, int(many[i])))
        assert np.array_equal(mx[i], O.sssp(og, int(many[i])))
    rg.close()
