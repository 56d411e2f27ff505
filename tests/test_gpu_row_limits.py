"""Rows that end at the last entry of a CSR of 2^31 - 1 entries (25 GB of
columns and weights, nearly all in a row that nothing reaches)."""
import numpy as np
import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

pytestmark = pytest.mark.gpu

M = 2**31 - 1
N = 700
ROW = 300  # entries of vertex 1, the last row that has any


@pytest.fixture(scope="module")
def graph():
    import graphhet_b200 as G
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 40 << 30:
        pytest.skip("needs 40 GB of free device memory")
    col = torch.zeros(M, dtype=torch.int32, device="cuda")
    w = torch.ones(M, dtype=torch.float64, device="cuda")
    rp = torch.full((N + 1,), M, dtype=torch.int32, device="cuda")
    rp[0], rp[1] = 0, M - ROW
    targets = np.random.default_rng(1).permutation(np.arange(2, N))[:ROW]
    targets.sort()
    weights = np.random.default_rng(2).uniform(0.1, 3.0, ROW)
    col[M - ROW:] = torch.from_numpy(targets.astype(np.int32)).cuda()
    w[M - ROW:] = torch.from_numpy(weights).cuda()
    want = np.full(N, np.inf)
    want[1] = 0.0
    want[targets] = weights
    yield G.CSRGraph(n=N, rowptr=rp, col=col, w=w, directed=True), want
    G.default_workspace().trim()


@pytest.mark.parametrize("delta", [10.0, 0.5])
def test_sssp(graph, delta):
    import graphhet_b200 as G
    g, want = graph
    dist, st = G.sssp(g, 1, inf=float("inf"), delta=delta)
    assert np.array_equal(dist.cpu().numpy(), want)
    assert st["reached"] == ROW + 1


@pytest.mark.parametrize("persistent", [0, 1])
@pytest.mark.parametrize("k", [1, 40, 70])  # a lane per entry; per source, one group of 32 and two
def test_multi_source(graph, persistent, k):
    import ctypes
    import graphhet_b200 as G
    g, want = graph
    ws = G.Workspace()
    G.tune_set("mssp_persistent", persistent, ws=ws)
    srcs = torch.ones(k, dtype=torch.int32, device="cuda")
    dist = torch.empty(k, N, dtype=torch.float64, device="cuda")
    st = G.TraversalStats()
    rc = G.lib().ghb_mssssp(ws.handle, N, G._ptr(g.rowptr), G._ptr(g.col), G._ptr(g.w), G._ptr(srcs), k,
                            float("inf"), G._ptr(dist), ctypes.byref(st))
    assert rc == 0, G.lib().ghb_last_error()
    assert (dist.cpu().numpy() == want).all()
    ws.close()
