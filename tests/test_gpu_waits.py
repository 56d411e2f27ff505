"""Host waits of a handle's calls: the source is mapped to the graph's ids on
the device, so a tree costs no wait beyond those of the traversal on the
caller's rows (the levels are the same), and SSSP's none beyond its distances'."""
import numpy as np
import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


def waits(call):
    call()
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU, torch.profiler.ProfilerActivity.CUDA],
                                acc_events=True) as prof:
        call()
    n = sum(e.count for e in prof.key_averages() if e.key == "cudaStreamSynchronize")
    assert n > 0, sorted(e.key for e in prof.key_averages())
    return n


@pytest.mark.parametrize("directed", [False, True])
def test_trees(directed):
    import graphhet_b200 as G
    og = O.rmat_graph(11, 8, 3, directed=directed)
    g = G.rmat_graph(11, 8, 3, directed=directed)
    rg = G.ResidentGraph(g)
    src = int(np.argmax(np.diff(og.rowptr)))
    assert waits(lambda: rg.bfs_pred(src)) == waits(lambda: G.bfs_pred(g, src))
    assert waits(lambda: rg.sssp_pred(src)) == waits(lambda: rg.sssp(src))
    timed = lambda h: (lambda: h(src, oracle_timing=True, trace_cap=64))  # levels driven by the host
    assert waits(timed(rg.bfs)) == waits(timed(lambda s, **k: G.bfs(g, s, **k)))
    depth, pred = (x.cpu().numpy() for x in rg.bfs_pred(src))
    want = O.bfs(og, src)
    assert np.array_equal(depth, want) and pred[src] == -1
    has = (want > 0) & (want < np.iinfo(np.int32).max)
    assert (pred[has] >= 0).all() and np.array_equal(want[pred[has]] + 1, want[has]) and (pred[~has] == -1).all()
    dist, pred = (x.cpu().numpy() for x in rg.sssp_pred(src))
    assert np.array_equal(dist, O.sssp(og, src)) and pred[src] == -1 and (pred[has] >= 0).all()
    rg.close()
