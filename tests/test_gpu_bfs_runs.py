"""Host-driven BFS, whose runs of small levels share one launch: the level at
which the direction rule ends a run is one that every block agrees on (the
rule's side changes from one level to the next on each of these graphs, so a
block that decided from another block's unsettled sum would leave the others
waiting until their barrier gives up)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(97, 131), (64, 1000), (211, 190)])
def test_runs_end_on_one_level(rows, cols):
    import graphhet_b200 as G
    g = G.grid_graph(rows, cols, weight_seed=3)
    n = rows * cols
    rg = G.ResidentGraph(g)
    for src in (0, 5, n // 2 + cols // 2):
        r, c = np.divmod(np.arange(n), cols)
        want = np.abs(r - src // cols) + np.abs(c - src % cols)
        for call in (lambda: G.bfs_pred(g, src), lambda: rg.bfs_pred(src)):
            for _ in range(8):
                depth, pred = call()
                assert np.array_equal(depth.cpu().numpy(), want)
        p = pred.cpu().numpy()
        assert p[src] == -1 and np.array_equal(want[p[want > 0]] + 1, want[want > 0])
    rg.close()
