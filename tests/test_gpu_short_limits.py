"""The shortest barrier limit (100 us) with passes that some blocks run alone
while the others wait: a mesh's traversals still end, with the results that
the default limit gives.  A call may meet a delay of the box's own, so one of
three has to succeed."""
import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(300, 300), (1501, 1999), (2999, 2001)])
def test_mesh(rows, cols):
    import graphhet_b200 as G
    g = G.grid_graph(rows, cols, weight_seed=3)
    rg = G.ResidentGraph(g)
    ws = G.Workspace()
    G.tune_set("barrier_limit_us", 100, ws=ws)
    calls = {"bfs": lambda **k: rg.bfs(5, **k), "raw bfs": lambda **k: G.bfs(g, 5, **k),
             "sssp": lambda **k: rg.sssp(5, **k), "raw sssp": lambda **k: G.sssp(g, 5, **k)}
    for name, call in calls.items():
        want = call()[0]
        got = []
        for _ in range(3):
            try:
                got.append(call(ws=ws)[0])
            except G.GhbError as e:
                assert "timed out" in str(e)
        assert got, name
        assert all(torch.equal(x, want) for x in got)
    rg.close()
