"""The BFS regret on a mesh, where a call by the rule runs small levels on a few
blocks and schedules and the network's calls do not: the ratios compare
decisions that ran alike, so the oracle is not beaten by another machinery."""
import pytest

pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def test_mesh():
    import graphhet_b200 as G
    from graphhet_b200 import policy as P
    P.install()
    try:
        rg = G.ResidentGraph(G.grid_graph(300, 300, weight_seed=3))
        r = P.regret(rg, [5, 45150], repeats=5)
        # Another order of top-down and bottom-up levels cannot gain a tenth over
        # the schedule that is cheapest by its measured levels.
        assert -0.1 < r["regret_heuristic"] < 0.25 and r["regret_beamer14"] > -0.1 and r["regret_learned"] > -0.1
        assert r["ms"]["rule_call"] < r["ms"]["heuristic"]
        rg.close()
    finally:
        G.policy_load(None, None)
