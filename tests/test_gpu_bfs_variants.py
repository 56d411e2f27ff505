"""Which variant of the one-launch BFS a call runs: the one with squad runs only
on graphs of low mean degree and only where a squad may run (the rule, forced
top-down), the lighter one for every other call; the depths are the same."""
import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

pytestmark = pytest.mark.gpu


def variant(call):
    """(depths, whether the launch was the variant with squad runs)"""
    call()  # a first launch loads the kernel
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as prof:
        depth = call()[0]
        torch.cuda.synchronize()
    names = {e.key for e in prof.key_averages() if "bfs_persistent_kernel" in e.key}
    assert len(names) == 1, names
    return depth, any(t in min(names) for t in ("<true>", "<1>", "<(bool)1>"))


@pytest.mark.parametrize("kind", ["grid", "rmat"])
def test_variant(kind):
    import graphhet_b200 as G
    from graphhet_b200 import policy as P
    g = G.grid_graph(120, 150, weight_seed=3) if kind == "grid" else G.rmat_graph(12, 8, 5)
    low = kind == "grid"
    rg = G.ResidentGraph(g)
    want, squad = variant(lambda: rg.bfs(7))
    assert squad == low
    levels = rg.bfs(7)[1]["levels"]
    calls = {"push": (lambda: rg.bfs(7, policy=G.POLICY_PUSH), low), "raw": (lambda: G.bfs(g, 7), low),
             "no network": (lambda: rg.bfs(7, policy=G.POLICY_LEARNED), low),
             "pull": (lambda: rg.bfs(7, policy=G.POLICY_PULL), False),
             "traced": (lambda: rg.bfs(7, trace_cap=4096), False),
             "schedule": (lambda: rg.bfs(7, policy=G.POLICY_SCHEDULE, schedule=[2] * levels), False)}
    for name, (call, expected) in calls.items():
        depth, squad = variant(call)
        assert squad == expected, name
        assert torch.equal(depth, want), name
    P.install()
    try:
        depth, squad = variant(lambda: rg.bfs(7, policy=G.POLICY_LEARNED))
        assert not squad and torch.equal(depth, want)
        ws = G.Workspace()  # a network with no level to decide is the rule
        G.tune_set("pol_band", 0, ws=ws)
        depth, squad = variant(lambda: rg.bfs(7, policy=G.POLICY_LEARNED, ws=ws))
        assert squad == low and torch.equal(depth, want)
        ws.close()
    finally:
        G.policy_load(None, None)
    rg.close()
