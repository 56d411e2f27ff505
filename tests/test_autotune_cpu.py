"""Which launch shapes the autotuner times: those whose blocks fit a
multiprocessor with PageRank's tiles beside the hub cache, each launch once."""
import types

import pytest

import graphhet_b200 as G
from graphhet_b200 import autotune as A


@pytest.mark.parametrize("kb,threads,blocks,ok", [
    (80, 1024, 1, True),
    (112, 1024, 2, False),  # 2 x (112 + 32 + 2) KB
    (80, 512, 2, True),     # 2 x (80 + 16 + 2)
    (64, 1024, 4, False),   # 4,096 threads
    (64, 512, 4, False),    # 4 x (64 + 16 + 2)
    (32, 512, 4, True),
])
def test_feasible(kb, threads, blocks, ok):
    assert A.feasible({"pr_cache_kb": kb, "pr_threads": threads, "pr_blocks_per_sm": blocks}) == ok


def test_feasible_defaults():
    assert A.feasible({"pr_threads": 512, "pr_blocks_per_sm": 2})  # with the default cache
    assert A.feasible({"ms_warp_rest": 64, "ms_pull_div": 4})      # other algorithms' values


@pytest.mark.parametrize("algo,entries", [("pagerank", 1 << 20), ("pagerank", 1 << 26), ("msbfs", 1 << 20)])
def test_each_launch_is_timed_once(algo, entries, monkeypatch):
    values = {"pr_cache_kb": 80, "pr_threads": 1024, "pr_blocks_per_sm": 1, "ms_warp_rest": 512, "ms_pull_div": 16}
    monkeypatch.setattr(G, "tune_get", lambda k, ws=None: values[k])
    monkeypatch.setattr(G, "tune_set", lambda k, v, ws=None: values.__setitem__(k, v))
    monkeypatch.setattr(A, "_workload", lambda *a: (lambda: None, lambda: True))

    def cost(run, reps):  # fewer threads and a large cache are better, up to what the call gives
        c = A.launched(values, entries)
        return 1.0 + c["pr_threads"] / 1024 - c["pr_cache_kb"] / 2**20 + values["ms_pull_div"] / 100
    monkeypatch.setattr(A, "_timer", cost)
    best, table = A.tune(types.SimpleNamespace(m=entries), algo, log=None)
    shapes = [tuple(sorted(A.launched({k: t[k] for k in A.SPACES[algo]}, entries).items())) for t in table]
    assert len(shapes) == len(set(shapes)) >= 6
    if algo == "pagerank":
        assert best["pr_threads"] == 256
        assert A.launched(best, entries)["pr_cache_kb"] == (112 if entries >= 1 << 24 else 16) * 1024
    else:
        assert best["ms_pull_div"] == 2
