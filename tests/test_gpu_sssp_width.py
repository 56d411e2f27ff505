"""The bucket width of a resident single-source call: half the weight rule's
from 2^26 entries on unless the rows are sparse, and the distances that any
width gives."""
import numpy as np
import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

pytestmark = pytest.mark.gpu


def build(kind, n, degree):
    import graphhet_b200 as G
    if kind == "grid":
        return G.grid_graph(n, n, weight_seed=3)
    g = torch.Generator(device="cuda").manual_seed(n + degree)
    src = torch.randint(0, n, (n * degree,), generator=g, device="cuda", dtype=torch.int32)
    dst = torch.randint(0, n, (n * degree,), generator=g, device="cuda", dtype=torch.int32)
    return G.make_graph(n, src, dst, False, weight_mode=G.WEIGHT_UNIFORM01, weight_seed=5)


@pytest.mark.parametrize("kind,n,degree,half", [
    ("uniform", 1 << 20, 9, False),
    ("uniform", 1 << 21, 15, False),  # below 2^26 entries
    ("uniform", 1 << 21, 17, True),   # above, 34 a vertex
    ("uniform", 10 << 20, 4, True),   # 8 a vertex
    ("grid", 4200, 0, False),         # above, 4 a vertex
])
def test_default_width(kind, n, degree, half):
    import graphhet_b200 as G
    g = build(kind, n, degree)
    rg = G.ResidentGraph(g)
    dist, st, row = rg.sssp(1, trace=True)
    assert row[15] == 0.0
    # Both are float32 roundings of a width and its exact half.
    assert row[12] == row[14] * (0.5 if half else 1.0)
    plain, _ = rg.sssp(1)
    wide, _ = rg.sssp(1, delta=float(row[14]) * 2)
    raw, _ = G.sssp(g, 1)
    assert torch.equal(dist, plain) and torch.equal(dist, wide) and torch.equal(dist, raw)
    assert st["reached"] > n // 2
    rg.close()
