"""The default bucket width of a resident graph with hubs: half the weight
rule's from 6 M entries on where the highest-ranked row is 32 times the mean,
the whole elsewhere; the distances do not depend on it."""
import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

pytestmark = pytest.mark.gpu


def star_and_uniform(n, degree, hub):
    """A uniform graph whose vertex 3 also meets `hub` others."""
    import graphhet_b200 as G
    gen = torch.Generator(device="cuda").manual_seed(n + degree)
    a, b = (torch.randint(0, n, (n * degree,), generator=gen, device="cuda", dtype=torch.int32) for _ in range(2))
    a = torch.cat([a, torch.full((hub,), 3, dtype=torch.int32, device="cuda")])
    b = torch.cat([b, torch.arange(10, 10 + hub, dtype=torch.int32, device="cuda")])
    return G.make_graph(n, a, b, False, weight_mode=G.WEIGHT_UNIFORM01, weight_seed=5)


def heavy_tail(g):
    g.w = torch.log(1 - g.w * 0.999999) ** 4
    return g


@pytest.mark.parametrize("make,half", [
    (lambda G: G.rmat_graph(18, 16, 1234567), False),                # 7.6 M entries
    (lambda G: G.rmat_graph(19, 16, 1234567), True),                 # 15 M
    (lambda G: G.rmat_graph(20, 8, 77, a=0.35, b=0.3, c=0.3), True),
    (lambda G: heavy_tail(G.rmat_graph(19, 16, 1234567)), False),
    (lambda G: G.rmat_graph(20, 16, 77, directed=True), True),
    (lambda G: star_and_uniform(1 << 19, 8, 500 * 16), True),        # 16 M, one hub of 500 times the mean
    (lambda G: star_and_uniform(1 << 19, 8, 16 * 16), False),        # of 17
    (lambda G: star_and_uniform(1 << 22, 2, 4000), False),           # sparse
])
def test_default_width(make, half):
    import graphhet_b200 as G
    g = make(G)
    rg = G.ResidentGraph(g)
    dist, st, row = rg.sssp(3, trace=True)
    assert row[12] == row[14] * (0.5 if half else 1.0) and row[15] == 0.0
    plain, _ = rg.sssp(3)
    raw, _ = G.sssp(g, 3)
    assert torch.equal(dist, plain) and torch.equal(dist, raw)
    rg.close()
