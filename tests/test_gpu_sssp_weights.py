"""The default bucket width of large resident graphs by their weights: half the
weight rule's where that pays, the whole where no weight is near zero, where a
few make up most of the sum of a graph with hubs, and for even weights on
uniform rows of 9 to 16 entries.  The distances are those of the caller's rows."""
import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

pytestmark = pytest.mark.gpu


def uniform(n, degree):
    import graphhet_b200 as G
    gen = torch.Generator(device="cuda").manual_seed(n + degree)
    a, b = (torch.randint(0, n, (n * degree,), generator=gen, device="cuda", dtype=torch.int32) for _ in range(2))
    return G.make_graph(n, a, b, False, weight_mode=G.WEIGHT_UNIFORM01, weight_seed=5)


def rmat(*a):
    import graphhet_b200 as G
    return G.rmat_graph(*a)


def exponential(u):
    return -torch.log(1 - u * 0.999999)


@pytest.mark.parametrize("make,cases", [
    (lambda: uniform(1 << 22, 9), [("u", lambda u: u, True), ("1 + u", lambda u: u + 1, False),
                                   ("0.05 + u", lambda u: u + 0.05, True), ("exp^5", lambda u: exponential(u) ** 5, True),
                                   ("equal", torch.ones_like, False)]),
    (lambda: uniform(1 << 23, 5), [("u", lambda u: u, False), ("exp", exponential, True)]),
    (lambda: rmat(22, 16, 9), [("u", lambda u: u, True), ("exp", exponential, True),
                               ("heavy tail", lambda u: exponential(u) ** 4 + 1e-3, False),
                               ("Pareto from 1 on", lambda u: (1 - u * 0.999999) ** -0.4, False)]),
])
def test_default_width(make, cases):
    import graphhet_b200 as G
    g = make()
    u = g.w
    for name, weights, half in cases:
        g.w = weights(u).contiguous()
        assert g.w.dtype == torch.float64 and g.w.numel() == g.m
        rg = G.ResidentGraph(g)
        dist, st, row = rg.sssp(1, trace=True)
        assert row[12] == row[14] * (0.5 if half else 1.0), name
        assert torch.equal(dist, G.sssp(g, 1)[0]), name
        rg.close()
