"""The shipped network's SSSP bucket width against the widths it can choose, by
the times of the present kernels, on graphs it was not trained on."""
import numpy as np
import pytest

pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale,edge_factor,seed", [(18, 16, 1234567), (20, 8, 77)])
def test_width_is_near_the_best(scale, edge_factor, seed):
    import graphhet_b200 as G
    from graphhet_b200 import policy as P
    g = G.rmat_graph(scale, edge_factor, seed)
    rg = G.ResidentGraph(g)
    P.install()
    try:
        net, best = 0.0, 0.0
        for s in P.pick_sources(g, 3, 99):
            rule = float(rg.sssp(s, trace=True)[2][14])

            def ms(**kw):
                rg.sssp(s, **kw)
                return np.median([rg.sssp(s, **kw)[1]["device_ms"] for _ in range(7)])
            times = [ms(delta=rule * 2.0 ** b) for b in range(-5, 2)]
            best += min(times)
            net += ms(policy=G.POLICY_LEARNED)
        # Neighbouring widths are within a tenth of each other around the best.
        assert net <= 1.15 * best
    finally:
        G.policy_load(None, None)
        rg.close()
