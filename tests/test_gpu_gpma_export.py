"""What an export and a look at the snapshot launch after a change of the
dynamic graph: a program that does both, or exports a version again and again,
pays for the rows' compaction once a version; one that exports each version
once never fills the snapshot."""
import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

pytestmark = pytest.mark.gpu


def test_launches_by_use():
    import graphhet_b200 as G
    g = G.rmat_graph(12, 8, 5)
    ws = G.Workspace()
    dyn = G.DynamicGraph.from_graph(g, ws=ws)
    gen = torch.Generator(device="cuda").manual_seed(1)

    def launches(f):
        before = ws.counters()[0]
        out = f()
        return ws.counters()[0] - before, out

    def change(k):
        s, t = (torch.randint(0, g.n, (50,), generator=gen, device="cuda", dtype=torch.int32) for _ in range(2))
        dyn.insert_edges(s, t)
        dyn.delete_edges(s[:20], t[:20])

    def check(ex):
        want = dyn.find(G.edge_keys(torch.repeat_interleave(torch.arange(g.n, device="cuda", dtype=torch.int32),
                                                            (ex.rowptr[1:] - ex.rowptr[:-1]).long()), ex.col))
        assert ex.col.numel() == dyn.m and torch.equal(ex.w, want)

    export = lambda: launches(lambda: dyn.csr_graph())
    look = lambda w=True: launches(lambda: dyn.csr_view(weights=w))[0]
    change(0)
    straight, ex = export()
    check(ex)
    for k in range(3):  # only exports
        change(k)
        assert export()[0] == straight > 0
    assert look() == straight  # the first look makes the snapshot
    for k in range(3):  # exports and looks
        change(k)
        made, ex = export()
        check(ex)
        assert made == straight and look() == 0
        assert export()[0] == 0  # a copy
    change(0)
    assert export()[0] == straight and look(False) == 0  # a habit, no look at the weights
    for k in range(3):  # exports again only: the first still by way of the snapshot
        change(k)
        n, ex = export()
        check(ex)
        assert n == straight
    assert look() == straight
    change(0)
    assert export()[0] == straight  # that version was looked at: by way of the snapshot
    for k in range(3):
        change(k)
        assert export()[0] == straight
    assert export()[0] == straight  # a version exported again: the snapshot is made
    for k in range(3):
        n, ex = export()
        assert n == 0
        check(ex)
    for k in range(3):  # and in the versions that follow with the first export
        change(k)
        assert export()[0] == straight and export()[0] == 0
