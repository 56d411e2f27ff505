"""Triangle counting on the caller's ids where the copy relabelled by degree
does not fit on the device: the call counts without the copy, as it did before
there was one, keeps no more than that took, and leaves no error behind."""
import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("free_mb", [420, 330])  # room for the copy but not its sort; not for the copy either
def test_counts_without_the_copy(free_mb):
    import graphhet_b200 as G
    g = G.rmat_graph(20, 16, 11, weight_mode=G.WEIGHT_NONE)
    assert g.m > 1 << 24
    ws = G.Workspace()
    want = G.tc(g, ws=ws)
    ws.close()
    G.default_workspace().trim()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    c64, c32 = torch.empty_like(want[0]), torch.empty_like(want[1])  # results: allocated beforehand
    ws = G.Workspace()
    held = []
    try:
        while (left := torch.cuda.mem_get_info()[0] - (free_mb << 20)) > 8 << 20:
            held.append(torch.empty(min(left, 16 << 30) - (4 << 20), dtype=torch.uint8, device="cuda"))
        rc = G.lib().ghb_tc(ws.handle, g.n, G._ptr(g.rowptr), G._ptr(g.col), G._ptr(c64), G._ptr(c32), None)
        assert rc == 0, G.lib().ghb_last_error()
        assert ws.counters()[1] <= 256 << 20
    finally:
        del held
        torch.cuda.empty_cache()
    assert torch.equal(c64, want[0]) and torch.equal(c32, want[1])
    got = G.tc(g, ws=ws)  # with room: the copy again
    assert got[2] == want[2] and torch.equal(got[0], want[0])
    ws.close()
