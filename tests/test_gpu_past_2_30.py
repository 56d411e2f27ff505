"""A CSR of over 2^30 entries, where the sum of two positions passes 2^31: a
circulant graph (vertex v next to v +- each offset), whose triangles have a
closed form.  About 70 GB of device memory at its largest."""
import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

pytestmark = pytest.mark.gpu

N = 32_500_000  # <= 2^25: resident SSSP keeps its light / heavy split
OFFSETS = [1, 2, 3, 5, 17, 40, 41, 333, 1600, 1603, 9001, 64000, 555555, 2560000, 4000000, 9999999, 12345678]


@pytest.fixture(scope="module")
def graph():
    import graphhet_b200 as G
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 110 << 30:
        pytest.skip("needs 110 GB of free device memory")
    deg = 2 * len(OFFSETS)
    m = deg * N
    assert m > 2**30
    around = torch.tensor(OFFSETS + [N - o for o in OFFSETS], device="cuda")
    col = torch.empty(m, dtype=torch.int32, device="cuda")
    for v0 in range(0, N, 1 << 20):
        v = torch.arange(v0, min(N, v0 + (1 << 20)), device="cuda")
        rows = ((v[:, None] + around) % N).to(torch.int32).sort(1).values
        col[v0 * deg:v0 * deg + rows.numel()] = rows.reshape(-1)
    rp = torch.arange(0, m + 1, deg, device="cuda").to(torch.int32)
    gen = torch.Generator(device="cuda").manual_seed(3)
    w = torch.rand(m, dtype=torch.float64, device="cuda", generator=gen)
    yield G.CSRGraph(n=N, rowptr=rp, col=col, w=w, directed=False)
    G.default_workspace().trim()


def test_triangles(graph):
    import graphhet_b200 as G
    near = set(OFFSETS) | {N - o for o in OFFSETS}
    each = sum((x - y) % N in near for x in near for y in near) // 2  # triangles at a vertex
    c64, _, total = G.tc(graph)
    assert total == each * N // 3
    assert int(c64.min()) == int(c64.max()) == 6 * each


def test_light_ends(graph):
    import graphhet_b200 as G
    far, st = G.sssp(graph, 12)
    assert st["reached"] == N
    G.default_workspace().trim()
    rg = G.ResidentGraph(graph)
    try:
        assert torch.equal(rg.sssp(12)[0], far)
        ws = G.Workspace()
        G.tune_set("sssp_persistent", 0, ws=ws)
        assert torch.equal(rg.sssp(12, ws=ws)[0], far)
        ws.close()
    finally:
        rg.close()
