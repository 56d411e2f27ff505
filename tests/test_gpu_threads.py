"""Two host threads, each with a workspace and a stream of its own, on graphs
whose PageRank blocks take different amounts of shared memory (the hub cache
is smaller below 2^24 entries)."""
import threading

import pytest

pytest.importorskip("torch")
import torch  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_pagerank_on_two_graphs(precision):
    import graphhet_b200 as G
    gen = torch.Generator(device="cuda").manual_seed(7)
    n, edges = 1 << 20, 9 << 20
    ends = [torch.randint(0, n, (edges,), generator=gen, device="cuda", dtype=torch.int32) for _ in range(2)]
    graphs = [G.ResidentGraph(G.make_graph(n, *ends, False, weight_mode=G.WEIGHT_NONE)),
              G.ResidentGraph(G.rmat_graph(12, 8, 3))]
    assert graphs[0].m > 1 << 24 > graphs[1].m
    want = [rg.pagerank(5, precision=precision)[0] for rg in graphs]
    torch.cuda.synchronize()
    failed = []

    def work(k, calls):
        try:
            ws = G.Workspace()
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(calls):
                    got = graphs[k].pagerank(5, precision=precision, ws=ws)[0]
                    if not torch.equal(got, want[k]):
                        failed.append("graph %d: other ranks" % k)
        except G.GhbError as e:
            failed.append("graph %d: %s" % (k, e))

    threads = [threading.Thread(target=work, args=(0, 100)), threading.Thread(target=work, args=(1, 400))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for rg in graphs:
        rg.close()
    assert not failed, failed[0]
