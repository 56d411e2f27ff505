"""Triangle counting on both sides of the probes per entry from which the hub
bitmaps (16, in a resident graph) and a copy relabelled by degree (24, on the
caller's ids) are used.  In disjoint cliques of c vertices the hash kernels make
(c - 2) / 6 probes per entry.  Counts are whole numbers: every comparison is exact."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu


def cliques(sizes, seed):
    """Disjoint cliques on shuffled ids: n, src, dst."""
    src, dst, n = [], [], 0
    for c in sizes:
        i, j = np.triu_indices(c, 1)
        src.append(i + n)
        dst.append(j + n)
        n += c
    ids = np.random.default_rng(seed).permutation(n)
    return n, ids[np.concatenate(src)], ids[np.concatenate(dst)]


def count(f):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        out = f()
        torch.cuda.synchronize()
    return out, " ".join(e.key for e in prof.key_averages())


def check(n, src, dst, hubs, copies):
    import graphhet_b200 as G
    og = O.make_graph(n, src.astype(np.int32), dst.astype(np.int32), False, weight_mode=0)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    g = G.CSRGraph(n=og.n, rowptr=t(og.rowptr), col=t(og.col), directed=False)
    rg = G.ResidentGraph(g)
    ref, ref_total = O.tc_oriented(og)
    for f, kernel, used in ((lambda: rg.tc(), "tc_hub_items_kernel", hubs), (lambda: G.tc(g), "tc_unrank_kernel", copies)):
        for _ in range(2):
            (c64, c32, total), names = count(f)
            assert (kernel in names) == used, names
            assert np.array_equal(c64.cpu().numpy(), ref) and total == ref_total
            assert np.array_equal(c32.cpu().numpy(), ref.astype(np.int32))
    rg.close()


@pytest.mark.parametrize("c", [3, 60, 90, 110, 130, 160])
def test_cliques(c):
    check(*cliques([c] * 100, c), hubs=c >= 110, copies=c >= 160)


def test_short_rows_beside_a_clique():
    """Rows at the edges of a bitmap (32 hub neighbours) and of a listed row (8)."""
    check(*cliques([400, 2, 3, 8, 9, 10, 31, 32, 33, 34, 35, 64, 65, 129, 130], 1), hubs=True, copies=False)


def test_past_the_bitmap_table_beside_a_clique():
    """More than 2^18 vertices of 33 hub neighbours or more, and a clique that
    brings the mean over the lines."""
    rng = np.random.default_rng(7)
    n, hubs, per = (1 << 18) + 6000, 512, 40
    low = np.repeat(np.arange(hubs, n), per)
    k, a, b = cliques([3000], 3)
    src = np.concatenate([low, np.arange(hubs, n - 1), a + n])
    dst = np.concatenate([rng.integers(0, hubs, low.size), np.arange(hubs + 1, n), b + n])
    check(n + k, src, dst, hubs=True, copies=True)


def test_no_entries():
    import graphhet_b200 as G
    g = G.CSRGraph(n=5, rowptr=torch.zeros(6, dtype=torch.int32, device="cuda"),
                   col=torch.zeros(0, dtype=torch.int32, device="cuda"), directed=False)
    assert G.ResidentGraph(g).tc()[2] == 0 and G.tc(g)[2] == 0
