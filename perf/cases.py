"""The work that programs do with this package, as cases to time: the six
analytics on small graphs (one call after another, where latency counts), each
of them at scale, many-source traversals, loading a graph and updating one.

Graphs are seeded and synthetic: RMAT (a = .57, b = c = .19, permuted ids, the
vertex count not always a power of two), Erdos-Renyi, and 2D grids with integer
weights for long diameters.  Weights are a hash of the unordered pair, so both
directions of an edge, and its duplicates, agree."""
import math

import torch

import graphhet_b200 as G

INF = math.inf
DEV = "cuda"


# ------------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _rmat(n, count, seed):
    """count RMAT edges over n vertices: ids permuted, then folded onto [0, n)."""
    g = _gen(seed)
    scale = max(1, (n - 1).bit_length())
    src = torch.zeros(count, dtype=torch.int32, device=DEV)
    dst = torch.zeros(count, dtype=torch.int32, device=DEV)
    for _ in range(scale):
        u = torch.rand(count, generator=g, device=DEV)
        src.mul_(2).add_(u >= 0.76)
        dst.mul_(2).add_(((u >= 0.57) & (u < 0.76)) | (u >= 0.95))
    perm = (torch.randperm(1 << scale, generator=g, device=DEV) % n).to(torch.int32)
    return perm[src], perm[dst]


def _er(n, count, seed):
    g = _gen(seed)
    return tuple(torch.randint(0, n, (count,), generator=g, device=DEV, dtype=torch.int32) for _ in range(2))


def _grid(rows, cols):
    v = torch.arange(rows * cols, dtype=torch.int32, device=DEV).view(rows, cols)
    src = torch.cat([v[:, :-1].reshape(-1), v[:-1].reshape(-1)])
    dst = torch.cat([v[:, 1:].reshape(-1), v[1:].reshape(-1)])
    return src, dst


def _edges(case, seed):
    """(n, src, dst) as a user has them: unsorted, with repeats and self-loops."""
    if case["family"] == "grid":
        return (case["rows"] * case["cols"],) + _grid(case["rows"], case["cols"])
    n = case["n"]
    make = _rmat if case["family"] == "rmat" else _er
    return (n,) + make(n, n * case["degree"], seed)


def _weights(case, seed, src, dst):
    """One weight per unordered pair: in (0, 1], on grids a whole number in [1, 100]."""
    lo, hi = torch.minimum(src, dst).to(torch.int64), torch.maximum(src, dst).to(torch.int64)
    h = (lo << 31) + hi + 0x1F3D5B79 * (seed + 1)
    del lo, hi
    for mul in (0x2545F4914F6CDD1D, 0x369DEA0F31A53F85):
        h ^= (h >> 29) & ((1 << 35) - 1)
        h *= mul
    h = (h >> 32) & 0x7FFFFFFF
    if case["family"] == "grid":
        return (1 + h % 100).to(torch.float64)
    return (h + 1).to(torch.float64) / float(1 << 31)


def _distinct(n, src, dst, count, seed):
    """count distinct unordered pairs of the edge list, in random order and direction."""
    key = torch.minimum(src, dst).to(torch.int64) * n + torch.maximum(src, dst)
    key = torch.unique(key[src != dst])
    g = _gen(seed + 3)
    key = key[torch.randperm(key.numel(), generator=g, device=DEV)[:count]]
    lo, hi = (key // n).to(torch.int32), (key % n).to(torch.int32)
    flip = torch.rand(lo.numel(), generator=g, device=DEV) < 0.5
    return torch.where(flip, hi, lo), torch.where(flip, lo, hi)


def _arriving(case, seed, n, src, dst):
    """An edge list of a known number of distinct pairs, with a sixteenth of
    them repeated and some self-loops, in random order."""
    if case["family"] != "grid":
        src, dst = _distinct(n, src, dst, n * case["degree"] // 2, seed)
    g = _gen(seed + 4)
    more = src.numel() // 16
    loops = torch.arange(0, n, 64, dtype=torch.int32, device=DEV)
    src, dst = torch.cat([src, src[:more], loops]), torch.cat([dst, dst[:more], loops])
    order = torch.randperm(src.numel(), generator=g, device=DEV)
    return src[order], dst[order]


def _drop_some(n, src, dst, seed):
    """A tenth of the vertices lose their out-edges (PageRank's dangling vertices)."""
    keep = (torch.rand(n, generator=_gen(seed + 77), device=DEV) >= 0.1)[src.long()]
    return src[keep], dst[keep]


def _case_edges(case, seed):
    n, src, dst = _edges(case, seed)
    if case["kind"] == "pagerank":
        src, dst = _drop_some(n, src, dst, seed)
    return n, src, dst


def _sources(case, seed, src, dst):
    """Seeded sources among the vertices that have an edge to another one."""
    k = case.get("sources", 1)
    pick = torch.randint(0, src.numel(), (64 * k + 256,), generator=_gen(seed + 1), device=DEV)
    s, d = src[pick], dst[pick]
    s = s[s != d][:k]
    return [int(x) for x in s.tolist()]


def _graph(case, n, src, dst, w):
    return G.make_graph(n, src, dst, case["directed"], w=w, weight_mode=G.WEIGHT_NONE)


WEIGHTED = ("suite", "sssp", "landmarks")


def prepare(case, seed):
    kind = case["kind"]
    n, src, dst = _case_edges(case, seed)
    if kind == "load":
        src, dst = _arriving(case, seed, n, src, dst)
        w = _weights(case, seed, src, dst) if case["weighted"] else None
        return {"case": case, "n": n, "src": src, "dst": dst, "w": w}
    if kind == "update":
        return _live(case, seed, n, src, dst)
    w = _weights(case, seed, src, dst) if kind in WEIGHTED else None
    sources = _sources(case, seed, src, dst)
    g = _graph(case, n, src, dst, w)
    del src, dst, w
    return {"case": case, "sources": sources, "g": G.ResidentGraph(g) if case["resident"] else g}


def _live(case, seed, n, src, dst):
    """A live graph, a batch of updates of it (half new edges, half deletes of
    present ones, each in both directions), and the batch that takes it back."""
    half, count = case["updates"] // 4, n * case["degree"] // 2
    src, dst = _distinct(n, src, dst, count + half, seed)
    w = _weights(case, seed, src, dst)
    g = _graph(case, n, src[:count], dst[:count], w[:count])
    gone = slice(0, half)
    new = slice(count, count + half)
    a, b = torch.cat([src[new], src[gone]]), torch.cat([dst[new], dst[gone]])
    v = torch.cat([w[new], torch.zeros(half, dtype=torch.float64, device=DEV)])
    order = torch.randperm(2 * half, generator=_gen(seed + 7), device=DEV)
    a, b, v = a[order], b[order], v[order]
    keys = torch.stack([G.edge_keys(a, b), G.edge_keys(b, a)], 1).reshape(-1)
    dyn = G.DynamicGraph.from_graph(g)
    return {"case": case, "dyn": dyn, "keys": keys, "values": v.repeat_interleave(2), "undo": dyn.find(keys)}


# ---------------------------------------------------------------- the passes
def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def _call(g, name, *args, **kw):
    return getattr(g, name)(*args, **kw) if isinstance(g, G.ResidentGraph) else getattr(G, name)(g, *args, **kw)


def _run_suite(state):
    """The six analytics of a benchmark run, one after another."""
    g, s = state["g"], state["sources"][0]
    out = {}
    if state["case"]["paths"]:  # shortest-path trees, not distances alone
        out["depth"], out["parent"] = _call(g, "bfs_pred", s)
        out["dist"], out["via"] = _call(g, "sssp_pred", s, inf=INF)
    else:
        out["depth"] = _call(g, "bfs", s)[0]
        out["dist"] = _call(g, "sssp", s, inf=INF)[0]
    out["component"] = _call(g, "wcc")
    out["rank"] = _call(g, "pagerank", 10, 0.85)[0]
    out["community"] = _call(g, "cdlp", 10)
    counts, _, triangles = _call(g, "tc")
    out["triangles_of"], out["triangles"] = counts, triangles
    return out


def _run_bfs(state):
    return [_call(state["g"], "bfs", s)[0] for s in state["sources"]]


def _run_sssp(state):
    return [_call(state["g"], "sssp", s, inf=INF)[0] for s in state["sources"]]


def _run_pagerank(state):
    return _call(state["g"], "pagerank", state["case"]["iterations"], 0.85)[0]


def _run_cdlp(state):
    return _call(state["g"], "cdlp", state["case"]["iterations"])


def _run_tc(state):
    counts, _, triangles = _call(state["g"], "tc")
    return counts, triangles


def _run_landmarks(state):
    """Hops and weighted distances from every landmark, each in one pass."""
    hops = state["g"].msbfs(state["sources"])[0]
    return {"hops": hops, "dist": state["g"].mssssp(state["sources"], inf=INF)[0]}


def _run_load(state):
    """Edge list -> CSR -> resident graph, and the first question asked of it."""
    g = G.make_graph(state["n"], state["src"], state["dst"], state["case"]["directed"], w=state["w"], weight_mode=G.WEIGHT_NONE)
    r = G.ResidentGraph(g)
    component = r.wcc()
    r.close()
    out = {"rowptr": g.rowptr, "col": g.col, "component": component}
    if g.w is not None:
        out["w"] = g.w
    return out


def _run_update(state):
    """A batch, the graph after it as a CSR, and the batch that takes it back."""
    dyn = state["dyn"]
    done = dyn.update(state["keys"], state["values"])
    g = dyn.csr_graph()
    undone = dyn.update(state["keys"], state["undo"])
    return {"rowptr": g.rowptr, "col": g.col, "w": g.w, "done": done, "undone": undone}


# --------------------------------------------------------------- the cases
def _resident(kind, name=None, family="rmat", **kw):
    c = {"kind": kind, "family": family, "directed": False, "resident": True, **kw}
    return {"name": name, **c} if name else c


def listed():
    return [
        # a small graph in an interactive session: every call is latency
        _resident("suite", "suite_small_directed", n=1000, degree=8, directed=True, resident=False, paths=False),
        # the standard small benchmark graph (scale 16), with path trees
        _resident("suite", "suite_rmat16", n=1 << 16, degree=16, paths=True),
        # hop distances on a social-size graph, source after source
        _resident("bfs", "bfs_rmat24", n=1 << 24, degree=16, sources=8),
        # hop distances on a road-like mesh: thousands of thin levels
        _resident("bfs", "bfs_grid", "grid", rows=2999, cols=2001, sources=1),
        # weighted distances on a social-size graph
        _resident("sssp", "sssp_rmat22", n=1 << 22, degree=16, sources=2),
        # weighted distances on a road-like mesh, straight on the caller's CSR
        _resident("sssp", "sssp_grid_raw", "grid", rows=1501, cols=1999, sources=1, resident=False),
        # ranks of a web-like directed graph with dangling pages
        _resident("pagerank", "pagerank_directed", n=12_000_017, degree=16, directed=True, iterations=10),
        # communities of an undirected social graph
        _resident("cdlp", "cdlp_rmat22", n=1 << 22, degree=16, iterations=10),
        # clustering counts of an undirected social graph
        _resident("tc", "tc_rmat21", n=1 << 21, degree=16),
        # distances from many landmarks at once
        _resident("landmarks", "landmarks_64", n=1 << 18, degree=16, sources=64),
        # a graph arrives as an edge list with weights
        _resident("load", "load_rmat22", n=1 << 22, degree=32, weighted=True),
        # a stream of edits on a live graph, its CSR taken after them
        _resident("update", "update_100k", n=1 << 21, degree=32, updates=100_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["suite", "bfs", "sssp", "pagerank", "cdlp", "tc", "landmarks", "load", "update"])
    top = {"suite": 1 << 17, "bfs": 1 << 23, "sssp": 1 << 21, "pagerank": 1 << 23, "cdlp": 1 << 21, "tc": 1 << 19, "landmarks": 1 << 17,
           "load": 1 << 21, "update": 1 << 21}[kind]
    low = {"suite": 60, "landmarks": 1000, "update": 50_000}.get(kind, 20_000)
    c = _resident(kind)
    c["directed"] = kind not in ("update",) and rng.random() < 0.4
    c["resident"] = kind == "landmarks" or rng.random() < 0.6
    if kind in ("bfs", "sssp", "load") and rng.random() < 0.35:
        c["family"], c["directed"] = "grid", False
        cells = min(top, 1 << 22)
        rows = _log_int(rng, 150, math.sqrt(cells))
        c["rows"], c["cols"] = rows, max(2, _log_int(rng, 20_000, cells) // rows)
    else:
        c["family"] = "er" if rng.random() < 0.25 else "rmat"
        c["n"], c["degree"] = _log_int(rng, low, top), rng.choice([3, 5, 8, 11, 16])
    if kind == "suite":
        c["paths"] = rng.random() < 0.5
    if kind in ("bfs", "sssp"):
        c["sources"] = rng.choice([1, 2, 3])
    if kind in ("pagerank", "cdlp"):
        c["iterations"] = rng.choice([5, 10, 20]) if kind == "pagerank" else rng.choice([3, 5, 10])
    if kind == "landmarks":
        c["sources"] = rng.choice([5, 16, 31, 64])
    if kind == "load":
        c["weighted"] = rng.random() < 0.5
    if kind == "update":
        c["updates"] = _log_int(rng, 500, 100_000)
    return c


# ------------------------------------------------------- what a pass must do
def work(case):
    """Each array read or written once: 4-byte ids and offsets, 8-byte weights,
    distances and ranks.  Entry counts are the generated ones (before repeats
    are dropped).  A call's iterations each read the graph."""
    kind = case["kind"]
    if case["family"] == "grid":
        n = case["rows"] * case["cols"]
        e = 2 * n
    else:
        n, e = case["n"], case["n"] * case["degree"]
    m = e if case["directed"] else 2 * e
    k = case.get("sources", 1)
    it = case.get("iterations", 1)
    graph = 4 * (n + 1) + 4 * m
    if kind == "suite":
        trees = 8 * n if case["paths"] else 0
        b = (graph + 4 * n) + (graph + 8 * m + 8 * n) + trees + (graph + 4 * n) + 10 * (graph + 16 * n) + 10 * (graph + 8 * n) + (graph + 8 * n)
        return {"bytes": b, "flops": 20 * m}
    if kind == "bfs":
        return {"bytes": k * (graph + 4 * n), "flops": 0}
    if kind == "sssp":
        return {"bytes": k * (graph + 8 * m + 8 * n), "flops": k * m}
    if kind == "pagerank":
        return {"bytes": it * (graph + 16 * n), "flops": 2 * it * m}
    if kind == "cdlp":
        return {"bytes": it * (graph + 8 * n), "flops": 0}
    if kind == "tc":
        return {"bytes": graph + 8 * n, "flops": 0}
    if kind == "landmarks":
        return {"bytes": 2 * graph + 8 * m + 12 * n * k, "flops": k * m}
    if kind == "load":
        w = 8 if case["weighted"] else 0
        if case["family"] != "grid":
            e //= 2
            m //= 2
            graph = 4 * (n + 1) + 4 * m
        both = 2 if case["directed"] else 1
        return {"bytes": (8 + w) * e + both * (4 * (n + 1) + (4 + w) * m) + graph + 4 * n, "flops": 0}
    return {"bytes": 2 * 16 * case["updates"] + 2 * (4 * (n + 1) + 6 * m), "flops": 0}


# ------------------------------------------------ the values in 64-bit torch
def _pairs(case, seed):
    """Directed entries without repeats or self-loops, by the CSR builder's rules."""
    n, src, dst = _case_edges(case, seed)
    if not case["directed"]:
        src, dst = torch.cat([src, dst]), torch.cat([dst, src])
    key = torch.unique((src.to(torch.int64) * n + dst)[src != dst])
    return n, key // n, key % n


def _exact_dist(n, u, v, w, source):
    dist = torch.full((n,), INF, dtype=torch.float64, device=u.device)
    dist[source] = 0.0
    while True:
        new = dist.scatter_reduce(0, v, dist[u] + w, "amin")
        if torch.equal(new, dist):
            return dist
        dist = new


def _exact_rank(n, u, v, iterations, damping=0.85):
    out = torch.bincount(u, minlength=n).to(torch.float64)
    sink = out == 0
    rank = torch.full((n,), 1.0 / n, dtype=torch.float64, device=u.device)
    for _ in range(iterations):
        share = torch.where(sink, 0.0, rank / out.clamp(min=1))
        base = (1 - damping) / n + damping * rank[sink].sum() / n
        rank = base + damping * torch.zeros_like(rank).index_add_(0, v, share[u])
    return rank


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("suite", "sssp", "pagerank", "landmarks"):
        return None
    entries = 4 * case["rows"] * case["cols"] if case["family"] == "grid" else case["n"] * case["degree"]
    if entries > (1 << 28):
        return None
    n0, src, dst = _case_edges(case, seed)
    sources = _sources(case, seed, src, dst)
    del src, dst
    n, u, v = _pairs(case, seed)
    if kind == "pagerank":
        return _exact_rank(n, u, v, case["iterations"])
    w = _weights(case, seed, u.to(torch.int32), v.to(torch.int32))
    if kind == "sssp":
        return [_exact_dist(n, u, v, w, s) for s in sources]
    if kind == "landmarks":
        return {"hops": None, "dist": torch.stack([_exact_dist(n, u, v, w, s) for s in sources])}
    out = {"depth": None, "dist": _exact_dist(n, u, v, w, sources[0]), "component": None, "rank": _exact_rank(n, u, v, 10), "community": None,
           "triangles_of": None, "triangles": None}
    if case["paths"]:
        out.update(parent=None, via=None)
    return out
