"""Performance cases: the calls a program that uses gswitch_b200 makes, over the
sizes it makes them at.

A program keeps one Context with the committed selector models and tuning table
loaded, uploads its graphs (host CSR) into it and runs applications on them.
`prepare` therefore builds a host CSR from the seed, uploads it and picks the
roots; `run` is one application call that returns the whole result to the host.
Calls on small graphs go through the Python methods of Graph, which return fresh
arrays; calls on large graphs go through the C ABI with a page-locked result
buffer that the program keeps, as bench.py's end-to-end leg does.

Graphs:
  rmat   Graph500 quadrant probabilities, ids folded into [0, n) when n is no
         power of two: the skewed graphs (social networks, web) of the benchmark;
  er     G(n, m): uniform degrees;
  grid   lattice plus 1% long-range edges: road-like, many levels;
  batch  a disjoint union of G(n, m) graphs, one BFS root in each.
Arc counts in `work` are those of the construction, before self-loops and
duplicates go.
"""
import ctypes
import math

import numpy as np
import torch

import gswitch_b200 as gs

DEV = "cuda:0"
INF = 2**31 - 1
_CTX = []


def _context():
    """The program's one context, with the learned selector and the tuned
    launch table loaded."""
    if not _CTX:
        from gswitch_b200 import autotune, selector_train

        c = gs.Context(0)
        autotune.load_into(c)
        model, conf = selector_train.load_model()
        if model is not None:
            c.mlp_load(model, conf)
        model, conf = selector_train.load_fusion_model()
        if model is not None:
            c.mlp_load_fusion(model, conf)
        _CTX.append(c)
    return _CTX[0]


# ---- the cases --------------------------------------------------------------
def listed():
    return [
        # the smallest call: one query on a small graph, where launches and host
        # round trips are all there is
        {"name": "bfs_tiny", "app": "bfs", "graph": "rmat", "n": 1024, "ef": 16, "selector": "rules", "pinned": False},
        # the benchmark's smallest named graph (RMAT 2^16), default options
        {"name": "bfs_rmat16", "app": "bfs", "graph": "rmat", "n": 1 << 16, "ef": 16, "selector": "rules", "pinned": False},
        # the benchmark's headline graph (RMAT 2^24) with the learned selector
        {"name": "bfs_rmat24", "app": "bfs", "graph": "rmat", "n": 1 << 24, "ef": 16, "selector": "mlp", "pinned": True},
        # shortest paths on a skewed graph, weights 1..64
        {"name": "sssp_rmat22", "app": "sssp", "graph": "rmat", "n": 1 << 22, "ef": 16, "wmax": 64, "selector": "mlp", "pinned": True},
        # shortest paths on a road-like graph: hundreds of small levels; odd sides
        {"name": "sssp_grid", "app": "sssp", "graph": "grid", "rows": 2047, "cols": 2049, "wmax": 1000, "selector": "mlp", "pinned": True},
        # 20 PageRank iterations on a skewed graph with the learned selector
        {"name": "pagerank_rmat22", "app": "pagerank", "graph": "rmat", "n": 1 << 22, "ef": 16, "iters": 20, "selector": "mlp", "pinned": True},
        # the same on a smaller directed graph of odd size with default options (a web crawl)
        {"name": "pagerank_directed", "app": "pagerank", "graph": "rmat", "n": 300007, "ef": 8, "directed": True, "iters": 20,
         "selector": "rules", "pinned": False},
        # connected components
        {"name": "cc_rmat22", "app": "cc", "graph": "rmat", "n": 1 << 22, "ef": 16, "selector": "rules", "pinned": True},
        # betweenness from one source: the forward and the backward sweep
        {"name": "bc_rmat20", "app": "bc", "graph": "rmat", "n": 1 << 20, "ef": 16, "sources": 1, "selector": "rules", "pinned": True},
        # greedy colouring by id: several hundred levels that shrink slowly
        {"name": "gc_rmat18", "app": "gc", "graph": "rmat", "n": 1 << 18, "ef": 16, "selector": "rules", "pinned": True},
        # 64 BFS queries answered together (one word of the bit-sliced form)
        {"name": "mbfs_rmat18", "app": "mbfs", "graph": "rmat", "n": 1 << 18, "ef": 16, "sources": 64, "selector": "rules", "pinned": True},
        # BFS over 256 graphs of mixed sizes in one level loop
        {"name": "bfs_graph_batch", "app": "bfs_multi", "graph": "batch", "count": 256, "nhi": 60000, "selector": "mlp", "pinned": True},
    ]


# largest drawn graph per application, in vertices at 16 edges each (n * ef is
# kept below the same product)
_TOP = {"bfs": 1 << 23, "sssp": 1 << 21, "pagerank": 1 << 21, "cc": 1 << 22, "bc": 1 << 20, "gc": 1 << 17, "mbfs": 1 << 18}


def draw(rng):
    app = rng.choice(["bfs", "bfs", "sssp", "pagerank", "cc", "bc", "gc", "mbfs", "bfs_multi"])
    case = {"app": app, "selector": rng.choice(["rules", "mlp"])}
    if app == "bfs_multi":
        case.update(graph="batch", count=rng.randint(2, 256), nhi=int(math.exp(rng.uniform(math.log(2000), math.log(60000)))))
        case["pinned"] = case["count"] * case["nhi"] > 1 << 20
        return case
    top = _TOP[app]
    n = int(math.exp(rng.uniform(math.log(1000), math.log(top))))
    case["graph"] = rng.choice(["rmat", "rmat", "er"] + (["grid"] if app in ("bfs", "sssp", "bc") else []))
    if case["graph"] == "grid":
        n = min(n, 1 << 21)
        case["rows"] = max(2, int(math.sqrt(n) * math.exp(rng.uniform(-0.7, 0.7))))
        case["cols"] = max(2, n // case["rows"])
    else:
        # components: a uniform graph above that density is one component
        case["ef"] = rng.randint(1, 2) if app == "cc" and case["graph"] == "er" else rng.randint(2, 24)
        case["n"] = max(1000, min(n, 16 * top // case["ef"]))
        if app in ("bfs", "pagerank") and n < 1 << 18 and rng.random() < 0.3:
            case["directed"] = True
    if app == "sssp":
        case["wmax"] = rng.choice([16, 64, 1000])
    if app == "pagerank":
        case["iters"] = rng.choice([5, 10, 20])
    if app == "bc":
        case["sources"] = rng.choice([1, 1, rng.randint(2, 32)]) if n <= 1 << 17 else 1
    if app == "mbfs":
        case["sources"] = rng.randint(2, 128)
    case["pinned"] = n > 100000
    return case


# ---- graphs -----------------------------------------------------------------
def _sizes(case):
    """(vertices, arcs) of the construction."""
    if case["graph"] == "grid":
        n = case["rows"] * case["cols"]
        return n, int(2 * 1.01 * (2 * n - case["rows"] - case["cols"]))
    if case["graph"] == "batch":
        lo, hi = 1000.0, float(case["nhi"])
        n = int(case["count"] * (hi - lo) / math.log(hi / lo))
        return n, 18 * n
    return case["n"], case["n"] * case["ef"] * (1 if case.get("directed") else 2)


def _rng(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 2654435761 % (1 << 62) + 12345)


def _rmat_pairs(n, m, r):
    """m pairs by quadrant (a, b, c, d) = (.57, .19, .19, .05), folded into [0, n)."""
    u = torch.zeros(m, dtype=torch.int64, device=DEV)
    v = torch.zeros(m, dtype=torch.int64, device=DEV)
    for _ in range(max(1, math.ceil(math.log2(n)))):
        x = torch.rand(m, generator=r, device=DEV)
        u.mul_(2).add_(x >= 0.76)
        v.mul_(2).add_(((x >= 0.57) & (x < 0.76)) | (x >= 0.95))
        del x
    return u.remainder_(n), v.remainder_(n)


def _pairs(case, r):
    """(n, sources, targets, first vertex of each part)."""
    kind = case["graph"]
    if kind == "grid":
        rows, cols = case["rows"], case["cols"]
        n = rows * cols
        at = torch.arange(n, device=DEV).view(rows, cols)
        near_u = torch.cat([at[:, :-1].reshape(-1), at[:-1].reshape(-1)])
        near_v = torch.cat([at[:, 1:].reshape(-1), at[1:].reshape(-1)])
        far = torch.randint(n, (2, max(1, near_u.numel() // 100)), generator=r, device=DEV)
        return n, torch.cat([near_u, far[0]]), torch.cat([near_v, far[1]]), None
    if kind == "batch":
        # the sizes are the case's; the seed draws the edges
        x = torch.rand((2, case["count"]), generator=_rng(case["count"]), device=DEV, dtype=torch.float64)
        sizes = (1000.0 * (case["nhi"] / 1000.0) ** x[0]).long()
        pairs = (sizes * (4.0 + 28.0 * x[1]) / 2).long()
        first = torch.cumsum(sizes, 0) - sizes
        part = torch.repeat_interleave(torch.arange(case["count"], device=DEV), pairs)
        f = torch.rand((2, part.numel()), generator=r, device=DEV, dtype=torch.float64)
        u, v = ((f * sizes[part]).long().clamp_(max=sizes[part] - 1) + first[part])
        return int(sizes.sum()), u, v, first
    n, m = case["n"], case["n"] * case["ef"]
    if kind == "rmat":
        return (n, *_rmat_pairs(n, m, r), None)
    u, v = torch.randint(n, (2, m), generator=r, device=DEV)
    return n, u, v, None


def _graph(case, seed):
    """The case's graph and roots on the device: offsets, columns (sorted, no
    duplicates, no self-loops), weights or None, roots."""
    r = _rng(seed)
    n, u, v, first = _pairs(case, r)
    keep = u != v
    u, v = u[keep], v[keep]
    key = u * n + v
    if not case.get("directed"):
        key = torch.cat([key, v * n + u])
    del u, v, keep
    key = torch.unique(key)
    src = key // n
    col = key - src * n
    del key
    deg = torch.bincount(src, minlength=n)
    off = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    torch.cumsum(deg, 0, out=off[1:])
    w = None
    if case.get("wmax"):
        h = torch.minimum(src, col) * 73856093 + torch.maximum(src, col) * 19349663 + int(seed) * 83492791
        h = (h ^ (h >> 15)) * 40503
        w = ((h ^ (h >> 13)) & 0x7FFFFFFF).remainder_(case["wmax"]).add_(1).to(torch.int32)
        del h
    del src
    if first is not None:  # one root in each part
        roots = first
    else:
        alive = torch.nonzero(deg).view(-1)
        roots = alive[torch.randint(alive.numel(), (case.get("sources", 1),), generator=r, device=DEV)]
    return off, col.to(torch.int32), w, roots.to(torch.int32)


# ---- one pass ---------------------------------------------------------------
class _State:
    """An uploaded graph, its roots, the options and the result buffers."""


def prepare(case, seed):
    off, col, w, roots = _graph(case, seed)
    s = _State()
    s.case = case
    s.g = _context().upload(off.cpu().numpy(), col.cpu().numpy(), None if w is None else w.cpu().numpy(),
                            directed=bool(case.get("directed")))
    s.roots = np.ascontiguousarray(roots.cpu().numpy())
    s.out = []
    if case["pinned"]:
        n, k = s.g.n, case.get("sources", 1)
        shape = (k, n) if case["app"] == "mbfs" or k > 1 else (n,)
        types = {"pagerank": [torch.float32], "bc": [torch.int32, torch.float32]}.get(case["app"], [torch.int32])
        s.out = [torch.empty(shape, dtype=t, pin_memory=True).numpy() for t in types]
    return s


def _opts(case):
    o = gs.RunOpts(selector=case["selector"])
    if case["app"] == "pagerank":  # a fixed number of iterations
        o.max_iters, o.eps = case["iters"], 0.0
    return o


def run(s):
    case, g, o = s.case, s.g, _opts(s.case)
    app, root = case["app"], int(s.roots[0])
    if case["pinned"]:
        L, roots = gs.lib(), s.roots.ctypes.data_as(ctypes.c_void_p)
        if app in ("bfs", "sssp") or (app == "bc" and len(s.roots) == 1):
            fn = {"bfs": L.gsw_bfs, "sssp": L.gsw_sssp, "bc": L.gsw_bc}[app]
            g._run(fn, ctypes.c_int32(root), outs=s.out, opts=o)
        elif app == "mbfs":
            g._run(L.gsw_mbfs, len(s.roots), roots, 1, outs=s.out, opts=o)
        elif app == "bc":
            g._run(L.gsw_bc_batch, len(s.roots), roots, outs=s.out, opts=o)
        elif app == "bfs_multi":
            g._run(L.gsw_bfs_multi, len(s.roots), roots, outs=s.out, opts=o)
        else:
            g._run({"cc": L.gsw_cc, "gc": L.gsw_gc, "pagerank": L.gsw_pagerank}[app], outs=s.out, opts=o)
        return s.out
    if app == "bfs":
        return [g.bfs(root, o)[0]]
    if app == "bfs_multi":
        return [g.bfs_multi(s.roots, o)[0]]
    if app == "sssp":
        return [g.sssp(root, o)[0]]
    if app == "mbfs":
        return [g.mbfs(s.roots, opts=o)[0]]
    if app == "bc":
        return list(g.bc(root, o)[:2]) if len(s.roots) == 1 else list(g.bc_batch(s.roots, o)[:2])
    if app == "pagerank":
        return [g.pagerank(iters=case["iters"], eps=0.0, opts=o)[0]]
    return [g.cc(o)[0] if app == "cc" else g.gc(o)[0]]


def work(case):
    """The CSR once (the two sweeps of betweenness and every PageRank iteration
    need it again), and the result once."""
    n, m = _sizes(case)
    app, k = case["app"], case.get("sources", 1)
    csr = 8 * (n + 1) + 4 * m
    if app == "pagerank":  # columns, offsets, old and new value of a vertex per iteration
        return {"bytes": case["iters"] * (csr + 8 * n) + 4 * n, "flops": case["iters"] * (m + 3 * n)}
    if app == "bc":
        return {"bytes": 2 * csr + 8 * n * k, "flops": 3 * m * k}
    if app == "sssp":
        csr += 4 * m
    return {"bytes": csr + 4 * n * k, "flops": 0}


def tolerance(case):
    """Levels, distances, labels, colours and path counts are whole numbers with
    one right answer.  PageRank and the dependencies are FP32 sums whose order is
    free: against 64 bits they are off by up to 3e-7 (2-norm) and, where a hub's
    sum runs serially, by up to 5e-5 of a value."""
    return {"rel": 2e-6, "max": 1e-4} if case["app"] in ("pagerank", "bc") else "exact"


# ---- the same results from plain torch --------------------------------------
def _levels(src, dst, n, roots):
    lvl = torch.full((n,), -1, dtype=torch.int64, device=DEV)
    lvl[roots] = 0
    level = 0
    while True:
        d = dst[lvl[src] == level]
        d = d[lvl[d] < 0]
        if d.numel() == 0:
            return lvl
        level += 1
        lvl[d] = level


def _dependencies(src, dst, n, root):
    lvl = _levels(src, dst, n, root)
    down = lvl[dst] == lvl[src] + 1
    down &= lvl[src] >= 0
    src, dst = src[down], dst[down]
    at = lvl[src]
    nsp = torch.zeros(n, dtype=torch.float64, device=DEV)
    nsp[root] = 1
    last = int(lvl.max())
    for level in range(last):
        e = at == level
        nsp.index_add_(0, dst[e], nsp[src[e]])
    dep = torch.zeros(n, dtype=torch.float64, device=DEV)
    for level in range(last - 1, -1, -1):
        e = at == level
        part = torch.zeros(n, dtype=torch.float64, device=DEV)
        part.index_add_(0, src[e], (1 + dep[dst[e]]) / nsp[dst[e]])
        dep += part * nsp
    return nsp.long(), dep


def _components(src, dst, n):
    lab = torch.arange(n, device=DEV)
    while True:
        new = lab.scatter_reduce(0, src, lab[dst], "amin")
        new = torch.minimum(new, lab.scatter_reduce(0, lab[src], lab[dst], "amin"))
        while not torch.equal(new, new[new]):
            new = new[new]
        if torch.equal(new, lab):
            return lab
        lab = new


def _colours(src, dst, n):
    """A vertex takes the first round in which no uncoloured neighbour has a
    larger id."""
    up = dst > src
    src, dst = src[up], dst[up]
    colour = torch.full((n,), -1, dtype=torch.int64, device=DEV)
    level = 0
    while True:
        level += 1
        held = torch.zeros(n, dtype=torch.bool, device=DEV)
        held[src] = True
        colour[(colour < 0) & ~held] = level
        if src.numel() == 0:
            return colour
        left = colour[dst] < 0
        src, dst = src[left], dst[left]


def exact(case, seed):
    off, col, w, roots = _graph(case, seed)
    n, dst, roots = off.numel() - 1, col.long(), roots.long()
    src = torch.repeat_interleave(torch.arange(n, device=DEV), off[1:] - off[:-1])
    app = case["app"]
    if app in ("bfs", "bfs_multi"):
        return [_levels(src, dst, n, roots)]
    if app == "mbfs":
        return [torch.stack([_levels(src, dst, n, r) for r in roots])]
    if app == "cc":
        return [_components(src, dst, n)]
    if app == "gc":
        return [_colours(src, dst, n)]
    if app == "bc":
        both = [_dependencies(src, dst, n, r) for r in roots]
        if len(both) == 1:
            return list(both[0])
        return [torch.stack([b[0] for b in both]), torch.stack([b[1] for b in both])]
    if app == "sssp":
        dist = torch.full((n,), INF, dtype=torch.int64, device=DEV)
        dist[roots[0]] = 0
        while True:
            new = dist.scatter_reduce(0, dst, (dist[src] + w).clamp_(max=INF), "amin")
            if torch.equal(new, dist):
                return [dist]
            dist = new
    # PageRank: value over out-degree (the value itself for a sink)
    od = (off[1:] - off[:-1]).double().clamp_(min=1)
    d = float(np.float32(0.85))
    x = (1 - d) / od
    for _ in range(case["iters"]):
        got = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, dst, x[src])
        x = (1 - d + d * got) / od
    return [x]
