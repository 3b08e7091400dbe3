"""The edge-balanced all-to-all expands (k_pull_all, k_push_all) at the sizes
where their tiles of 256 slots can go wrong: degrees around a tile and around a
lane's eight edges, hubs over many tiles, long runs of vertices without edges,
directed and undirected graphs, host and captured loops."""
import numpy as np
import pytest

import gswitch_b200 as gs

pytestmark = pytest.mark.gpu


def csr(n, u, v):
    """Arcs u -> v without duplicates or self-loops."""
    key = np.unique(u.astype(np.int64) * n + v)
    u, v = key // n, key % n
    u, v = u[u != v], v[u != v]
    off = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(u, minlength=n), out=off[1:])
    return off, v.astype(np.int32), u


def pagerank(n, off, col, src, iters, d=np.float32(0.85)):
    d = float(d)
    od = np.maximum(np.diff(off), 1).astype(np.float64)
    x = (1 - d) / od
    for _ in range(iters):
        x = (1 - d + d * np.bincount(col, weights=x[src], minlength=n)) / od
    return x


def graphs():
    r = np.random.default_rng(5)
    for deg in (1, 7, 8, 9, 255, 256, 257, 511, 512, 513, 5000):
        # every vertex past a gap of in-edge-free ones points at vertex 3
        n = deg + 700
        yield f"star{deg}", n, np.arange(n - deg, n), np.full(deg, 3)
    for gap in (31, 256, 3000):  # vertices with in-edges are `gap` apart
        n = 40 * gap + 5
        yield f"gap{gap}", n, r.integers(0, n, 900), r.integers(0, 40, 900) * gap
    yield "one", 2, np.array([0]), np.array([1])
    yield "random", 5001, r.integers(0, 5001, 60000), (r.random(60000) ** 3 * 5001).astype(np.int64)


@pytest.mark.parametrize("directed", [True, False])
@pytest.mark.parametrize("case", list(graphs()), ids=lambda c: c[0])
def test_tile_edges(ctx, case, directed):
    name, n, u, v = case
    if not directed:
        u, v = np.concatenate([u, v]), np.concatenate([v, u])
    off, col, src = csr(n, u, v)
    g = ctx.upload(off, col, directed=directed)
    ref = pagerank(n, off, col, src, 3)
    # FP32: eight serial and five shuffled additions a lane, one atomic a tile,
    # the filter's few operations, three iterations that carry 0.85 of the last one's error
    # (a push: one atomic an arc, so as many additions as the vertex has)
    top = np.bincount(col, minlength=n).max()
    bound = {"Pull": 2.6 * (20 + top / 256) * 2.0**-24, "Push": 2.6 * (20 + top) * 2.0**-24}
    for cfg in ("Pull-Bitmap-STRICT", "Push-Bitmap-STRICT"):
        for captured in (False, True):
            pr, st = g.pagerank(iters=3, eps=0.0, opts=gs.RunOpts.from_config(cfg, captured=captured))
            assert {t[:3] for t in st.trace} == {tuple(cfg.split("-"))}
            assert np.max(np.abs(pr - ref) / ref) <= bound[cfg[:4]], (name, cfg, captured)
    g.close()


def test_captured_graph_outlives_no_table(ctx):
    """A captured loop, a run on a larger graph that replaces the tables its
    bodies name, and the captured loop again: it is captured anew."""
    r = np.random.default_rng(9)
    small = csr(3000, r.integers(0, 3000, 20000), r.integers(0, 3000, 20000))
    big = csr(200000, r.integers(0, 200000, 3000000), (r.random(3000000) ** 4 * 200000).astype(np.int64))
    gs_, gb = (ctx.upload(x[0], x[1], directed=True) for x in (small, big))
    for cfg in ("Pull-Bitmap-STRICT", "Push-Bitmap-STRICT", "Pull-Bitmap-WM", "Push-Bitmap-CM"):
        cap = gs.RunOpts.from_config(cfg, captured=True)
        ref = pagerank(3000, small[0], small[1], small[2], 3)
        for _ in range(2):
            pr, _ = gs_.pagerank(iters=3, eps=0.0, opts=cap)
            # in-degrees below 40: 2.6 * (20 + 40) * 2^-24
            assert np.max(np.abs(pr - ref) / ref) <= 1e-5, cfg
            gb.pagerank(iters=2, eps=0.0, opts=cfg, out=False)
    gs_.close()
    gb.close()
