"""Colouring in dependency order (k_gc_dag), the default form of Graph.gc, where
it can go wrong: frontiers on either side of what one CTA takes, chains longer
than one stay on a CTA, rows longer than a warp's share, duplicates, directed
graphs, rows that are not sorted, arcs listed from one end only, and vertices
that are their own neighbour."""
import numpy as np
import pytest

import gswitch_b200 as gs
import oracle

pytestmark = pytest.mark.gpu


def colours(n, u, v):
    """A vertex takes the first level at which no uncoloured in-neighbour has a
    larger id (u -> v)."""
    u, v = u[u > v], v[u > v]
    colour = np.full(n, -1, np.int32)
    level = 0
    while True:
        level += 1
        held = np.zeros(n, bool)
        held[v] = True
        colour[(colour < 0) & ~held] = level
        if len(u) == 0:
            return colour
        left = colour[u] < 0
        u, v = u[left], v[left]


def csr(n, u, v, order=None):
    o = np.lexsort((v if order is None else order, u))
    off = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(u, minlength=n), out=off[1:])
    return off, v[o].astype(np.int32)


def both(u, v):
    return np.concatenate([u, v]), np.concatenate([v, u])


def hubs(sizes, k, late):
    """One vertex above d leaves for each d of sizes, k pairs; late: the hubs wait for
    one vertex, the pairs' larger ends for k others."""
    leaves, at = int(sum(sizes)), np.cumsum([0] + sizes)
    top = leaves + k + np.arange(len(sizes) + k)  # hubs, then the pairs' larger ends
    u = np.concatenate([np.repeat(top[:len(sizes)], sizes), top[len(sizes):]])
    v = np.concatenate([np.arange(leaves), leaves + np.arange(k)])
    if late:
        above = top[-1] + 1 + np.concatenate([np.zeros(len(sizes), int), 1 + np.arange(k)])
        u, v = np.concatenate([u, above]), np.concatenate([v, top])
    return u, v


def graphs():
    r = np.random.default_rng(3)
    for n in (1, 2, 33, 5000):  # a chain of n levels
        yield f"path{n}", n, np.arange(n - 1), np.arange(1, n)
    for n in (1023, 1025, 3000):  # frontiers of n - 1 vertices around one hub, smallest or largest
        yield f"star_low{n}", n, np.zeros(n - 1, int), np.arange(1, n)
        yield f"star_high{n}", n, np.full(n - 1, n - 1), np.arange(n - 1)
    # rows on either side of what a warp takes and of a piece, in frontiers of fewer
    # and of more vertices than the grid has warps, found by CTA 0 and by the grid
    for k, late in ((3, 0), (3, 1), (3000, 0), (6000, 0), (6000, 1)):
        u, v = hubs([255, 256, 1023, 1024, 1025, 1279, 1281, 8191, 8193, 30000], k, late)
        yield f"hubs{k}_{late}", int(max(u.max(), v.max())) + 1, u, v
    yield "clique", 300, *np.nonzero(np.triu(np.ones((300, 300), int), 1))
    yield "layers", 9000, np.repeat(np.arange(6000), 3), np.minimum(np.repeat(np.arange(6000), 3) + 3000 * (
        1 + np.arange(18000) % 2) // 2 + r.integers(0, 900, 18000), 8999)
    n = 40000
    yield "skewed", n, (r.random(400000) ** 4 * n).astype(int), r.integers(0, n, 400000)


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("case", list(graphs()), ids=lambda c: c[0])
def test_matches_the_levels(ctx, case, directed):
    name, n, u, v = case
    u, v = u[u != v], v[u != v]  # duplicates stay
    if not directed:
        u, v = both(u, v)
    ref = colours(n, u, v)
    off, col = csr(n, u, v)
    g = ctx.upload(off, col, directed=directed)
    got, st = g.gc()
    assert np.array_equal(got, ref)
    assert st.levels == ref.max() and st.device_error == 0
    g.close()
    # rows in another order: the level loop colours them
    off, col = csr(n, u, v, order=np.random.default_rng(1).random(len(v)))
    if n <= 5000 and len(col) and name != "path5000":
        g = ctx.upload(off, col, directed=directed)
        got, st = g.gc()
        assert np.array_equal(got, ref)
        assert st.levels == ref.max()
        g.close()


def test_more_levels_than_one_launch(ctx):
    n = (1 << 16) + 5000
    off, col = csr(n, *both(np.arange(n - 1), np.arange(1, n)))
    g = ctx.upload(off, col)
    got, st = g.gc()
    assert np.array_equal(got, np.arange(n, 0, -1, dtype=np.int32))
    assert st.levels == n
    g.close()


def test_own_neighbour_never_settles(ctx):
    u, v = both(np.array([0, 1, 2]), np.array([1, 2, 2]))
    off, col = csr(3, u, v)
    g = ctx.upload(off, col)
    with pytest.raises(gs.GswError) as e:
        g.gc()
    assert gs.STATUS[e.value.code] == "TIMEOUT"
    g.close()


def test_forced_and_recorded_runs_keep_the_level_loop(ctx):
    h = oracle.rmat(10, 8, seed=2)
    g = ctx.upload(h.off, h.col)
    ref = oracle.gc_levels(h)
    for o in ("Push-Queue-WM", "x-Bitmap", gs.RunOpts(timing=True), gs.RunOpts(persistent=False),
              gs.RunOpts(sorted_queue=False), gs.RunOpts(hub_path=0)):
        got, st = g.gc(o)
        assert np.array_equal(got, ref) and len(st.trace) == st.levels
    g.close()


def one_sided():
    r = np.random.default_rng(7)
    yield "pair", 2, np.array([0]), np.array([1])
    yield "mixed", 6, np.array([0, 1, 2, 3, 3, 3, 4, 5]), np.array([1, 3, 0, 1, 4, 5, 3, 3])
    for n, m in ((40, 60), (3000, 9000)):
        u, v = r.integers(0, n, m), r.integers(0, n, m)
        u, v = u[u != v], v[u != v]
        yield f"up{n}", n, np.minimum(u, v), np.maximum(u, v)
        yield f"down{n}", n, np.maximum(u, v), np.minimum(u, v)
        yield f"some{n}", n, u, v
        # as many arcs up as down, none listed from both ends
        yield f"balanced{n}", n, np.concatenate([np.arange(0, n - 1, 2), np.arange(2, n, 2)]), np.concatenate(
            [np.arange(1, n, 2), np.arange(1, n - 1, 2)])


@pytest.mark.parametrize("case", list(one_sided()), ids=lambda c: c[0])
def test_one_sided_arcs_keep_the_loop(ctx, case):
    """An undirected graph that lists an arc from one end only is coloured by
    the level loop, as it pulls and pushes along such arcs."""
    name, n, u, v = case
    off, col = csr(n, u, v)
    g = ctx.upload(off, col)
    want, ls = g.gc(gs.RunOpts(timing=True))
    got, st = g.gc()
    assert np.array_equal(got, want) and st.levels == ls.levels and st.trace == ls.trace
    if name == "mixed":
        assert got.tolist() == [4, 3, 1, 2, 1, 1]
    g.close()


def test_no_arcs(ctx):
    g = ctx.upload(np.zeros(71, np.int64), np.zeros(0, np.int32))
    got, st = g.gc()
    assert np.array_equal(got, np.ones(70, np.int32)) and st.levels == 1
    g.close()


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("late", [0, 1])
def test_long_rows_are_spread(ctx, directed, late):
    """A row of 2^18 smaller neighbours in a frontier of more vertices than the grid
    has warps takes no longer than the loop's sweeps (a lone warp: 7 ms)."""
    u, v = hubs([1 << 18], 6000, late)
    n = int(u.max()) + 1
    ref = colours(n, u, v)
    off, col = csr(n, u, v) if directed else csr(n, *both(u, v))
    g = ctx.upload(off, col, directed=directed)
    ms = []
    for _ in range(4):
        got, st = g.gc()
        assert np.array_equal(got, ref)
        ms.append(st.ms)
    loop = min(g.gc(gs.RunOpts(timing=True))[1].ms for _ in range(4))
    assert min(ms) <= 2 * loop + 0.3, (ms, loop)
    g.close()
