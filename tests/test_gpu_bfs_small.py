"""A small graph's BFS in one launch, where it can go wrong: rows on either side
of a piece and of several pieces, frontiers around a warp and a CTA, chains,
several roots (also repeated), directed graphs, the sizes around the line to the
level loop, and the runs that keep the loop."""
import numpy as np
import pytest

import gswitch_b200 as gs
import oracle
from test_gpu_cc_forest import csr

pytestmark = pytest.mark.gpu


def graphs():
    r = np.random.default_rng(2)
    for d in (1, 31, 32, 127, 128, 129, 255, 256, 257, 384, 385, 5000):
        # root - hub of d - each with 0..3 more
        mid = np.arange(2, d + 2)
        deep = r.integers(0, 4, d)
        tail = d + 2 + np.arange(deep.sum())
        yield f"hub{d}", d + 2 + int(deep.sum()), np.concatenate([[0], np.ones(d, int), np.repeat(mid, deep)]), np.concatenate(
            [[1], mid, tail])
    p = r.permutation(3000)
    yield "chain", 3000, p[:-1], p[1:]
    yield "random", 70001, r.integers(0, 70001, 300000), r.integers(0, 70001, 300000)
    yield "one", 1, np.zeros(0, int), np.zeros(0, int)
    yield "loops", 5, np.array([0, 0, 0, 1, 4]), np.array([0, 1, 1, 2, 4])


@pytest.mark.parametrize("directed", [False, True])
@pytest.mark.parametrize("case", list(graphs()), ids=lambda c: c[0])
def test_matches_the_oracle(ctx, case, directed):
    name, n, u, v = case
    off, col = csr(n, u, v) if directed else csr(n, np.concatenate([u, v]), np.concatenate([v, u]))
    h = oracle.Csr(off, col)
    g = ctx.upload(off, col, directed=directed)
    roots = sorted({0, n // 2, n - 1})
    for root in roots:
        ref = oracle.bfs(h, root)
        loop, ls = g.bfs(root, gs.RunOpts(persistent=False))
        got, st = g.bfs(root)
        assert np.array_equal(got, ref) and np.array_equal(loop, ref), (name, root)
        assert st.edges == ls.edges and st.device_error == 0
        # the last level finds nothing, or is the last that has arcs to follow
        assert ref.max() <= st.levels <= ref.max() + 1
    many = np.array(roots + roots[:1], np.int32)
    ref = np.stack([oracle.bfs(h, r) for r in roots]).astype(np.int64)
    ref = np.where(ref < 0, 1 << 40, ref).min(axis=0)
    got, st = g.bfs_multi(many)
    assert np.array_equal(got, np.where(ref == 1 << 40, -1, ref))
    loop, ls = g.bfs_multi(many, gs.RunOpts(persistent=False))
    assert np.array_equal(loop, got) and ls.edges == st.edges
    cap, sc = g.bfs_multi(many, gs.RunOpts(captured=True))
    assert np.array_equal(cap, got) and sc.edges == st.edges
    g.close()


@pytest.mark.parametrize("n,m", [((1 << 18) - 1, 400000), (1 << 18, 400000), ((1 << 18) + 1, 400000),
                                 (1 << 18, (1 << 22) - 2), (1 << 18, 1 << 22), (1 << 18, (1 << 22) + 2),
                                 (5000, 1 << 22), (5000, (1 << 22) + 2)])
def test_line_to_the_level_loop(ctx, n, m):
    """One launch up to 2^18 vertices and 2^22 arcs, the loop from there, with a hub of
    n - 1 arcs (duplicates too) so that the pieces of one row fill the queues."""
    r = np.random.default_rng(n + m)
    u, v = r.integers(0, n, m // 2), r.integers(0, n, m // 2)
    u[:n // 2] = 7
    off, col = csr(n, np.concatenate([u, v]), np.concatenate([v, u]))
    assert len(col) == m
    g = ctx.upload(off, col)
    h = oracle.Csr(off, col)
    for root in (int(v[-1]), 7):
        lv, st = g.bfs(root)
        assert np.array_equal(lv, oracle.bfs(h, root))
        one = n <= 1 << 18 and m <= 1 << 22
        assert (len(st.trace) == 1 and st.level_persistent == [True]) == one, (len(st.trace), st.level_persistent)
        loop, ls = g.bfs(root, gs.RunOpts(timing=True))
        assert np.array_equal(loop, lv) and ls.edges == st.edges
    g.close()


def test_asked_for_levels_keep_the_loop(ctx):
    h = oracle.rmat(11, 8, seed=2)
    g = ctx.upload(h.off, h.col)
    ref = oracle.bfs(h, 0)
    for o in (gs.RunOpts(timing=True), gs.RunOpts(account=True), gs.RunOpts(persistent=False),
              gs.RunOpts(captured=True), gs.RunOpts(sorted_queue=False), gs.RunOpts(hub_path=1),
              gs.RunOpts(captured=True, selector="mlp"), "Push-Queue-TM", "x-x-x-Standalone"):
        lv, st = g.bfs(0, o)
        assert np.array_equal(lv, ref) and len(st.trace) > 1, o
    for o in (None, gs.RunOpts(selector="mlp")):  # who picks variants is no wish for a loop
        lv, st = g.bfs(0, o)
        assert np.array_equal(lv, ref) and len(st.trace) == 1 and st.level_persistent == [True], o
    g.close()
