"""Components by sampled hooking (the default form of Graph.cc) where it can go
wrong: rows on either side of what a lane, a warp and a piece take, hubs outside
the most common component, chains (also in id order), many equal components,
graphs that list each edge once, directed graphs, self-loops and duplicates."""
import numpy as np
import pytest

import gswitch_b200 as gs
import oracle

pytestmark = pytest.mark.gpu


def csr(n, u, v):
    o = np.lexsort((v, u))
    off = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(u, minlength=n), out=off[1:])
    return off, v[o].astype(np.int32)


def labels(n, u, v):
    """The smallest vertex of each vertex's component."""
    lab = np.arange(n)
    while True:
        new = lab.copy()
        np.minimum.at(new, u, lab[v])
        np.minimum.at(new, v, lab[u])
        new = np.minimum(new, new[new])
        if np.array_equal(new, lab):
            return lab.astype(np.int32)
        lab = new


def graphs():
    r = np.random.default_rng(11)
    for d in (1, 2, 3, 15, 16, 17, 4095, 4096, 4097, 9000):
        # a hub of d leaves in ids above a larger component
        m = 3 * d + 40
        n = m + d + 1
        yield f"hub{d}", n, np.concatenate([np.arange(m - 1), np.full(d, n - 1)]), np.concatenate(
            [np.arange(1, m), np.arange(m, m + d)])
    p = r.permutation(4000)
    yield "chain", 4000, p[:-1], p[1:]
    yield "many", 6000, np.repeat(np.arange(0, 6000, 6), 6) + r.integers(0, 6, 6000), np.repeat(
        np.arange(0, 6000, 6), 6) + r.integers(0, 6, 6000)
    yield "random", 20000, r.integers(0, 20000, 18000), r.integers(0, 20000, 18000)
    yield "pair", 2, np.array([0]), np.array([1])
    yield "loops", 9, np.array([0, 3, 3, 4, 8]), np.array([0, 4, 4, 4, 3])


@pytest.mark.parametrize("case", list(graphs()), ids=lambda c: c[0])
def test_every_form_agrees(ctx, case):
    name, n, u, v = case
    ref = labels(n, u, v)
    lo, hi = np.minimum(u, v), np.maximum(u, v)
    both = (np.concatenate([u, v]), np.concatenate([v, u]))
    edges = int((lo < hi).sum())
    for a, b, directed in ((*both, False), (lo, hi, False), (u, v, True)):
        off, col = csr(n, a, b)
        g = ctx.upload(off, col, directed=directed)
        for o in (None, "x-Bitmap", "x-Queue"):
            lab, st = g.cc(o)
            assert np.array_equal(lab, ref), (name, directed, o)
            assert st.device_error == 0
            if not directed:
                assert st.edges == edges, (name, o)
        g.close()


def test_many_components_of_an_er_batch(ctx):
    g, voff = ctx.er_batch(60, seed=4, nlo=50, nhi=3000, dlo=0.5, dhi=9.0)
    off, col, _ = g.download()
    lab, st = g.cc()
    assert np.array_equal(lab, oracle.cc(oracle.Csr(off, col)))
    g.close()


def test_one_sided_arcs_keep_the_loop(ctx):
    """Arcs listed from one end only, in equal numbers up and down: the loop
    takes those whose column is the larger."""
    u, v = np.array([0, 1, 5, 4]), np.array([3, 2, 2, 0])
    off, col = csr(6, u, v)
    g = ctx.upload(off, col)
    want = g.cc("x-Bitmap")[0]
    assert np.array_equal(g.cc()[0], want)
    g.close()


def chains():
    n = 1 << 18
    yield "path", n, np.arange(n - 1), np.arange(1, n)
    # two paths, of the even and the odd ids, joined where both end
    yield "interleaved", n, np.concatenate([np.arange(n - 2), [n - 2]]), np.concatenate([np.arange(2, n), [n - 1]])
    at = np.arange(n).reshape(n // 4, 4)
    yield "strip", n, np.concatenate([at[:-1].ravel(), at[:, :-1].ravel()]), np.concatenate(
        [at[1:].ravel(), at[:, 1:].ravel()])


@pytest.mark.parametrize("case", list(chains()), ids=lambda c: c[0])
def test_chains_in_id_order(ctx, case):
    """Trees as deep as the graph is long (ids along a path or a mesh) are
    flattened before anything climbs them: the time stays near the loop's, where
    a climb of one vertex at a time takes a hundred times as long."""
    name, n, u, v = case
    off, col = csr(n, np.concatenate([u, v]), np.concatenate([v, u]))
    g = ctx.upload(off, col)
    loop = min(g.cc("x-Bitmap", out=False)[1].ms for _ in range(4))
    runs = [g.cc() for _ in range(4)]
    assert all(not lab.any() for lab, _ in runs)  # one component
    assert min(st.ms for _, st in runs) <= 4 * loop + 0.2, (loop, [st.ms for _, st in runs])
    g.close()


def test_passes_see_what_the_one_before_wrote(ctx):
    """The passes are set up while the one before still runs: many runs in a row on
    graphs of a few and of many CTAs, with other work on the same buffers between."""
    r = np.random.default_rng(5)
    for n, m in ((300, 280), (5000, 4000), (200000, 150000), (700000, 600000)):
        u, v = r.integers(0, n, m), r.integers(0, n, m)
        off, col = csr(n, np.concatenate([u, v]), np.concatenate([v, u]))
        g = ctx.upload(off, col)
        ref = g.cc("x-Bitmap")[0]
        for k in range(30):
            assert np.array_equal(g.cc()[0], ref), (n, k)
            if k % 3 == 0:
                g.bfs(int(u[k]), out=False)  # takes the labels' buffer for its levels
        g.close()
