"""The batched pulls and their hub pieces where they can go wrong: in-degrees on
either side of a round, a tile, the hub lines and a hub piece, whole and divided
vertices at the ends of a window, every mapping and STRICT tile; hubs of a directed
graph, whose in-degrees no out-degree bounds."""
import numpy as np
import pytest

import gswitch_b200 as gs
import oracle
from test_gpu_push_batch import csr

pytestmark = pytest.mark.gpu


def layers(d, r):
    """0 - a layer of d - one vertex joined to all of it - 40 vertices of odd
    degrees - a tail: levels that pull d messages into one vertex and a few into
    many."""
    a = np.arange(1, d + 1)
    hub = d + 1
    odd = np.arange(hub + 1, hub + 41)
    deg = r.integers(1, 70, 40)
    tail = hub + 41 + np.arange(sum(deg))
    u = np.concatenate([np.zeros(d, int), a, np.full(40, hub), np.repeat(odd, deg)])
    v = np.concatenate([a, np.full(d, hub), odd, tail])
    return csr(int(tail[-1]) + 1, np.concatenate([u, v]), np.concatenate([v, u]), np.ones(2 * len(u), int))


@pytest.mark.parametrize("d", [1, 31, 32, 33, 127, 129, 511, 512, 1021, 1023, 1024, 1025, 2047, 4095, 4096, 8191, 8193,
                               20000])
def test_every_pull(ctx, d):
    h = layers(d, np.random.default_rng(d))
    lv, (nsp, _) = oracle.bfs(h, 0), oracle.bc_f32(h, 0)
    _, dep, _ = oracle.bc_f64(h, 0)
    lab = oracle.gc_levels(h)
    g = ctx.upload(h.off, h.col, h.w)
    dist = oracle.sssp_dijkstra(h, 0)
    try:
        for shape in (0, 1, 2):
            t = np.zeros(gs.TUNE_ENTRIES, np.int32)
            for fmt in ("Queue", "Bitmap"):
                t[ctx.tune_index("Pull", fmt, "STRICT")] = shape
            ctx.tune_load_shapes(t)
            for fmt in ("Queue", "Bitmap"):
                for lb in ("WM", "CM", "STRICT") if shape == 0 else ("STRICT",):
                    cfg = f"Pull-{fmt}-{lb}-Standalone"
                    assert np.array_equal(g.bfs(0, cfg)[0], lv), cfg
                    assert np.array_equal(g.sssp(0, cfg)[0], dist), cfg
                    got, gdep, _ = g.bc(0, cfg)
                    assert np.array_equal(got, nsp), cfg
                    assert np.max(np.abs(gdep - dep) / np.maximum(np.abs(dep), 1)) <= 1e-5, cfg
                    if d <= 1025:
                        assert np.array_equal(g.gc(cfg)[0], lab), cfg
    finally:
        ctx.tune_load_shapes(None)
        g.close()


@pytest.mark.parametrize("lb", ["WM", "CM"])
@pytest.mark.parametrize("d", [8191, 8192, 8193, 400000])
def test_directed_hub(ctx, d, lb):
    """0 -> a layer of d -> one vertex, with 3 or with 5,000 columns of its own: its
    in-edges are spread over the CTAs whichever out-degree it has (a lone warp or
    CTA takes 400,000 of them 30 times as long as the grid)."""
    ms = {}
    for own in (3, 5000):
        a, hub = np.arange(1, d + 1), d + 1
        u = np.concatenate([np.zeros(d, int), a, np.full(own, hub)])
        v = np.concatenate([a, np.full(d, hub), hub + 1 + np.arange(own)])
        h = csr(hub + 1 + own, u, v, np.ones(len(u), int))
        lv = oracle.bfs(h, 0)
        g = ctx.upload(h.off, h.col, directed=True)
        cfg = f"Pull-Bitmap-{lb}-Standalone"
        runs = []
        for _ in range(4):
            got, st = g.bfs(0, gs.RunOpts.from_config(cfg, timing=True))
            assert np.array_equal(got, lv), (d, cfg, own)
            runs.append(st.level_ms[1])  # the level that finds the hub
        ms[own] = min(runs)
        nsp, _, _ = g.bc(0, cfg)
        assert np.array_equal(nsp, oracle.bc_f32(h, 0)[0]), (d, cfg, own)
        g.close()
    if d == 400000:
        assert ms[3] <= 3 * ms[5000] + 0.05, ms
