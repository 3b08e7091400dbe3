"""The batched pushes (several edges of a thread in flight) at the edges of their
rounds: frontier and row sizes around 32, 128, 256 and 1,024 slots, every mapping
and tile, messages that a target already drops, duplicates and self-loops."""
import numpy as np
import pytest

import gswitch_b200 as gs
import oracle

pytestmark = pytest.mark.gpu


def csr(n, u, v, w):
    o = np.lexsort((v, u))
    off = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(u, minlength=n), out=off[1:])
    return oracle.Csr(off, v[o].astype(np.int32), w[o].astype(np.int32))


def fan(k, d, r):
    """0 -> k vertices -> d arcs each among 3k + 7 targets, a longer arc too."""
    mid, top = np.arange(1, k + 1), k + 1 + r.integers(0, 3 * k + 7, k * d)
    u = np.concatenate([np.zeros(k, int), np.repeat(mid, d), np.zeros(5, int)])
    v = np.concatenate([mid, top, top[:5] if len(top) >= 5 else np.zeros(5, int)])
    w = np.concatenate([r.integers(1, 9, k), r.integers(1, 50, k * d), np.full(5, 60)])
    return csr(4 * k + 8, np.concatenate([u, v]), np.concatenate([v, u]), np.concatenate([w, w]))


@pytest.mark.parametrize("k,d", [(1, 1), (31, 4), (32, 4), (33, 3), (127, 1), (128, 9), (255, 4), (257, 3), (1023, 1),
                                 (1025, 2), (3, 1021), (2, 4099)])
def test_sssp_and_bfs_every_push(ctx, k, d):
    h = fan(k, d, np.random.default_rng(k * 31 + d))
    ref, lv = oracle.sssp_dijkstra(h, 0), oracle.bfs(h, 0)
    g = ctx.upload(h.off, h.col, h.w)
    try:
        for shape in (0, 1, 2):  # STRICT tiles of 1,024, 512 and 2,048 slots
            t = np.zeros(gs.TUNE_ENTRIES, np.int32)
            for fmt in ("Queue", "Bitmap"):
                for fused in (False, True):
                    t[ctx.tune_index("Push", fmt, "STRICT", fused)] = shape
            ctx.tune_load_shapes(t)
            for fmt in ("Queue", "Bitmap"):
                for lb in ("TM", "WM", "CM", "STRICT", "TWC") if shape == 0 else ("STRICT",):
                    for fu in ("Standalone", "Fused"):
                        for persistent in ((None, False) if fu == "Fused" else (None,)):
                            o = gs.RunOpts.from_config(f"Push-{fmt}-{lb}-{fu}", persistent=persistent)
                            assert np.array_equal(g.sssp(0, o)[0], ref), vars(o)
                            assert np.array_equal(g.bfs(0, o)[0], lv), vars(o)
    finally:
        ctx.tune_load_shapes(None)
        g.close()
