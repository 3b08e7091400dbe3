"""The inspection's counters on either side of every line of its launch plan (two
or four thread groups, one virtual block per CTA or a resident wave), against the
oracle's restatement of the reference's grid."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 5, 511, 513, 131071, 131073, (1 << 19) - 3, 1 << 19, (1 << 19) + 1, (1 << 19) + 513,
                               3 * (1 << 19) + 7, (1 << 24) - 1, 1 << 24, (1 << 24) + 5])
def test_counters(ctx, n):
    r = np.random.default_rng(n)
    deg = np.zeros(n, np.int64)
    at = r.integers(0, n, 4000)
    deg[at] = r.integers(1, 300, 4000)
    off = np.zeros(n + 1, np.int64)
    np.cumsum(deg, out=off[1:])
    col = r.integers(0, n, off[-1]).astype(np.int32)
    h = oracle.Csr(off, col)
    levels = r.integers(-1, 3, n).astype(np.int32)
    g = ctx.upload(off, col)
    for level in (0, 2, 7):
        got = g.bfs_inspect(levels, level)
        ref = oracle.inspect_bfs(h, levels, level)
        assert np.array_equal(got, ref), (n, level)
        assert np.array_equal(g.bfs_inspect(levels, level), ref)  # the scratch is clean again
    g.close()
