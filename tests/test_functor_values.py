"""Functors over vertex values of one to nine words: every expand builds for them
(one that stages values in shared memory is taken for 4-byte values only and must
not be compiled for wider ones), and every variant gives the sums of the messages,
ints and floats side by side in one value."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

import gswitch_b200 as gs
from gswitch_b200.build import ARCH, NVCC

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "gswitch_b200", "csrc")
SOURCE = os.path.join(HERE, "functor_values.cu")
FLAGS = [*ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-w", "-I", CSRC]


@pytest.mark.parametrize("words", [5, 9])
def test_every_expand_builds(tmp_path, words):
    r = subprocess.run([NVCC, *FLAGS, "-O1", f"-DVALUE_WORDS={words}", "-c", "-o", str(tmp_path / "f.o"), SOURCE],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]


# words of a value, and whether the functor sums its last float only (as betweenness
# sums the dependency beside a path count)
KINDS = [(1, 0), (2, 0), (2, 1), (3, 0), (4, 1), (9, 0)]


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    d = tmp_path_factory.mktemp("functors")
    jobs = {(w, one): subprocess.Popen([NVCC, *FLAGS, "-O3", "-Xcompiler", "-fPIC", "-shared", f"-DVALUE_WORDS={w}",
                                        *(["-DONE_WORD"] if one else []), "-o", str(d / f"f{w}{one}.so"), SOURCE])
            for w, one in KINDS}
    assert all(p.wait() == 0 for p in jobs.values())
    return {k: ctypes.CDLL(str(d / f"f{k[0]}{k[1]}.so")) for k in jobs}


def rows(n, u, v):
    o = np.lexsort((v, u))
    off = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(u, minlength=n), out=off[1:])
    return off, v[o].astype(np.int32)


def value_type(words):
    return np.dtype([("a", np.int32, ((words + 1) // 2,)), ("b", np.float32, (words // 2,))])


def level(L, words, n, u, v, directed, active, sends, cfg, everything=0, pruning=0, passes=1):
    p = lambda x: x.ctypes.data_as(ctypes.c_void_p)
    (off, col), (roff, rcol) = rows(n, u, v), rows(n, v, u)
    senders = np.zeros(n, np.dtype([("active", np.int32), ("sends", value_type(words))]))
    senders["active"], senders["sends"] = active, sends
    sums = np.zeros(n, value_type(words))
    d, f, lb = cfg
    rc = L.gather_level(n, ctypes.c_longlong(len(u)), p(off), p(col), p(roff), p(rcol), int(bool(directed)), p(senders), p(sums),
                        int(d == "Pull"), int(f == "Bitmap"), gs.LB[lb], everything, pruning, passes)
    assert rc == 0, (rc, cfg)
    return sums


def graph(directed):
    """Skewed, with a hub of 9,000 neighbours and long runs of vertices without any."""
    r = np.random.default_rng(8)
    n = 20000
    u = np.concatenate([(r.random(60000) ** 3 * n).astype(int), np.full(9000, 17)])
    v = np.concatenate([r.integers(0, n // 2, 60000), r.integers(0, n // 2, 9000)])
    return (n, u, v) if directed == "out" else (n, v, u) if directed == "in" else (n, np.concatenate([u, v]),
                                                                                   np.concatenate([v, u]))


def values(words, n, r):
    x = np.zeros(n, value_type(words))
    x["a"] = r.integers(-999, 999, x["a"].shape)
    x["b"] = r.integers(0, 16, x["b"].shape)  # whole: sums in any order are exact
    return x


def sums_of(n, u, v, x):
    out = np.zeros(n, x.dtype)
    np.add.at(out["a"], v, x["a"][u])
    np.add.at(out["b"], v, x["b"][u])
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("directed", ["", "out", "in"])
@pytest.mark.parametrize("words,one", KINDS)
def test_every_variant_sums_every_word(built, words, one, directed):
    n, u, v = graph(directed)
    L = built[words, one]
    r = np.random.default_rng(words)
    x, active = values(words, n, r), r.integers(0, 2, n).astype(np.int32)
    sent = (active[u] == 1) & (active[v] == 0)
    ref = sums_of(n, u[sent], v[sent], x)
    ref_all = sums_of(n, u, v, x)
    if one:
        for y in (ref, ref_all):
            y["a"], y["b"][:, :-1] = 0, 0
    for d in ("Push", "Pull"):
        for f in ("Queue", "Bitmap"):
            for lb in ("TM", "WM", "CM", "STRICT", "TWC"):
                got = level(L, words, n, u, v, directed, active, x, (d, f, lb))
                assert np.array_equal(got, ref), (d, f, lb)
                if f == "Bitmap":
                    got = level(L, words, n, u, v, directed, active, x, (d, f, lb), everything=1)
                    assert np.array_equal(got, ref_all), (d, f, lb, "all")


@pytest.mark.gpu
@pytest.mark.parametrize("lb", ["TM", "WM", "CM", "STRICT", "TWC"])
def test_pruned_push_delivers_to_a_target_once(built, lb):
    """conf_pruning: a target that has been sent to takes nothing in later levels, also
    where every vertex sends to every vertex."""
    n, u, v = graph("out")
    x = np.ones(n, value_type(1))
    indeg = np.bincount(v, minlength=n)
    got = level(built[1, 0], 1, n, u, v, "out", np.ones(n, np.int32), x, ("Push", "Bitmap", lb), everything=1, pruning=1,
                passes=2)["a"][:, 0]
    assert np.array_equal(got > 0, indeg > 0) and (got <= indeg).all()


@pytest.mark.gpu
@pytest.mark.parametrize("degree", [1, 2, 3, 4, 5, 31, 33, 300])
def test_pulls_of_few_messages_and_of_many_vertices(built, degree):
    """A CTA-mapped pull sends a warp's messages on one by one where they are few, or of
    many vertices, and folds them otherwise: on either side of both lines."""
    r = np.random.default_rng(degree)
    targets = 1500
    deg = r.integers(max(1, degree - 1), degree + 2, targets)
    v = np.repeat(np.arange(targets), deg)
    u = targets + r.integers(0, 5000, len(v))
    n = targets + 5000
    x = values(2, n, r)
    for share in (0.03, 0.22, 0.25, 0.28, 1.0):
        active = np.concatenate([np.zeros(targets, int), r.random(5000) < share]).astype(np.int32)
        sent = active[u] == 1
        ref = sums_of(n, u[sent], v[sent], x)
        for lb in ("WM", "CM"):
            got = level(built[2, 0], 2, n, u, v, "out", active, x, ("Pull", "Bitmap", lb))
            assert np.array_equal(got, ref), (share, lb)
