"""The reference strategies where edges change kernels: lists of 47 to 50 entries around the bound of
the one-lane form, tails whose heads have short and long lists, groups cut by their entries and by
their tails, lists put together from several pieces.  Exact against the oracle for every method."""
import numpy as np
import pytest

from katric_gb300 import Config, Graph

pytestmark = pytest.mark.gpu


def csr(edges, n, shuffled):
    e = np.random.default_rng(2).permutation(n)[np.asarray(edges, dtype=np.int64)]
    src, dst = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    order = np.lexsort((np.random.default_rng(3).random(len(dst)) if shuffled else dst, src))
    fo = np.zeros(n + 1, dtype=np.uint64)
    fo[1:] = np.cumsum(np.bincount(src, minlength=n))
    return fo, dst[order].astype(np.uint32)


def cliques(sizes, fan):
    edges, n = [], 0
    for s in sizes:
        i, j = np.triu_indices(s, 1)
        edges.append(np.stack([i + n, j + n], 1))
        n += s
    if fan:  # `fan` triangles on one edge: tails of two entries, one edge between two hubs
        k = np.arange(fan) + n + 2
        edges += [np.array([[n, n + 1]]), np.stack([np.full(fan, n), k], 1), np.stack([np.full(fan, n + 1), k], 1)]
        n += 2 + fan
    return np.concatenate(edges), n


@pytest.mark.parametrize("method", ["merge", "binary-search", "binary", "hybrid"])
@pytest.mark.parametrize("sizes,fan", [((3,), 0), (tuple(range(2, 20)), 300), ((47, 48, 49, 50, 51, 52), 2000),
                                       ((60, 5, 70, 6, 97), 100)])
@pytest.mark.parametrize("shuffled", [False, True])
@pytest.mark.parametrize("wide", [False, True])
def test_short_and_long_lists(counter, oracle, method, sizes, fan, shuffled, wide):
    fo, hd = csr(*cliques(sizes, fan), shuffled)
    total, pv, _ = oracle.count(fo, hd, method="merge", num_threads=4)
    t, p = counter.count(fo, hd, Config(intersection_method=method, force_wide_offsets=wide))
    assert t == total and np.array_equal(p, pv)


@pytest.mark.parametrize("method", ["merge", "binary-search", "binary", "hybrid"])
@pytest.mark.parametrize("graph", ["rmat", "rgg", "gnm"])
def test_families(counter, oracle, method, graph):
    g = {"rmat": lambda: Graph.rmat(13, 24, seed=6), "rgg": lambda: Graph.rgg2d(30011, 70.0, seed=7),
         "gnm": lambda: Graph.gnm(20011, 900000, seed=8)}[graph]()
    total, pv, _ = oracle.count(g.first_out, g.head, method="merge", num_threads=8)
    t, p = counter.count(g.first_out, g.head, Config(intersection_method=method))
    assert t == total and np.array_equal(p, pv)
