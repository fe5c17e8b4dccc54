"""Split out-lists (hubs as 16-bit indices counted in bitmaps, the rest hashed): exact against the
oracle on graphs above the size line, at the edges of the hub choice and of the hub lists."""
import functools

import numpy as np
import pytest

from katric_gb300 import Config, TriangleCounter, _native

pytestmark = pytest.mark.gpu

N = 1 << 21  # most vertices isolated: every graph is above the size line


def csr(e, n=N, shuffled=False):
    e = np.unique(np.sort(e, axis=1), axis=0)
    e = e[e[:, 0] != e[:, 1]]
    e = np.random.default_rng(7).permutation(n)[e]  # hubs anywhere in the id range
    src, dst = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    order = np.lexsort((np.random.default_rng(8).random(len(dst)) if shuffled else dst, src))
    fo = np.zeros(n + 1, dtype=np.uint64)
    fo[1:] = np.cumsum(np.bincount(src, minlength=n))
    return fo, dst[order].astype(np.uint32)


def dense_core(core, density, seed=1):
    """A random core of the given density, every core vertex with 150 pendant neighbours, and a fringe
    of vertices adjacent to 1..40 core vertices."""
    rng = np.random.default_rng(seed)
    i, j = np.triu_indices(core, 1)
    keep = rng.random(len(i)) < density
    parts = [np.stack([i[keep], j[keep]], 1)]
    parts.append(np.stack([np.repeat(np.arange(core), 150), rng.integers(core, N, core * 150)], 1))
    fringe = np.repeat(np.arange(core, core + 20000), 1 + np.arange(20000) % 40)
    parts.append(np.stack([fringe, rng.integers(0, core, len(fringe))], 1))
    return np.concatenate(parts)


def circulant(n, k):
    """Every vertex has the same degree 2k: all hubs, or none, fall into one degree bin."""
    v = np.arange(n)
    return np.concatenate([np.stack([v, (v + d) % n], 1) for d in range(1, k + 1)])


@functools.lru_cache(maxsize=None)
def graph(name, shuffled):
    edges = {
        "core-64": lambda: dense_core(64, 1.0),
        "core-300": lambda: dense_core(300, 0.9),
        "core-2500": lambda: dense_core(2500, 0.45),
        "ring-31000": lambda: circulant(31000, 64),   # one bin that fits: the ranks come from ids alone
        "ring-40000": lambda: circulant(40000, 64),   # one bin that does not fit: no hubs
        "ring-below": lambda: circulant(20000, 63),   # degree 126: below every hub's
    }[name]()
    fo, hd = csr(edges, shuffled=shuffled)
    from oracle import oracle as O
    O.build()
    total, pv, _ = O.count(fo, hd, method="merge", num_threads=8)
    return fo, hd, total, pv


@pytest.mark.parametrize("name", ["core-64", "core-300", "core-2500", "ring-31000", "ring-40000", "ring-below"])
@pytest.mark.parametrize("conf", [Config(), Config(small_outdegree=4, medium_outdegree=32, segment=64),
                                  Config(small_outdegree=48, tile_order=1), Config(collect_stats=True)],
                         ids=["default", "small4", "cost", "stats"])
@pytest.mark.parametrize("shuffled", [False, True])
def test_hub_lists(counter, name, conf, shuffled):
    fo, hd, total, pv = graph(name, shuffled)
    t, p = counter.count(fo, hd, conf)
    assert t == total and np.array_equal(p, pv)
    t, p = counter.count_dag(*oriented(fo, hd), conf)
    assert t == total and np.array_equal(p, pv)


def oriented(fo, hd):
    """Every edge at its smaller id: caller-oriented lists."""
    src = np.repeat(np.arange(N, dtype=np.uint32), np.diff(fo.astype(np.int64)))
    keep = src < hd
    out = np.zeros(N + 1, dtype=np.uint64)
    out[1:] = np.cumsum(np.bincount(src[keep], minlength=N))
    return out, hd[keep]


def test_budget_without_room_for_hub_lists():
    """A budget that holds the plain workspace but not the hub lists is still accepted."""
    fo, hd, total, pv = graph("core-300", False)
    plain = _native.load().ktri_workspace_bytes(N, len(hd), _native.METHOD_AUTO)
    with TriangleCounter(0, memory_budget=plain + 8 * (N + 2) + 4 * len(hd) + (1 << 20)) as c:
        t, p = c.count(fo, hd)
        assert t == total and np.array_equal(p, pv)
