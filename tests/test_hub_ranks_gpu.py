"""The order of the hubs (needs a GB300): bins of degrees that hold one vertex, about as many (4096)
as make a bin crowded and as many as there are hub indices, sorted chunks that several bins share,
ids that ascend and descend with the degree.  The work counters depend on the exact (degree, id) order."""
import numpy as np
import pytest

from katric_gb300 import Config

pytestmark = pytest.mark.gpu


def ring(n, half, extra):
    """A ring lattice of n vertices; vertex v also gets extra[v] pendant neighbours."""
    v = np.arange(n)
    leaf = n + np.arange(extra.sum())
    edges = np.concatenate([np.stack([v, (v + d) % n], 1) for d in range(1, half + 1)] +
                           [np.stack([np.repeat(v, extra), leaf], 1)])
    return n + len(leaf), edges


SHAPES = {
    "one-bin": lambda: ring(32767, 64, np.zeros(32767, int)),
    "1024": lambda: ring(1024, 70, np.full(1024, 1000)),
    "4095": lambda: ring(4095, 70, np.full(4095, 100)),
    "4096": lambda: ring(4096, 70, np.full(4096, 100)),
    "4097": lambda: ring(4097, 70, np.full(4097, 100)),
    "crowded-and-not": lambda: ring(12000, 70, np.where(np.arange(12000) % 5, 100, 300 + np.arange(12000) // 100)),
    "two-degrees": lambda: ring(30000, 64, np.arange(30000) % 2),
    "ascending": lambda: ring(20000, 64, np.arange(20000) // 4500),
    "descending": lambda: ring(20000, 64, np.arange(20000)[::-1] // 4500),
    "wide-bins": lambda: ring(6000, 64, np.random.default_rng(1).integers(300, 1200, 6000)),
}


@pytest.mark.parametrize("name", list(SHAPES))
@pytest.mark.parametrize("permuted", [False, True])
def test_order_of_the_hubs(counter, oracle, name, permuted):
    n, e = SHAPES[name]()
    n = max(n, (1 << 21) - len(e) * 2 + n)
    if permuted:
        e = np.random.default_rng(7).permutation(n)[e]
    if 2 * len(e) < 1 << 21:  # above the size line of split lists: a star of one more vertex
        fill = (1 << 20) - len(e)
        e = np.concatenate([e, np.stack([np.full(fill, n), n + 1 + np.arange(fill)], 1)])
        n += 1 + fill
    src, dst = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    order = np.lexsort((dst, src))
    fo = np.zeros(n + 1, dtype=np.uint64)
    fo[1:] = np.cumsum(np.bincount(src, minlength=n))
    hd = dst[order].astype(np.uint32)
    assert len(hd) >= 1 << 21
    total, pv, _ = oracle.count(fo, hd, method="merge", num_threads=8)
    t, p = counter.count(fo, hd, Config(collect_stats=True))
    assert t == total and np.array_equal(p, pv)
    st = counter.stats()
    degree = np.diff(fo.astype(np.int64))
    up = (degree[src] < degree[dst]) | ((degree[src] == degree[dst]) & (src < dst))
    out = np.bincount(src[up], minlength=n)
    assert st.oriented_edges == len(e)
    assert st.wedge_checks == int(out[dst[up]].sum())
    assert st.intersection_size_local == int(out[dst[up]].sum() + out[src[up]].sum())
