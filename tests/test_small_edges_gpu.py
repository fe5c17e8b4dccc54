"""The small kernel (edges between out-degrees up to small_outdegree, counted at their tail) at
the sizes where its groups and tables change: tails of out-degree 0, 1 and 2, the bound and one
above it, groups cut by their key capacity (tails of 43 and more keys) and by their tail count
(more than 16 tails of two keys), graphs smaller than one vertex batch.  Exact against the oracle."""
import numpy as np
import pytest

from katric_gb300 import Config

pytestmark = pytest.mark.gpu


def cliques_and_fans(sizes, fans, seed):
    """Disjoint cliques K_s (out-degrees 0..s-1) and fans of `fans` triangles on one edge, ids permuted."""
    edges, n = [], 0
    for s in sizes:
        edges += [(n + i, n + j) for i in range(s) for j in range(i + 1, s)]
        n += s
    if fans:
        edges.append((n, n + 1))
        edges += [(n + c, n + 2 + i) for i in range(fans) for c in (0, 1)]
        n += 2 + fans
    e = np.random.default_rng(seed).permutation(n)[np.asarray(edges, dtype=np.int64).reshape(-1, 2)]
    src, dst = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    order = np.lexsort((dst, src))
    fo = np.zeros(n + 1, dtype=np.uint64)
    fo[1:] = np.cumsum(np.bincount(src, minlength=n))
    return fo, dst[order].astype(np.uint32)


@pytest.mark.parametrize("bound", [1, 2, 4, 5, 31, 47, 48, 0])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("shuffled", [False, True])
def test_tails_at_the_bounds(counter, oracle, bound, wide, shuffled):
    for sizes, fans in [((3,), 0), ((2, 3, 4, 5, 6), 40), (tuple(range(1, 53)), 100)]:
        fo, hd = cliques_and_fans(sizes, fans, seed=len(sizes))
        if shuffled:
            rng = np.random.default_rng(1)
            for a, b in zip(fo[:-1].astype(int), fo[1:].astype(int)):
                rng.shuffle(hd[a:b])
        total, pv, _ = oracle.count(fo, hd, method="merge", num_threads=4)
        t, p = counter.count(fo, hd, Config(small_outdegree=bound, force_wide_offsets=wide))
        assert t == total and np.array_equal(p, pv)
