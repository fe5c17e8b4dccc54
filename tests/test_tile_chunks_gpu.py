"""Owners at the bounds of a table chunk of the warp-per-tile kernel, 256 keys (needs a GB300): one and
two chunks of whole lists, and one to three of the part of split lists that holds no hubs.  Exact
against the oracle."""
import numpy as np
import pytest

from katric_gb300 import Config

pytestmark = pytest.mark.gpu


def csr(n, edges, shuffled):
    src, dst = np.concatenate([edges[:, 0], edges[:, 1]]), np.concatenate([edges[:, 1], edges[:, 0]])
    order = np.lexsort((np.random.default_rng(3).random(len(dst)) if shuffled else dst, src))
    fo = np.zeros(n + 1, dtype=np.uint64)
    fo[1:] = np.cumsum(np.bincount(src, minlength=n))
    return fo, dst[order].astype(np.uint32)


@pytest.mark.parametrize("shuffled", [False, True])
def test_whole_lists(counter, oracle, shuffled):
    edges, n = [], 0
    for s in (254, 255, 256, 257, 258, 259):  # out-degrees up to s - 1
        i, j = np.triu_indices(s, 1)
        edges.append(np.stack([i + n, j + n], 1))
        n += s
    fo, hd = csr(n, np.random.default_rng(5).permutation(n)[np.concatenate(edges)], shuffled)
    total, pv, _ = oracle.count(fo, hd, method="merge", num_threads=4)
    for conf in (Config(), Config(force_wide_offsets=True), Config(small_outdegree=8, segment=64)):
        t, p = counter.count(fo, hd, conf)
        assert t == total and np.array_equal(p, pv)


@pytest.mark.parametrize("half", [128, 256, 258])
def test_split_lists(counter, oracle, half):
    """A ring lattice of more vertices than there are hub indices, all of one degree, beside a clique of
    hubs: the ring's lists hold half to 2 half entries, none of them a hub."""
    ring, clique = 33000, 900
    v = np.arange(ring)
    i, j = np.triu_indices(clique, 1)
    edges = np.concatenate([np.stack([v, (v + d) % ring], 1) for d in range(1, half + 1)] +
                           [np.stack([i + ring, j + ring], 1)])
    fo, hd = csr(ring + clique, edges, False)
    total, pv, _ = oracle.count(fo, hd, method="merge", num_threads=8)
    t, p = counter.count(fo, hd)
    assert t == total and np.array_equal(p, pv)
