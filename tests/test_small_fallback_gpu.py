"""Tails whose table cannot be built (needs a GB300).  The small kernel gives a tail of d keys 3 d buckets
of two and starts over with another multiplier where a bucket overflows, 16 times; the entries of a
tail that fails every time are compared one by one.  Random lists of 48 entries get there about once
in 10^5, so the neighbours are chosen for it here: ids, hub indices, ascending lists and others."""
import functools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

D, TRIES = 48, 16


def overfull(keys, mult):
    """Some bucket gets more than two of the keys (rows of keys): floor(key * mult mod 2^32 * 3 d / 2^32)."""
    h = ((keys.astype(np.uint64) * np.uint64(mult)) & np.uint64(0xFFFFFFFF)) * np.uint64(3 * D) >> np.uint64(32)
    h = np.sort(h, axis=1)
    return (h[:, 2:] == h[:, :-2]).any(axis=1)


@functools.lru_cache(maxsize=None)
def stubborn(first, count, sets, seed):
    """Sets of D numbers below count, which as keys first + number overflow a bucket under all multipliers."""
    rng, found = np.random.default_rng(seed), []
    while len(found) < sets:
        pick = rng.integers(0, count, (50000, D))
        mult = 0x9E3779B1
        for _ in range(TRIES):
            pick = pick[overfull(first + pick, mult)]
            mult = (mult * 0x2C1B3C6D + 2) & 0xFFFFFFFF
        found += [np.sort(p) for p in pick if len(np.unique(p)) == D]
    return found[:sets]


def csr(n, edges, shuffled):
    e = np.unique(np.sort(edges, axis=1), axis=0)
    src, dst = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    order = np.lexsort((np.random.default_rng(2).random(len(dst)) if shuffled else dst, src))
    fo = np.zeros(n + 1, dtype=np.uint64)
    fo[1:] = np.cumsum(np.bincount(src, minlength=n))
    return fo, dst[order].astype(np.uint32)


CORE, TAILS = 3000, 40


def graph(hubs, shuffled):
    """Core vertices that all get the same degree by leaves of their own, a sparse random graph between
    them, and tails: four with each stubborn set of core vertices for neighbours, beside ordinary ones.
    With hubs the core vertices are the hubs, the one of the highest id first."""
    degree = 700 if hubs else 150
    n = CORE + TAILS + CORE * degree
    sets = [CORE - 1 - s for s in stubborn(n, CORE, 3, 11)] if hubs else stubborn(0, CORE, 3, 11)
    rng = np.random.default_rng(4)
    parts = [rng.integers(0, CORE, (40000, 2))]
    for t in range(TAILS):
        mine = sets[t // 4] if t < 4 * len(sets) else rng.permutation(CORE)[:rng.integers(2, D + 1)]
        parts.append(np.stack([np.full(len(mine), CORE + t), mine], 1))
        parts.append(np.stack([mine[:-1], mine[1:]], 1))  # so that tails have triangles
    e = np.unique(np.sort(np.concatenate(parts), axis=1), axis=0)
    e = e[e[:, 0] != e[:, 1]]
    leaves = degree - np.bincount(e.ravel(), minlength=CORE)[:CORE]
    assert leaves.min() > 0
    leaf = CORE + TAILS + np.arange(leaves.sum())
    return csr(n, np.concatenate([e, np.stack([np.repeat(np.arange(CORE), leaves), leaf], 1)]), shuffled)


@pytest.mark.parametrize("hubs", [False, True])
@pytest.mark.parametrize("shuffled", [False, True])
def test_tails_without_a_table(counter, oracle, hubs, shuffled):
    fo, hd = graph(hubs, shuffled)
    assert (len(hd) >= 1 << 21) == hubs
    degree = np.diff(fo.astype(np.int64))
    assert (degree[:CORE] == (700 if hubs else 150)).all() and (degree[CORE:] <= D).all()
    total, pv, _ = oracle.count(fo, hd, method="merge", num_threads=4)
    t, p = counter.count(fo, hd)
    assert t == total and np.array_equal(p, pv)
