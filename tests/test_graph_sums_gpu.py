"""Totals of a batch are a third of the per-vertex counts of each range, rounded down, by one block per
range and by several (needs a GB300): also where the ranges cut graphs, so that the sums need not be
multiples of three."""
import numpy as np
import pytest

from katric_gb300 import Batch, Graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5000, 40_000, 600_000])  # one block, a few, the most per range
@pytest.mark.parametrize("ranges", [1, 2, 7, 60])
def test_ranges_that_cut_the_graph(counter, n, ranges):
    g = Graph.rgg2d(n, 20.0, seed=ranges)
    cuts = np.sort(np.random.default_rng(n + ranges).integers(0, n + 1, ranges - 1))
    first = np.concatenate([[0], cuts, [n]]).astype(np.uint64)
    for _ in range(3):
        totals, pv = counter.count_batch(Batch(g, first))
        want = [int(pv[int(a):int(b)].sum()) // 3 for a, b in zip(first[:-1], first[1:])]
        assert totals.tolist() == want
