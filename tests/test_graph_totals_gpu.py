"""Totals of a batch's graphs when several blocks share a graph (needs a GB300).

Up to 64 blocks share one graph, each with at least 4096 vertices if one graph had them all; their
sums need not be multiples of three.  Covered here: one graph, few graphs of very different sizes
(some without vertices or edges), and more graphs than blocks."""
import numpy as np
import pytest

from katric_gb300 import Batch, Graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[16384], [16385], [4096, 0, 70_000, 3, 0, 8191], [300_000, 100],
                                   [600_000], [64] * 1500], ids=lambda s: f"{len(s)}x{max(s)}")
def test_totals_of_few_and_many_graphs(counter, oracle, sizes):
    graphs = [Graph.gnm(n, 5 * n, seed=i) if n > 16 else Graph(np.zeros(n + 1, np.uint64), np.zeros(0, np.uint32))
              for i, n in enumerate(sizes)]
    totals, per_vertex = counter.count_batch(Batch.pack(graphs))
    at = 0
    for i, g in enumerate(graphs):
        want = oracle.count(g.first_out, g.head, num_threads=4)[:2] if g.nnz else (0, np.zeros(g.n, np.uint64))
        assert int(totals[i]) == want[0]
        assert np.array_equal(per_vertex[at:at + g.n], want[1])
        at += g.n
