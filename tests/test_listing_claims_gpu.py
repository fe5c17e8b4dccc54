"""Triangle listing on vertex counts around one claim of the listing kernel, 32 vertices, and around one
for every warp of the device (needs a GB300): each triangle once, none left out."""
import numpy as np
import pytest

from katric_gb300 import Graph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 31, 32, 33, 63, 64, 65, 1000, 300_000, 311_297])
def test_listing(counter, n):
    g = Graph.gnm(n, min(n * (n - 1) // 2, 4 * n), seed=n)
    total, pv = counter.count(g.first_out, g.head)
    rows = counter.list_triangles(g.first_out, g.head)
    assert len(rows) == total
    if total:
        assert (rows[:, 0] < rows[:, 1]).all() and (rows[:, 1] < rows[:, 2]).all()
        assert len(np.unique(rows, axis=0)) == total
        assert np.array_equal(np.bincount(rows.ravel(), minlength=n).astype(np.uint64), pv)
