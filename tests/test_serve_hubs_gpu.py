"""Served batches that split their out-lists (needs a GB300).

A batch of at least 2^21 entries with vertices of high degree counts by hub lists where the server's
memory budget has room for their workspace, and by plain lists where it only has room for those.
Both give the oracle's counts, and a budget without room for either is refused as before."""
import numpy as np
import pytest

from katric_gb300 import Graph, KtriError, Server, _native

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def served(oracle):
    g = Graph.rmat(16, 24, seed=31)
    assert g.nnz >= 1 << 21
    return g, oracle.count(g.first_out, g.head, num_threads=8)[:2]


def plain_bytes(g):
    union = 8 * (g.n + 1) + 4 * (g.nnz + 1) + 8 * (g.n + 1) + 5 * 4096
    return union + int(_native.load().ktri_workspace_bytes(g.n, g.nnz, 0))


@pytest.mark.parametrize("room", ["both", "plain", "none"])
def test_budget_decides_the_lists(served, room):
    g, (total, pv) = served
    budget = {"both": 4 << 30, "plain": plain_bytes(g), "none": plain_bytes(g) // 2}[room]
    with Server(slots=1, memory_budget=budget, max_batch_nnz=1 << 14) as srv:
        for _ in range(2):
            i = srv.submit(g)
            if room == "none":
                with pytest.raises(KtriError):
                    srv.wait(i)
                continue
            t, p = srv.wait(i)[:2]
            assert t == total
            assert np.array_equal(p, pv)
