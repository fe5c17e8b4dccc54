"""Both kinds of owner tiles in one array, one from its front and one from its back, and both orders
in one pass (needs a GB300): graphs below and above the size from which tiles are ordered, all
large, nearly all medium, and both; lists with and without hubs.  Exact against the oracle."""
import numpy as np
import pytest

from katric_gb300 import Config, Graph

pytestmark = pytest.mark.gpu

GRAPHS = {"unordered": lambda: Graph.rmat(14, 24, seed=41),   # below 2^20 entries
          "ordered": lambda: Graph.rmat(15, 24, seed=42),     # above, still without hubs
          "hubs": lambda: Graph.rmat(16, 24, seed=43)}        # above 2^21 entries


@pytest.fixture(scope="module")
def counted(oracle):
    kept = {}

    def get(name):
        if name not in kept:
            g = GRAPHS[name]()
            kept[name] = g, oracle.count(g.first_out, g.head, num_threads=8)[:2]
        return kept[name]
    return get


@pytest.mark.parametrize("name", list(GRAPHS))
@pytest.mark.parametrize("small,medium", [(0, 0), (1, 64), (1, 1), (4, 256), (48, 48)])
@pytest.mark.parametrize("order,segment", [(0, 0), (1, 0), (0, 64), (1, 1024)])
def test_both_kinds_of_tiles(counter, counted, name, small, medium, order, segment):
    g, (total, pv) = counted(name)
    assert (g.nnz >= 1 << 20) == (name != "unordered") and (g.nnz >= 1 << 21) == (name == "hubs")
    conf = Config(small_outdegree=small, medium_outdegree=medium, tile_order=order, segment=segment)
    t, p = counter.count(g.first_out, g.head, conf)
    assert t == total
    assert np.array_equal(p, pv)
