"""The warp-per-tile kernel at the sizes where its tables and units change: owners one above the small
bound, at and above the keys of one table chunk (192), lists of 4, 5, 32 and 33 entries, segments
of one and of many tiles, and keys that crowd one bucket.  Exact against the oracle."""
import numpy as np
import pytest

from katric_gb300 import Config

pytestmark = pytest.mark.gpu


def csr(edges, n, perm_seed, shuffled):
    e = np.asarray(edges, dtype=np.int64)
    if perm_seed is not None:
        e = np.random.default_rng(perm_seed).permutation(n)[e]
    src, dst = np.concatenate([e[:, 0], e[:, 1]]), np.concatenate([e[:, 1], e[:, 0]])
    order = np.lexsort((np.random.default_rng(3).random(len(dst)) if shuffled else dst, src))
    fo = np.zeros(n + 1, dtype=np.uint64)
    fo[1:] = np.cumsum(np.bincount(src, minlength=n))
    return fo, dst[order].astype(np.uint32)


def cliques(sizes):
    edges, n = [], 0
    for s in sizes:
        i, j = np.triu_indices(s, 1)
        edges.append(np.stack([i + n, j + n], 1))
        n += s
    return np.concatenate(edges), n


def crowded():
    """A clique of 256 whose ids share the top bits of their hash (id * 0x9E3779B1 mod 2^32): one run of
    buckets overflows again and again."""
    ids = np.arange(1 << 21, dtype=np.uint64)
    close = ids[((ids * np.uint64(0x9E3779B1)) & np.uint64(0xFFFFFFFF)) < np.uint64(1 << 21)]
    assert len(close) >= 256
    i, j = np.triu_indices(256, 1)
    return np.stack([close[i], close[j]], 1), 1 << 21


@pytest.mark.parametrize("name", ["bounds", "chunks", "units", "crowded"])
@pytest.mark.parametrize("conf", [Config(), Config(small_outdegree=1, segment=64), Config(force_wide_offsets=True),
                                  Config(small_outdegree=3, medium_outdegree=256, tile_order=1)],
                         ids=["default", "small1", "wide", "cost"])
@pytest.mark.parametrize("shuffled", [False, True])
def test_owner_tiles(counter, oracle, name, conf, shuffled):
    edges, n = {
        "bounds": lambda: cliques([49, 50, 51, 52, 60]),
        "chunks": lambda: cliques([192, 193, 194, 195, 257]),
        "units": lambda: cliques([5, 6, 33, 34, 35, 65, 66, 130]),
        "crowded": crowded,
    }[name]()
    fo, hd = csr(edges, n, None if name == "crowded" else 5, shuffled)
    total, pv, _ = oracle.count(fo, hd, method="merge", num_threads=4)
    t, p = counter.count(fo, hd, conf)
    assert t == total and np.array_equal(p, pv)
