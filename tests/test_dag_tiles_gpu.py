"""Symmetrisation of oriented lists by tiles of entries (needs a GB300).

A warp takes 128 entries whatever lists they are of and finds their owners in windows of 32 lists.
Covered here: totals around a tile, lists longer than many tiles, more than 32 lists in a row of 32
entries' window, long runs of empty lists between two entries, and offsets that do not start at 0 in
the caller's buffer.  The bar is the oracle's count of the undirected graph."""
import numpy as np
import pytest

from katric_gb300 import KtriError

pytestmark = pytest.mark.gpu


def lists_of(n, edges):
    """Out-lists (a, b) in order of a, and the undirected CSR of the same edges."""
    e = np.array(sorted(edges), dtype=np.int64).reshape(-1, 2)
    fo = np.zeros(n + 1, dtype=np.uint64)
    fo[1:] = np.cumsum(np.bincount(e[:, 0], minlength=n))
    both = np.concatenate([e, e[:, ::-1]])
    both = both[np.lexsort((both[:, 1], both[:, 0]))]
    ufo = np.zeros(n + 1, dtype=np.uint64)
    ufo[1:] = np.cumsum(np.bincount(both[:, 0], minlength=n))
    return fo, e[:, 1].astype(np.uint32), ufo, both[:, 1].astype(np.uint32)


def shape(name):
    if name == "star-out":  # one list of many tiles, the others empty but for a path
        return 5000, [(0, v) for v in range(1, 5000)] + [(v, v + 1) for v in range(1, 4000, 2)]
    if name == "star-in":  # every entry names one vertex
        return 5000, [(v, 4999) for v in range(4999)] + [(v, v + 1) for v in range(0, 4000, 2)]
    if name == "empty-runs":  # entries thousands of empty lists apart
        at = np.arange(0, 200_000, 4999)
        return 200_000, [(int(a), int(b)) for i, a in enumerate(at) for b in at[i + 1:i + 4]]
    if name == "two-lists":  # both long, one at either end of the ids
        return 3000, [(0, v) for v in range(1, 2999)] + [(2999, v) for v in range(1, 2999)] + [(0, 2999)]
    k = int(name)  # a fan of k edges and its chords
    return k + 2, [(0, v) for v in range(1, k // 2 + 1)] + [(v, v + 1) for v in range(1, k - k // 2 + 1)]


SHAPES = ["1", "2", "31", "33", "127", "128", "129", "257", "star-out", "star-in", "empty-runs", "two-lists"]


@pytest.mark.parametrize("name", SHAPES)
def test_entries_find_their_lists(counter, oracle, name):
    n, edges = shape(name)
    fo, hd, ufo, uhd = lists_of(n, edges)
    total, pv, _ = oracle.count(ufo, uhd, num_threads=4)
    t, p = counter.count_dag(fo, hd)
    assert t == total
    assert np.array_equal(p, pv)


def test_offsets_into_a_larger_buffer_and_descending_offsets(counter, oracle):
    torch = pytest.importorskip("torch")
    n, edges = shape("129")
    fo, hd, ufo, uhd = lists_of(n, edges)
    total = oracle.count(ufo, uhd, num_threads=4)[0]
    buf = torch.from_numpy(np.concatenate([np.full(7, 5, np.int32), hd.view(np.int32)])).cuda()
    tot = torch.zeros(1, dtype=torch.int64, device="cuda")
    shifted = torch.from_numpy((fo + np.uint64(7)).view(np.int64)).cuda()
    counter.count_dag_device(shifted.data_ptr(), buf.data_ptr(), n, len(hd), tot.data_ptr(), None)
    counter.check()
    assert int(tot.item()) == total
    bad = fo.copy()
    bad[2], bad[3] = bad[3], bad[2]
    assert (np.diff(bad.view(np.int64)) < 0).any()
    offsets = torch.from_numpy(bad.view(np.int64)).cuda()
    counter.count_dag_device(offsets.data_ptr(), buf[7:].contiguous().data_ptr(), n, len(hd), tot.data_ptr(), None)
    with pytest.raises(KtriError):
        counter.check()
