"""Pieces of lists at the edges of the orientation's tiles and rows (needs a GB300).

A tile holds 256 diagonals in rows of 32 slots.  Circulant graphs give every list the same length,
so the lists' ends fall on every slot of a row and of a tile: lists shorter than a row, of one or
several rows, of a tile, and of several tiles (a tile without a vertex end holds 256 slots).  The
out-lists must equal the oracle's, and an entry repeated anywhere in a list that spans tiles is
reported, also where the two copies lie in two tiles."""
import numpy as np
import pytest

from katric_gb300 import KtriError

pytestmark = pytest.mark.gpu


def circulant(n, degree):
    offsets = np.concatenate([np.arange(1, degree // 2 + 1), -np.arange(1, degree // 2 + 1)])
    head = np.sort((np.arange(n)[:, None] + offsets[None, :]) % n, axis=1).astype(np.uint32)
    return np.arange(n + 1, dtype=np.uint64) * degree, head.reshape(-1)


@pytest.mark.parametrize("degree", [2, 30, 32, 62, 64, 254, 256, 300, 512, 766])
def test_lists_of_every_length(counter, oracle, degree):
    fo, hd = circulant(1543, degree)
    ofo, oh = counter.orient(fo, hd)
    efo, eh = oracle.oriented_csr(fo, hd)
    assert np.array_equal(ofo, efo)
    assert np.array_equal(oh, eh)
    total, pv = counter.count(fo, hd)
    expect, epv, _ = oracle.count(fo, hd, num_threads=4)
    assert total == expect
    assert np.array_equal(pv, epv)


@pytest.mark.parametrize("degree", [64, 300])
def test_a_repeated_entry_is_reported_at_every_slot(counter, degree):
    fo, hd = circulant(601, degree)
    v = 300
    for k in range(int(fo[v]), int(fo[v + 1]) - 1):
        bad = hd.copy()
        bad[k + 1] = bad[k]
        with pytest.raises(KtriError):
            counter.count(fo, bad)
    counter.count(fo, hd)
