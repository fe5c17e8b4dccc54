"""Lists that hold a neighbour twice, far apart (needs a GB300).  Such lists do not ascend, so the
counting tables are the only check: the repeat is reported whatever the list's length, on each side
of the bounds at which another kernel or another chunk of the table takes it, with whole and with
split lists, in adjacency lists and in oriented ones."""
import functools

import numpy as np
import pytest

from katric_gb300 import Config, KtriError

pytestmark = pytest.mark.gpu


def csr(lists):
    fo = np.concatenate([[0], np.cumsum([len(x) for x in lists])])
    return fo.astype(np.uint64), np.concatenate(lists).astype(np.uint32)


def fan(k, repeat):
    """Vertex 0 lists 1..k, `repeat` of them twice more than k entries apart where possible; the
    others order above it by their leaves."""
    leaves = 1 + k + np.arange(k * (k + 3)).reshape(k, k + 3)
    first = np.concatenate([np.arange(1, k + 1), np.arange(1, repeat + 1)])
    middle = [np.concatenate([[0], leaves[i], [0] if i < repeat else []]) for i in range(k)]
    return csr([first] + middle + [np.array([1 + i // (k + 3)]) for i in range(k * (k + 3))])


LENGTHS = [2, 3, 46, 47, 48, 49, 100, 190, 191, 192, 193, 254, 255, 256, 257, 300, 600]


@pytest.mark.parametrize("k", LENGTHS)
@pytest.mark.parametrize("wide", [False, True])
def test_repeat_in_an_adjacency_list(counter, k, wide):
    conf = Config(force_wide_offsets=wide)
    fo, hd = fan(k, 0)
    assert counter.count(fo, hd, conf)[0] == 0
    with pytest.raises(KtriError, match="duplicate"):
        counter.count(*fan(k, 1), conf)


@pytest.mark.parametrize("k", LENGTHS)
def test_edge_listed_at_both_ends(counter, k):
    """Oriented lists: vertex 0 lists 1..k, and k lists 0 again."""
    lists = [np.arange(1, k + 1)] + [k + 1 + (k + 3) * i + np.arange(k + 3) for i in range(k)]
    lists += [np.zeros(0, np.int64)] * (k * (k + 3))
    assert counter.count_dag(*csr(lists))[0] == 0
    lists[k] = np.concatenate([lists[k], [0]])
    with pytest.raises(KtriError, match="duplicate"):
        counter.count_dag(*csr(lists))


RING, HALF = 33000, 300  # more vertices of one degree than there are hub indices: none of them is a hub


@functools.lru_cache(maxsize=None)
def ring_rows():
    return (np.arange(RING)[:, None] + np.concatenate([np.arange(1, HALF + 1), -np.arange(1, HALF + 1)])) % RING


def split_lists(k, at, hubs):
    """A ring lattice, the centre of a star, and an owner x that lists k vertices, the one at at[0] again
    at at[1]: k ring vertices, or with hubs so many vertices of still higher degree."""
    rows = ring_rows()
    x, centre, leaf = RING, RING + 1, RING + 2
    many = 1500
    named = RING + 2 + many + np.arange(k) if hubs else RING - k + np.arange(k)
    n = RING + 2 + many + (k if hubs else 0)
    mine = named.copy()
    mine[at[1]] = mine[at[0]]
    leaves = np.arange(leaf, leaf + many)
    lists = [rows[:RING - k].ravel(), np.concatenate([rows[RING - k:], np.full((k, 1), x)], 1).ravel() if not hubs
             else rows[RING - k:].ravel(), mine, leaves]
    degree = [np.full(RING - k, 2 * HALF), np.full(k, 2 * HALF + (0 if hubs else 1)), [k], [many]]
    if hubs:  # every leaf lists the centre and all of the named vertices
        lists += [np.concatenate([np.full((many, 1), centre), np.tile(named, (many, 1))], 1).ravel(),
                  np.concatenate([np.full((k, 1), x), np.tile(leaves, (k, 1))], 1).ravel()]
        degree += [np.full(many, k + 1), np.full(k, many + 1)]
    else:
        lists += [np.full(many, centre)]
        degree += [np.full(many, 1)]
    fo = np.concatenate([[0], np.cumsum(np.concatenate(degree))])
    assert len(fo) == n + 1
    return fo.astype(np.uint64), np.concatenate(lists).astype(np.uint32)


@pytest.mark.parametrize("hubs", [False, True], ids=["others", "hubs"])
@pytest.mark.parametrize("k,at", [(40, (0, 39)), (49, (0, 48)), (192, (0, 191)), (193, (0, 192)), (250, (100, 240)),
                                  (257, (0, 256)), (400, (10, 390)), (599, (250, 598))])
def test_repeat_in_a_split_list(counter, k, at, hubs):
    fo, hd = split_lists(k, (at[0], at[0]), hubs)
    assert len(hd) >= 1 << 21
    counter.count(fo, hd, per_vertex=False)
    with pytest.raises(KtriError, match="duplicate"):
        counter.count(*split_lists(k, at, hubs), per_vertex=False)
