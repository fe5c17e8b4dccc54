"""Sorting lists at the bound of what a block sorts in shared memory, 8192 entries (needs a GB300): the
contraction of lists in any order, some of them longer than that, gives every list sorted."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [[8191, 5], [8192, 33, 32], [8193], [8192, 8193, 1], [20_000] * 70, [3, 40_000, 8193]],
                         ids=lambda x: f"{len(x)}x{max(x)}")
@pytest.mark.parametrize("ascending", [False, True])
def test_contracted_lists_are_sorted(counter, lengths, ascending):
    rng = np.random.default_rng(len(lengths))
    local, ghosts = len(lengths), 50_000
    lists = [local + rng.permutation(ghosts)[:k] for k in lengths]
    if ascending:
        lists = [np.sort(x) for x in lists]
    fo = np.zeros(local + ghosts + 1, dtype=np.uint64)
    fo[1:local + 1] = np.cumsum(lengths)
    fo[local + 1:] = fo[local]
    kept, out_fo, out = counter.contract_dag(fo, np.concatenate(lists).astype(np.uint32), local)
    assert kept.tolist() == list(range(local)) and np.array_equal(out_fo, fo[:local + 1])
    assert np.array_equal(out, np.concatenate([np.sort(x) for x in lists]))
