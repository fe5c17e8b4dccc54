"""Offsets of oriented lists that do not hold the number of entries that the call names (needs a GB300):
refused, whatever the lists hold, and without a read outside [first_out[0], first_out[n]).  The lists
lie inside a larger buffer, so that the entries around them are there."""
import numpy as np
import pytest

from katric_gb300 import KtriError

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N, M = 300, 299  # a path and the chords of its first vertex


def lists():
    deg = np.ones(N, dtype=np.int64)
    deg[0], deg[N - 1] = 2, 0
    fo = np.concatenate([[0], np.cumsum(deg)])
    hd = np.concatenate([[1, 2], np.arange(2, N)])
    assert fo[-1] == len(hd) == M + 1
    return fo, hd.astype(np.int32)


@pytest.mark.parametrize("start,entries", [(0, M), (0, M + 2), (0, 2 * (M + 1)), (0, (M + 1) // 2), (1, M), (1, M + 2), (7, 0),
                                           (200, 1)])
def test_offsets_that_hold_another_number(counter, start, entries):
    fo, hd = lists()
    buffer = torch.from_numpy(np.concatenate([np.full(start, 3, np.int32), hd, np.full(2 * M + 400, 5, np.int32)])).cuda()
    offsets = torch.from_numpy(fo + start).cuda()
    total = torch.zeros(1, dtype=torch.int64, device="cuda")
    counter.count_dag_device(offsets.data_ptr(), buffer.data_ptr(), N, entries, total.data_ptr(), None)
    with pytest.raises(KtriError):
        counter.check()
    counter.count_dag_device(offsets.data_ptr(), buffer.data_ptr(), N, len(hd), total.data_ptr(), None)
    counter.check()
    assert int(total[0]) == 1


def test_last_offset_names_the_end_of_the_buffer(counter):
    """First offset above 0, last offset equal to the number of entries named: shorter lists by as much."""
    fo, hd = lists()
    buffer = torch.from_numpy(np.concatenate([hd, np.full(64, 5, np.int32)])).cuda()
    short = fo.copy()
    short[0] = 1
    offsets = torch.from_numpy(short).cuda()
    total = torch.zeros(1, dtype=torch.int64, device="cuda")
    counter.count_dag_device(offsets.data_ptr(), buffer.data_ptr(), N, len(hd), total.data_ptr(), None)
    with pytest.raises(KtriError):
        counter.check()
