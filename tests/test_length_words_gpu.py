"""Out-lists of 2^16 and more entries on graphs whose lists are split (needs a GB300).  Their length
word keeps 16 bits for each part, which is enough where no list holds a neighbour twice: a longer
list is refused as one with duplicates, also where the part's length would wrap to almost nothing."""
import numpy as np
import pytest

from katric_gb300 import KtriError, TriangleCounter

pytestmark = pytest.mark.gpu


def repeated_pair(k):
    """Vertex 0 lists 1 and 2 in turn, k entries; both order above it, and a star of another centre
    puts the graph above the size line of split lists."""
    side, star = k + 10, 1 << 20
    n = 4 + 2 * side + star
    lists = [np.resize(np.array([1, 2]), k), np.concatenate([[0], np.arange(4, 4 + side)]),
             np.concatenate([[0], np.arange(4 + side, 4 + 2 * side)]), np.arange(4 + 2 * side, n)]
    leaves = np.repeat([1, 2, 3], [side, side, star])
    fo = np.concatenate([[0], np.cumsum([len(x) for x in lists])])
    fo = np.concatenate([fo, fo[-1] + np.arange(1, len(leaves) + 1)])
    return fo.astype(np.uint64), np.concatenate(lists + [leaves]).astype(np.uint32)


@pytest.mark.parametrize("k", [65535, 65536, 65537, 65538, 65600, 131072])
def test_lists_past_the_length_word(counter, k):
    fo, hd = repeated_pair(k)
    assert len(hd) >= 1 << 21
    with pytest.raises(KtriError, match="duplicate"):
        counter.count(fo, hd)


def test_list_longer_than_any_vertex_count():
    """A list of 2^30 entries and more has none but repeated neighbours: refused before orientation."""
    torch = pytest.importorskip("torch")
    d = (1 << 30) + 1000
    if torch.cuda.mem_get_info()[0] < 24 << 30:
        pytest.skip("needs 24 GiB of device memory")
    fo = torch.tensor([0, d, d + 1, d + 2], dtype=torch.int64, device="cuda")
    head = torch.zeros(d + 2, dtype=torch.int32, device="cuda")
    head[0:d:2] = 1
    head[1:d:2] = 2
    total = torch.zeros(1, dtype=torch.int64, device="cuda")
    with TriangleCounter(0) as ctr:
        ctr.count_device(fo.data_ptr(), head.data_ptr(), 3, d + 2, total.data_ptr())
        with pytest.raises(KtriError, match="duplicate"):
            ctr.check()
    del head
    torch.cuda.empty_cache()
