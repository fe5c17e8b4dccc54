"""The device memory a server holds while its batches may split their out-lists (needs a GB300): the
larger workspaces of all slots stay within the budget, and one that an earlier batch left makes room
when graphs are kept resident, without evicting any."""
import numpy as np
import pytest

from katric_gb300 import Graph, Server, TriangleCounter, _native

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

SLACK = 32 << 20  # allocation granularity and the runtime's own


@pytest.fixture(scope="module")
def big():
    g = Graph.rmat(17, 250, seed=5)  # its count takes longer than the packing of the next batch
    with TriangleCounter(0) as ctr:
        return g, ctr.count(g.first_out, g.head)


def used_by(run):
    """Device bytes in use where run() read the free memory, above those in use before it."""
    warm = Graph.rmat(16, 24, seed=1)
    with Server(slots=1, max_batch_nnz=1 << 16) as srv:  # modules and local memory are set up
        srv.wait(srv.submit(warm))
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    return before - run()


def sizes(g):
    """Grown sizes of a slot's union, of its plain workspace, and of what split lists add to that."""
    union = 8 * (g.n + 1) + 4 * (g.nnz + 1) + 8 * (g.n + 1) + 5 * 4096
    plain = int(_native.load().ktri_workspace_bytes(g.n, g.nnz, 0))
    split = int(2.4 * g.nnz + 18 * g.n)
    return union + union // 4, plain + plain // 8, split + split // 8


def test_two_slots_share_the_budget(big):
    g, (total, pv) = big
    union, plain, split = sizes(g)
    budget = 2 * (union + plain) + split + split // 4  # split lists in one slot, not in both

    def run():
        with Server(slots=2, memory_budget=budget, max_batch_nnz=1 << 16) as srv:
            for _ in range(3):
                for i in [srv.submit(g, borrow=True) for _ in range(4)]:
                    t, p = srv.wait(i)[:2]
                    assert t == total and np.array_equal(p, pv)
            assert srv.stats()["peak_inflight_batches"] == 2
            return torch.cuda.mem_get_info()[0]

    assert used_by(run) <= budget + SLACK


def test_resident_graphs_take_the_room_of_split_lists(big):
    g, (total, pv) = big
    union, plain, split = sizes(g)
    budget = union + plain + split + (64 << 20)
    kept = [Graph.gnm(100_000, 1_900_000, seed=s) for s in range(12)]  # 17 MB each
    with TriangleCounter(0) as ctr:
        want = [ctr.count(k.first_out, k.head)[0] for k in kept]

    def run():
        with Server(slots=1, memory_budget=budget, max_batch_nnz=1 << 16) as srv:
            t, p = srv.wait(srv.submit(g))[:2]
            assert t == total and np.array_equal(p, pv)
            for i, k in enumerate(kept):
                assert srv.wait(srv.submit(k, key=1 + i))[0] == want[i]
            st = srv.stats()
            assert st["evictions"] == 0 and st["resident_graphs"] == len(kept)
            free = torch.cuda.mem_get_info()[0]
            assert srv.wait(srv.submit(g))[0] == total
            return free

    assert used_by(run) <= budget + SLACK
