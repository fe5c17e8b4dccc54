"""Calls after an unread device call that start nothing on the context's workspace (needs a GB300): a
graph without vertices, and a call that is refused for its size.  The unread call still ends before
the next one takes the workspace, and its status is not read from a workspace that is gone."""
import numpy as np
import pytest
import torch

from katric_gb300 import Graph, KtriError, TriangleCounter

pytestmark = pytest.mark.gpu


def on_device(g):
    return (torch.from_numpy(g.first_out.view(np.int64).copy()).cuda(),
            torch.from_numpy(g.head.view(np.int32).copy()).cuda(),
            torch.zeros(1, dtype=torch.int64, device="cuda"), torch.zeros(g.n, dtype=torch.int64, device="cuda"))


@pytest.fixture(scope="module")
def graphs(oracle):
    made = [Graph.rmat(18, 16, seed=1), Graph.gnm(3000, 20000, seed=2), Graph.rgg2d(50000, 24.0, seed=4)]
    return [(g, oracle.count(g.first_out, g.head, method="merge", num_threads=8)[:2]) for g in made]


@pytest.mark.parametrize("empty", ["csr", "dag", "batch"])
def test_empty_call_between_two_counts(graphs, empty):
    streams = [torch.cuda.Stream() for _ in range(3)]
    dev = [on_device(g) for g, _ in graphs]
    nothing = torch.ones(4, dtype=torch.int64, device="cuda")
    with TriangleCounter(0) as ctr:
        def count(i, stream):
            fo, hd, t, p = dev[i]
            ctr.count_device(fo.data_ptr(), hd.data_ptr(), graphs[i][0].n, graphs[i][0].nnz, t.data_ptr(), p.data_ptr(),
                             stream=stream)

        for i in range(3):
            count(i, 0)
            ctr.check()
        for _ in range(3):
            torch.cuda.synchronize()
            count(0, streams[0].cuda_stream)
            st = streams[1].cuda_stream
            if empty == "csr":
                ctr.count_device(0, 0, 0, 0, nothing.data_ptr(), stream=st)
            elif empty == "dag":
                ctr.count_dag_device(0, 0, 0, 0, nothing.data_ptr(), stream=st)
            else:
                ctr.count_batch_device(0, 0, 0, 0, nothing.data_ptr(), 1, nothing.data_ptr(), stream=st)
            count(1, streams[2].cuda_stream)
            host = ctr.count(graphs[2][0].first_out, graphs[2][0].head)
            torch.cuda.synchronize()
            assert int(nothing[0]) == 0
            for i in range(2):
                total, pv = graphs[i][1]
                assert int(dev[i][2][0]) == total
                assert np.array_equal(dev[i][3].cpu().numpy().view(np.uint64), pv)
                dev[i][3].zero_()
            assert host[0] == graphs[2][1][0] and np.array_equal(host[1], graphs[2][1][1])


def test_refused_size_after_an_unread_call(graphs):
    (g, (total, pv)), (fo, hd, t, p) = graphs[1], on_device(graphs[1][0])
    torch.cuda.synchronize()
    with TriangleCounter(0) as ctr:
        ctr.count_device(fo.data_ptr(), hd.data_ptr(), g.n, g.nnz, t.data_ptr(), p.data_ptr())
        with pytest.raises(KtriError):  # a workspace of terabytes
            ctr.count_device(fo.data_ptr(), hd.data_ptr(), g.n, 1 << 41, t.data_ptr(), p.data_ptr())
        ctr.check()
        assert int(t[0]) == total and np.array_equal(p.cpu().numpy().view(np.uint64), pv)
        ctr.count_device(fo.data_ptr(), hd.data_ptr(), g.n, g.nnz, t.data_ptr(), p.data_ptr())
        ctr.check()
        assert int(t[0]) == total
