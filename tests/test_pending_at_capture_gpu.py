"""A device call captured while the context's previous call, on another stream, is unread (needs a
GB300): what is captured runs later, so the unread call is ended from the host first, and both results
are their own graph's."""
import numpy as np
import pytest
import torch

from katric_gb300 import Graph, TriangleCounter

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [12, 17])  # without and with split lists
def test_unread_call_when_capture_starts(oracle, scale):
    graphs = [Graph.rmat(scale, 16, seed=71), Graph.rmat(18, 16, seed=72)]
    want = [oracle.count(g.first_out, g.head, num_threads=8)[:2] for g in graphs]
    dev = [(torch.from_numpy(g.first_out.view(np.int64).copy()).cuda(),
            torch.from_numpy(g.head.view(np.int32).copy()).cuda(),
            torch.zeros(1, dtype=torch.int64, device="cuda"), torch.zeros(g.n, dtype=torch.int64, device="cuda"))
           for g in graphs]
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with TriangleCounter(0) as ctr:
        def count(i, stream):
            fo, hd, t, p = dev[i]
            ctr.count_device(fo.data_ptr(), hd.data_ptr(), graphs[i].n, graphs[i].nnz, t.data_ptr(), p.data_ptr(),
                             stream=stream.cuda_stream)

        def check(i):
            torch.cuda.synchronize()
            assert int(dev[i][2][0]) == want[i][0]
            assert np.array_equal(dev[i][3].cpu().numpy().view(np.uint64), want[i][1])
            dev[i][2].zero_()
            dev[i][3].zero_()
            torch.cuda.synchronize()

        count(1, other)
        ctr.check()
        check(1)
        count(1, other)  # unread when the capture starts
        captured = torch.cuda.CUDAGraph()
        with torch.cuda.graph(captured, stream=side, capture_error_mode="relaxed"):
            count(0, side)
        captured.replay()
        check(0)
        check(1)
        count(1, other)
        check(1)
        captured.replay()
        check(0)
