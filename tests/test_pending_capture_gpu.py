"""A device call captured into a CUDA graph on a context whose previous call was checked, replayed, and
followed by ordinary calls on other streams (needs a GB300): each result is its own graph's."""
import numpy as np
import pytest
import torch

from katric_gb300 import Graph, TriangleCounter

pytestmark = pytest.mark.gpu


def on_device(g):
    return (torch.from_numpy(g.first_out.view(np.int64).copy()).cuda(),
            torch.from_numpy(g.head.view(np.int32).copy()).cuda(),
            torch.zeros(1, dtype=torch.int64, device="cuda"), torch.zeros(g.n, dtype=torch.int64, device="cuda"))


@pytest.mark.parametrize("scale", [12, 17])  # without and with hub lists
def test_captured_call_between_ordinary_ones(oracle, scale):
    graphs = [Graph.rmat(scale, 16, seed=61), Graph.gnm(5000, 40000, seed=62)]
    want = [oracle.count(g.first_out, g.head, num_threads=8)[:2] for g in graphs]
    dev = [on_device(g) for g in graphs]
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with TriangleCounter(0) as ctr:
        def count(i, stream):
            g, (fo, hd, t, p) = graphs[i], dev[i]
            ctr.count_device(fo.data_ptr(), hd.data_ptr(), g.n, g.nnz, t.data_ptr(), p.data_ptr(),
                             stream=stream.cuda_stream)

        def check(i):
            torch.cuda.synchronize()
            assert int(dev[i][2][0]) == want[i][0]
            assert np.array_equal(dev[i][3].cpu().numpy().view(np.uint64), want[i][1])
            dev[i][2].zero_()
            dev[i][3].zero_()
            torch.cuda.synchronize()

        count(0, side)  # the workspace grows outside the capture
        ctr.check()
        check(0)
        captured = torch.cuda.CUDAGraph()
        with torch.cuda.graph(captured, stream=side):
            count(0, side)
        for _ in range(2):
            captured.replay()
            check(0)
        count(1, other)
        count(1, side)
        check(1)
        captured.replay()
        check(0)
