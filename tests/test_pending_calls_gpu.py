"""Device calls that follow one another on a context without a status check in between, on one
stream and on several: each call's counts are its own graph's (the calls share the workspace)."""
import numpy as np
import pytest
import torch

from katric_gb300 import Graph, TriangleCounter

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("streams", [1, 2, 3])
def test_unchecked_calls_in_a_row(oracle, streams):
    graphs = [Graph.rmat(16, 16, seed=1), Graph.gnm(3000, 20000, seed=2), Graph.rmat(18, 12, seed=3),
              Graph.rgg2d(50000, 24.0, seed=4)]
    want = [oracle.count(g.first_out, g.head, method="merge", num_threads=8)[:2] for g in graphs]
    dev = [(torch.from_numpy(g.first_out.view(np.int64).copy()).cuda(),
            torch.from_numpy(g.head.view(np.int32).copy()).cuda()) for g in graphs]
    out = [(torch.zeros(1, dtype=torch.int64, device="cuda"), torch.zeros(g.n, dtype=torch.int64, device="cuda"))
           for g in graphs]
    torch.cuda.synchronize()
    side = [torch.cuda.Stream() for _ in range(streams)]
    with TriangleCounter(0) as ctr:
        for repeat in range(3):
            for i, g in enumerate(graphs):
                st = side[i % streams]
                ctr.count_device(dev[i][0].data_ptr(), dev[i][1].data_ptr(), g.n, g.nnz, out[i][0].data_ptr(),
                                 out[i][1].data_ptr(), stream=st.cuda_stream)
        ctr.check()
        torch.cuda.synchronize()
        for (total, pv), (t, p) in zip(want, out):
            assert int(t[0]) == total and np.array_equal(p.cpu().numpy().view(np.uint64), pv)
