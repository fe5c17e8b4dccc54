"""Unchecked device calls on streams that share a handle (needs a GB300): cudaStreamPerThread names
another stream in every thread, and a destroyed stream's handle may be handed out again.  The calls
share the context's workspace, so each result is its own graph's only if they run one after the other."""
import ctypes
import threading

import numpy as np
import pytest
import torch

from katric_gb300 import Graph, TriangleCounter

pytestmark = pytest.mark.gpu

PER_THREAD = 2  # cudaStreamPerThread


@pytest.fixture(scope="module")
def graphs(oracle):
    made = [Graph.rmat(18, 16, seed=1), Graph.gnm(3000, 20000, seed=2), Graph.rgg2d(50000, 24.0, seed=4)]
    return [(g, torch.from_numpy(g.first_out.view(np.int64).copy()).cuda(),
             torch.from_numpy(g.head.view(np.int32).copy()).cuda(),
             oracle.count(g.first_out, g.head, method="merge", num_threads=8)[:2]) for g in made]


def outputs(graphs):
    out = [(torch.zeros(1, dtype=torch.int64, device="cuda"), torch.zeros(g.n, dtype=torch.int64, device="cuda"))
           for g, *_ in graphs]
    torch.cuda.synchronize()
    return out


def launch(ctr, graph, out, stream):
    g, fo, hd, _ = graph
    ctr.count_device(fo.data_ptr(), hd.data_ptr(), g.n, g.nnz, out[0].data_ptr(), out[1].data_ptr(), stream=stream)


def check(graphs, out):
    torch.cuda.synchronize()
    for (_, _, _, (total, pv)), (t, p) in zip(graphs, out):
        assert int(t[0]) == total and np.array_equal(p.cpu().numpy().view(np.uint64), pv)


def test_per_thread_stream_of_several_threads(graphs):
    with TriangleCounter(0) as ctr:
        for i in range(3):  # the workspace has its size, so no call waits for it to grow
            launch(ctr, graphs[i], outputs(graphs)[i], 0)
            ctr.check()
        for _ in range(3):
            out = outputs(graphs)
            for i in range(3):  # one thread after the other, as the context asks
                t = threading.Thread(target=launch, args=(ctr, graphs[i], out[i], PER_THREAD))
                t.start()
                t.join()
            ctr.check()
            check(graphs, out)


def test_streams_destroyed_while_their_call_runs(graphs):
    driver = ctypes.CDLL("libcuda.so.1")
    with TriangleCounter(0) as ctr:
        for i in range(3):
            launch(ctr, graphs[i], outputs(graphs)[i], 0)
            ctr.check()
        for _ in range(3):
            out = outputs(graphs)
            for i in range(3):
                stream = ctypes.c_void_p()
                assert driver.cuStreamCreate(ctypes.byref(stream), 1) == 0  # non-blocking
                launch(ctr, graphs[i], out[i], stream.value)
                assert driver.cuStreamDestroy_v2(stream) == 0
            ctr.check()
            check(graphs, out)
