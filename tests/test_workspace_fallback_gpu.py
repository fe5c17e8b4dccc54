"""Counts that could split their out-lists but have no room for the larger workspace (needs a GB300): an
allocation that fails although the device reports the memory as free, and a call captured on a
context whose workspace only holds the plain lists.  Both are counted with plain lists."""
import glob
import os
import subprocess
import sys
import textwrap

import numpy as np
import pytest

from katric_gb300 import Graph, TriangleCounter, _native, build

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# cudaMalloc that refuses what is larger than a limit
WRAP = """
#include <cuda_runtime_api.h>
size_t test_limit = ~(size_t)0;
unsigned test_refused;
cudaError_t __real_cudaMalloc(void**, size_t);
cudaError_t __wrap_cudaMalloc(void** p, size_t bytes) {
    if (bytes <= test_limit) return __real_cudaMalloc(p, bytes);
    ++test_refused;
    return cudaErrorMemoryAllocation;
}
"""

# counts by every entry point of a context, with the limit between the plain and the larger workspace
CHILD = """
import ctypes, sys
import numpy as np, torch
from katric_gb300 import Batch, Config, Graph, TriangleCounter, _native
lib = ctypes.CDLL(sys.argv[1])
for name, (res, args) in _native.SIGNATURES.items():
    getattr(lib, name).restype, getattr(lib, name).argtypes = res, args
_native._lib = lib
limit, refused = ctypes.c_size_t.in_dll(lib, "test_limit"), ctypes.c_uint.in_dll(lib, "test_refused")
g = Graph.rmat(16, 24, seed=9)
src = np.repeat(np.arange(g.n, dtype=np.uint32), np.diff(g.first_out.astype(np.int64)))
up = src < g.head
dag_fo = np.zeros(g.n + 1, np.uint64)
dag_fo[1:] = np.cumsum(np.bincount(src[up], minlength=g.n))
dag_hd = g.head[up]
dev = [torch.from_numpy(x.view(t).copy()).cuda() for x, t in
       ((g.first_out, np.int64), (g.head, np.int32), (dag_fo, np.int64), (dag_hd, np.int32))]
gf = torch.tensor([0, g.n], dtype=torch.int64, device="cuda")
total = torch.zeros(1, dtype=torch.int64, device="cuda")
pv = torch.zeros(g.n, dtype=torch.int64, device="cuda")
p = [x.data_ptr() for x in dev]
one = Batch(g, np.array([0, g.n], np.uint64))
calls = {
    "device": lambda c: c.count_device(p[0], p[1], g.n, g.nnz, total.data_ptr(), pv.data_ptr()),
    "dag_device": lambda c: c.count_dag_device(p[2], p[3], g.n, len(dag_hd), total.data_ptr(), pv.data_ptr()),
    "batch_device": lambda c: c.count_batch_device(p[0], p[1], g.n, g.nnz, gf.data_ptr(), 1, total.data_ptr(),
                                                   pv.data_ptr()),
    "host": lambda c: c.count(g.first_out, g.head),
    "dag_host": lambda c: c.count_dag(dag_fo, dag_hd),
    "batch_host": lambda c: c.count_batch(one),
}
def answer(c, name):
    total.zero_()
    pv.zero_()
    r = calls[name](c)
    c.check()
    t, v = (int(total[0]), pv.cpu().numpy().view(np.uint64)) if r is None else (int(np.ravel(r[0])[0]), r[1])
    return t, v.copy()
with TriangleCounter(0) as c:
    want = answer(c, "device")
for name in calls:
    plain = int(lib.ktri_workspace_bytes(g.n, g.nnz, 0)) + (8 * g.n + 4 * g.nnz if "host" in name or "dag" in name else 0)
    if name == "dag_host":
        plain += 8 * g.n + 4 * len(dag_hd)
    limit.value = plain + 2 * g.nnz  # the larger lists take 2.4 bytes per entry and more
    with TriangleCounter(0) as c:
        for repeat in range(3):
            t, v = answer(c, name)
            assert t == want[0] and np.array_equal(v, want[1]), name
            assert refused.value == 2, (name, refused.value)  # with and without headroom, once
    refused.value, limit.value = 0, 2 ** 64 - 1
print("counted")
"""


def test_allocation_that_fails(tmp_path):
    built = glob.glob(os.path.join(build.BUILD, "*.o"))
    build.build(force=len(built) != len(build.sources()))
    wrap = tmp_path / "wrap.c"
    wrap.write_text(textwrap.dedent(WRAP))
    lib = tmp_path / "libktri_wrapped.so"
    objects = sorted(glob.glob(os.path.join(build.BUILD, "*.o")))
    assert len(objects) == len(build.sources())
    subprocess.run([build.nvcc(), "-shared", "-o", str(lib), str(wrap), *objects, *build.ARCH, "-Xcompiler",
                    "-fPIC,-fopenmp", "-Xlinker", "--wrap=cudaMalloc", "-lgomp"], check=True, capture_output=True)
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(CHILD), str(lib)], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "counted" in r.stdout, r.stdout + r.stderr


def test_capture_grows_no_workspace(oracle):
    import torch
    g = Graph.rmat(16, 24, seed=9)
    total, pv, _ = oracle.count(g.first_out, g.head, num_threads=8)
    fo = torch.from_numpy(g.first_out.view(np.int64).copy()).cuda()
    hd = torch.from_numpy(g.head.view(np.int32).copy()).cuda()
    t = torch.zeros(1, dtype=torch.int64, device="cuda")
    p = torch.zeros(g.n, dtype=torch.int64, device="cuda")
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    with TriangleCounter(0) as ctr:
        def count():
            ctr.count_device(fo.data_ptr(), hd.data_ptr(), g.n, g.nnz, t.data_ptr(), p.data_ptr(),
                             stream=side.cuda_stream)

        ctr.set_memory_budget(int(_native.load().ktri_workspace_bytes(g.n, g.nnz, 0)) + 4096)  # plain lists only
        count()
        ctr.check()
        ctr.set_memory_budget(0)
        captured = torch.cuda.CUDAGraph()
        with torch.cuda.graph(captured, stream=side):
            count()
        for _ in range(2):
            t.zero_()
            p.zero_()
            captured.replay()
            torch.cuda.synchronize()
            assert int(t[0]) == total and np.array_equal(p.cpu().numpy().view(np.uint64), pv)
