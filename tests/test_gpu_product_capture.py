"""emg_spmv under stream capture on a matrix that a solver has used: the product
allocates nothing, so the captured graph can be replayed, and products outside
it stand on their own after the graph is gone."""
import ctypes as C

import numpy as np
import pytest

from emagddm_b200 import _abi
from tests.helpers import HostCsr, lib, solve

pytestmark = pytest.mark.gpu


def test_captured_product_after_a_solve():
    import torch
    n = 5000
    i = np.arange(n)
    rows = np.concatenate([i[1:], i, i[:-1]])
    cols = np.concatenate([i[:-1], i, i[1:]])
    vals = np.concatenate([np.full(n - 1, -1.0), 4.0 + i % 7, np.full(n - 1, -1.0)])
    order = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    A = HostCsr(rp, cols[order], vals[order])
    _, out = solve(A.h, np.ones(n), "cg", tol=1e-10, precond=1)
    assert out.status == 0

    def want(x):
        y = (4.0 + i % 7) * x
        y[1:] -= x[:-1]
        y[:-1] -= x[1:]
        return y

    def product(x, y):
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        _abi.check(lib().emg_spmv(A.h, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), stream), "emg_spmv")

    xd = torch.zeros(n, dtype=torch.float64, device="cuda")
    yd = torch.zeros_like(xd)
    for _ in range(2):  # a second capture after the first graph is gone
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            product(xd, yd)
        for seed in range(2):
            x = np.random.default_rng(seed).standard_normal(n)
            xd.copy_(torch.from_numpy(x))
            yd.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert np.abs(yd.cpu().numpy() - want(x)).max() <= 1e-13 * 100
        graph.reset()
        del graph
        torch.cuda.empty_cache()
        x = np.random.default_rng(7).standard_normal(n)
        xd.copy_(torch.from_numpy(x))
        product(xd, yd)
        torch.cuda.synchronize()
        assert np.abs(yd.cpu().numpy() - want(x)).max() <= 1e-13 * 100


def test_first_use_under_capture_is_refused_and_leaves_nothing():
    """A matrix that nothing has used yet allocates: refused while the stream is
    captured, without ending the capture, and good afterwards."""
    import torch
    n = 1000
    i = np.arange(n, dtype=np.int32)
    A = HostCsr(np.arange(n + 1, dtype=np.int32), i, 2.0 + i)
    x = torch.ones(n, dtype=torch.float64, device="cuda")
    y = torch.zeros_like(x)
    z = torch.zeros_like(x)
    rc = []
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        rc.append(lib().emg_spmv(A.h, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), stream))
        z.add_(1.0)
    assert rc[0] == _abi.EMG_ERR_CUDA and b"captured" in lib().emg_last_error()
    graph.replay()
    torch.cuda.synchronize()
    assert (z == 1.0).all() and (y == 0.0).all()
    del graph
    _abi.check(lib().emg_spmv(A.h, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), None), "emg_spmv")
    torch.cuda.synchronize()
    assert np.array_equal(y.cpu().numpy(), 2.0 + i)
    b, out = solve(A.h, np.ones(n), "cg", tol=1e-10, precond=1)
    assert out.status == 0
