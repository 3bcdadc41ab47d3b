"""emg_spmv through the slots' own columns: one row, partial slices, empty rows
and columns, a matrix first used by a solver, and x and y in one array, against
NumPy (at most 40 terms a row: 40 roundings of 1e-14 at most)."""
import ctypes as C

import numpy as np
import pytest

from emagddm_b200 import _abi
from tests.helpers import HostCsr, lib, solve

pytestmark = pytest.mark.gpu


def random_csr(n, seed, empty=False):
    rng = np.random.default_rng(seed)
    rows, cols = [], []
    for i in range(n):
        k = 0 if empty and i % 3 else int(rng.integers(1, min(n, 40) + 1))
        c = np.sort(rng.choice(n, k, replace=False))
        rows.append(np.full(k, i))
        cols.append(c)
    rows, cols = np.concatenate(rows), np.concatenate(cols)
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    return rp, cols.astype(np.int32), rng.standard_normal(cols.size)


@pytest.mark.parametrize("n", [1, 31, 32, 33, 257, 4095, 4097])
@pytest.mark.parametrize("empty", [False, True])
@pytest.mark.parametrize("alias", [False, True])
def test_product(n, empty, alias):
    import torch
    rp, col, val = random_csr(n, n, empty)
    A = HostCsr(rp, col, val)
    x = np.random.default_rng(1).standard_normal(n)
    want = np.zeros(n)
    np.add.at(want, np.repeat(np.arange(n), np.diff(rp)), val * x[col])
    xd = torch.tensor(x, device="cuda")
    yd = xd if alias else torch.full_like(xd, np.nan)
    _abi.check(lib().emg_spmv(A.h, C.c_void_p(xd.data_ptr()), C.c_void_p(yd.data_ptr()), None), "emg_spmv")
    torch.cuda.synchronize()
    assert np.abs(yd.cpu().numpy() - want).max() <= 1e-14 * max(np.abs(want).max(), 1.0) * 40


def test_product_after_a_solve():
    import torch
    n = 500
    i = np.arange(n)
    rp = np.arange(n + 1, dtype=np.int32)
    A = HostCsr(rp, i.astype(np.int32), 2.0 + i)
    b = np.ones(n)
    x, out = solve(A.h, b, "cg", tol=1e-12, precond=1)
    assert out.status == 0
    xd = torch.tensor(x, device="cuda")
    yd = torch.empty_like(xd)
    _abi.check(lib().emg_spmv(A.h, C.c_void_p(xd.data_ptr()), C.c_void_p(yd.data_ptr()), None), "emg_spmv")
    torch.cuda.synchronize()
    assert np.abs(yd.cpu().numpy() - b).max() <= 1e-12
