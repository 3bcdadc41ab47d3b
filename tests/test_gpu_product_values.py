"""emg_spmv with infinities and NaN in x: they reach the rows that hold an entry
in their column and no other row, whatever padding the rows have."""
import ctypes as C

import numpy as np
import pytest

from emagddm_b200 import _abi
from tests.helpers import HostCsr, lib
from tests.test_gpu_product import random_csr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 257, 4097])
@pytest.mark.parametrize("empty", [False, True])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_product_keeps_infinities_and_nan_to_their_rows(n, empty, value):
    import torch
    rp, col, val = random_csr(n, n, empty)
    A = HostCsr(rp, col, val)
    rows = np.repeat(np.arange(n), np.diff(rp))
    for j in (0, 1, n // 2, n - 1):
        x = np.random.default_rng(1).standard_normal(n)
        x[j] = value
        hit = np.zeros(n, bool)
        hit[rows[col == j]] = True
        want = np.zeros(n)
        keep = col != j
        np.add.at(want, rows[keep], val[keep] * x[col[keep]])
        xd = torch.tensor(x, device="cuda")
        yd = torch.zeros_like(xd)
        _abi.check(lib().emg_spmv(A.h, C.c_void_p(xd.data_ptr()), C.c_void_p(yd.data_ptr()), None), "emg_spmv")
        torch.cuda.synchronize()
        y = yd.cpu().numpy()
        assert not np.isfinite(y[hit]).any()
        assert np.abs(y - want)[~hit].max(initial=0.0) <= 4e-13 * max(np.abs(want).max(), 1.0)
