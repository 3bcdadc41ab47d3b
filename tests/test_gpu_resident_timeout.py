"""The bounded waits of the resident CG and BiCGSTAB at every poll limit: whatever
limit makes some of the blocks give up and at whichever reduction, a solve
either reports EMG_ERR_TIMEOUT or has the solution, and the next solve with the
limit restored is good."""
import numpy as np
import pytest

from emagddm_b200 import _abi
from oracle import oracle as O
from tests.helpers import HostCsr, lib, solve
from tests.test_gpu_resident import tridiagonal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["cg", "bicgstab"])
@pytest.mark.parametrize("n", [500, 20000])
def test_a_solve_times_out_or_is_right(kind, n):
    rp, col, val = tridiagonal(n)
    b = np.random.default_rng(n).standard_normal(n)
    A = HostCsr(rp.astype(np.int32), col, val)

    def check(x, out):
        assert out.status == 0
        assert np.linalg.norm(b - O.spmv(rp, col, val, x)) <= 1.1e-10 * np.linalg.norm(b)

    seen = set()
    try:
        for spins in [0, 1, 2, 3, 4, 5, 6, 7, 8, 10, 12, 14, 16, 20, 24, 32, 48, 64, 128, 1024]:
            _abi.check(lib().emg_test_set_barrier_spins(spins), "emg_test_set_barrier_spins")
            for _ in range(5):
                x, out = solve(A.h, b, kind, tol=1e-10, max_iter=200, precond=0)
                seen.add(out.status)
                if out.status != _abi.EMG_ERR_TIMEOUT:
                    check(x, out)
    finally:
        _abi.check(lib().emg_test_set_barrier_spins(-1), "emg_test_set_barrier_spins")
    assert _abi.EMG_ERR_TIMEOUT in seen
    check(*solve(A.h, b, kind, tol=1e-10, max_iter=200, precond=0))
