"""ILU0 solves after one with a NaN right-hand side: the triangular solves read
nothing that an earlier solve left behind, also in a level wider than the values
kept on the SM, so the next solve of the same matrix is as good as the first
(ILU(0) of these matrices is their exact LU; condition numbers below 10)."""
import numpy as np
import pytest

from emagddm_b200 import _abi
from tests.helpers import HostCsr, solve
from tests.test_gpu_ilu0_sweeps import CASES, build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["diagonal", "chain 600", "arrow 50", "old value"])
def test_good_solve_after_a_nan_right_hand_side(name):
    n, pairs = CASES[name]
    rp, col, val = build(n, pairs)
    A = HostCsr(rp, col, val)
    b = np.random.default_rng(n).standard_normal(n)
    bad = np.full(n, np.nan)
    _, out = solve(A.h, bad, "cg", tol=1e-12, max_iter=3, precond=_abi.PRECOND_ILU0)
    assert not out.residual_norm < 1e-12
    x, out = solve(A.h, b, "cg", tol=1e-12, max_iter=50, precond=_abi.PRECOND_ILU0)
    assert out.status == 0 and out.iterations <= 2, (out.status, out.iterations)
    r = b.copy()
    np.subtract.at(r, np.repeat(np.arange(n), np.diff(rp)), val * x[col])
    assert np.linalg.norm(r) <= 1e-11 * np.linalg.norm(b)
