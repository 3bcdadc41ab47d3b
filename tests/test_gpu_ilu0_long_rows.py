"""ILU0 solves of band matrices whose rows end at and past the entries that the
one-block triangular solves hold in registers (8 a row) and on both sides of the
row length where a launch per level takes over.  ILU(0) of a band is its exact
LU (fill stays inside the band), so CG takes one or two iterations; condition
numbers are below 10 and the tolerance is 1e-12."""
import numpy as np
import pytest

from emagddm_b200 import _abi
from tests.helpers import HostCsr, solve

pytestmark = pytest.mark.gpu


def band(n, w):
    rows = np.repeat(np.arange(n), 2 * w + 1)
    cols = rows + np.tile(np.arange(-w, w + 1), n)
    keep = (cols >= 0) & (cols < n)
    rows, cols = rows[keep], cols[keep]
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return rp.astype(np.int32), cols.astype(np.int32), np.where(rows == cols, 1.0, -0.4 / w)


@pytest.mark.parametrize("w", [1, 4, 5, 8, 9, 12, 13, 20, 24, 25, 28, 60])
def test_band_solves_exactly(w):
    n = 700
    rp, col, val = band(n, w)
    A = HostCsr(rp, col, val)
    b = np.random.default_rng(w).standard_normal(n)
    x, out = solve(A.h, b, "cg", tol=1e-12, max_iter=50, precond=_abi.PRECOND_ILU0)
    assert out.status == 0 and out.iterations <= 2, (out.status, out.iterations)
    r = b.copy()
    np.subtract.at(r, np.repeat(np.arange(n), np.diff(rp)), val * x[col])
    assert np.linalg.norm(r) <= 1e-11 * np.linalg.norm(b)
