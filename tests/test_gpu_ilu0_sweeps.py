"""Triangular solves of the ILU0 preconditioner where their layout can go
wrong: a chain (one row a level), one level of all rows, rows longer than the
entries held in registers, and a dependency older than the values kept on the
SM, against dense solves.  ILU(0) of these matrices (no fill outside the
pattern) is their exact LU, so CG takes one or two iterations; condition numbers
are below 10 and the tolerance is 1e-12, so solutions agree to 1e-10."""
import numpy as np
import pytest

from emagddm_b200 import _abi
from tests.helpers import HostCsr, solve

pytestmark = pytest.mark.gpu


def build(n, pairs):
    """Symmetric, unit diagonally dominant, off-diagonal -1 / (2 degree)."""
    a = np.array(pairs, np.int64).reshape(-1, 2)
    deg = np.bincount(a.reshape(-1), minlength=n).max() if a.size else 1
    i = np.arange(n)
    rows = np.concatenate([i, a[:, 0], a[:, 1]])
    cols = np.concatenate([i, a[:, 1], a[:, 0]])
    vals = np.concatenate([np.ones(n), np.full(2 * len(a), -0.45 / max(deg, 1))])
    order = np.lexsort((cols, rows))
    rp = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    return rp.astype(np.int32), cols[order].astype(np.int32), vals[order]


CASES = {
    "diagonal": (100, []),                                            # one level
    "chain 1": (1, []),
    "chain 33": (33, [(k, k + 1) for k in range(32)]),                # a row a level
    "chain 600": (600, [(k, k + 1) for k in range(599)]),
    # the last row depends on all others (an arrow: no fill)
    "arrow 50": (50, [(k, 49) for k in range(49)]),
    # rows of the second level need values of a first level wider than the ring
    # (the chain behind them only adds levels)
    "old value": (14050, [(k, 13000 + k % 1000) for k in range(13000)] + [(k, k + 1) for k in range(13999, 14049)]),
    "long chain": (7000, [(k, k + 1) for k in range(6999)]),
}


@pytest.mark.parametrize("name", list(CASES))
def test_sweeps_solve_exactly(name):
    n, pairs = CASES[name]
    rp, col, val = build(n, pairs)
    A = HostCsr(rp, col, val)
    b = np.random.default_rng(n).standard_normal(n)
    x, out = solve(A.h, b, "cg", tol=1e-12, max_iter=50, precond=_abi.PRECOND_ILU0)
    assert out.status == 0 and out.iterations <= 2, (out.status, out.iterations)
    r = b.copy()
    np.subtract.at(r, np.repeat(np.arange(n), np.diff(rp)), val * x[col])
    assert np.linalg.norm(r) <= 1e-11 * np.linalg.norm(b)
