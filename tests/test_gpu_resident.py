"""CG and BiCGSTAB of small matrices (one persistent kernel a solve) at the
edges of its blocks: one row, a partial slice, the last row counts of each
block shape (148 SMs: 256, 512, 1024 threads, two rows a thread) and the first
one past them, and a row too long for the shared-memory stage.  The matrices
are diagonally dominant with a condition number below 4, so a residual of
1e-10 leaves each solution within 4e-10 of the exact one."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.helpers import HostCsr, solve

pytestmark = pytest.mark.gpu


def tridiagonal(n):
    i = np.arange(n)
    rows = np.concatenate([i[1:], i, i[:-1]])
    cols = np.concatenate([i[:-1], i, i[1:]])
    vals = np.concatenate([np.full(n - 1, -1.0), 4.0 + (i % 7) * 0.1, np.full(n - 1, -1.0)])
    return csr(n, rows, cols, vals)


def arrow(n):
    """Row and column 0 full, the rest diagonal."""
    i = np.arange(1, n)
    z = np.zeros(n - 1, np.int64)
    rows = np.concatenate([[0], z, i, i])
    cols = np.concatenate([[0], i, z, i])
    off = np.full(n - 1, 0.5 / np.sqrt(n))
    return csr(n, rows, cols, np.concatenate([[2.0], off, off, np.full(n - 1, 1.0)]))


def csr(n, rows, cols, vals):
    order = np.lexsort((cols, rows))
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(np.bincount(rows, minlength=n))
    return rp, cols[order].astype(np.int32), vals[order]


@pytest.mark.parametrize("kind,precond", [("cg", 0), ("cg", 1), ("bicgstab", 0)])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 257, 37888, 37889, 75777, 151553, 303104, 303105])
def test_resident_solves_at_block_edges(kind, precond, n):
    rp, col, val = tridiagonal(n)
    check(rp, col, val, kind, precond)


@pytest.mark.parametrize("kind", ["cg", "bicgstab"])
def test_row_longer_than_the_stage(kind):
    check(*arrow(3001), kind, 1 if kind == "cg" else 0)


def check(rp, col, val, kind, precond):
    n = rp.size - 1
    b = np.random.default_rng(n).standard_normal(n)
    A = HostCsr(rp.astype(np.int32), col, val)
    x, out = solve(A.h, b, kind, tol=1e-10, max_iter=200, precond=precond)
    xo, st, it, _ = (O.pcg if kind == "cg" else O.bicgstab)(rp, col, val, b, tol=1e-10, max_iter=200, precond=precond)
    assert out.status == st == 0
    assert abs(out.iterations - it) <= 2
    assert np.linalg.norm(b - O.spmv(rp, col, val, x)) <= 1.1e-10 * np.linalg.norm(b)
    assert np.linalg.norm(x - xo) <= 8e-10 * np.linalg.norm(xo)
