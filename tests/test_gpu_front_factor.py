"""Panel Cholesky and front solves of the direct solver at the edges of their
tiles: fronts from 18 unknowns (one narrow panel) through widths that end
inside a 16-column sub-panel to fronts of several 64-column panels, against a
dense solve of the oracle's matrix.  The solver refines to a true residual of
1e-12 and these one-material systems have a condition number below 2e3, so the
solutions agree to 2e-9."""
import numpy as np
import pytest

from emagddm_b200 import _abi, fetidp, mesh
from tests.helpers import oracle_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 3, 4, 5, 6, 7, 8, 9])
def test_direct_solve_at_panel_edges(n):
    m = mesh.perturbed(mesh.plain_small(n), 0.2, n)
    ds = fetidp.DirectSolver(m)
    rp, col, kv, _, _ = oracle_system(m, ds.l2g)
    size = rp.size - 1
    K = np.zeros((size, size))
    K[np.repeat(np.arange(size), np.diff(rp)), col] = kv
    b = np.random.default_rng(n).normal(size=size)
    for _ in range(3):  # the eager, the captured and the replayed factorization
        assert ds.factor() == 0, _abi.lib().emg_last_error()
        x, rc, out = ds.solve(b, tol=1e-12)
        assert rc == 0 and out.residual_norm <= 1e-12
        want = np.linalg.solve(K, b)
        assert np.linalg.norm(x - want) <= 2e-9 * np.linalg.norm(want)
