"""The multifrontal factor over the range of double precision: materials scaled
by 1e-170 and 1e160 (squares of the matrix entries leave the range) give the
unscaled solution over the scale.  Both solves refine to a true residual of
1e-12 and these systems have a condition number below 2e3: 4e-9 between them."""
import numpy as np
import pytest

from emagddm_b200 import _abi, fetidp, mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-170, 1e-150, 1e150, 1e160])
@pytest.mark.parametrize("n", [3, 9])
def test_direct_solve_of_a_scaled_system(n, scale):
    m = mesh.perturbed(mesh.plain_small(n), 0.2, n)
    ds = fetidp.DirectSolver(m)
    b = np.random.default_rng(n).normal(size=ds.n_dofs)
    x = []
    for s in (1.0, scale, scale, scale):  # the eager, the captured and the replayed factorization
        assert ds.factor(nu=m.nu * s) == 0, _abi.lib().emg_last_error()
        y, rc, out = ds.solve(b, tol=1e-12)
        assert rc == 0 and out.residual_norm <= 1e-12, (rc, out.residual_norm)
        x.append(y * s)
    for y in x[1:]:
        assert np.linalg.norm(y - x[0]) <= 4e-9 * np.linalg.norm(x[0])
