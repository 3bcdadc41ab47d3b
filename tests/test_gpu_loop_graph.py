"""The loop graph of CG and BiCGSTAB, which matrices too large for one kernel a
solve run, at the sizes, values, statuses and failures of the small tests: those
tests again with the resident kernels switched off."""
import numpy as np
import pytest

from emagddm_b200 import _abi, mesh
from oracle import oracle as O
from tests import test_gpu_resident as resident
from tests.helpers import HostCsr, System, lib, oracle_system, solve
from tests.test_gpu_failures import (  # noqa: F401
    test_grid_barrier_wait_runs_out_with_timeout_status, test_nan_rhs_follows_reference_rules)
from tests.test_gpu_hex import test_hex_pcg_matches_oracle  # noqa: F401
from tests.test_gpu_krylov import (  # noqa: F401
    test_assembled_solve_matches_oracle, test_breakdown_reports_numerical_error, test_cg_tight_solution_within_1e8_of_oracle,
    test_config_plain_small_16_to_1e10, test_golden_reference_solves, test_history_records_every_iteration,
    test_unmerged_host_csr_is_summed, test_zero_rhs_and_iteration_limits)
from tests.test_gpu_prism_pyramid import test_pcg_matches_oracle  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def loop_graph():
    lib().emg_test_set_resident(0)
    yield
    lib().emg_test_set_resident(1)


@pytest.mark.parametrize("kind,precond", [("cg", 0), ("cg", 1), ("bicgstab", 0)])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 257, 8193, 37889])
def test_loop_graph_at_small_sizes(kind, precond, n):
    resident.check(*resident.tridiagonal(n), kind, precond)


@pytest.mark.parametrize("kind,precond", [("cg", 0), ("cg", 1), ("bicgstab", 0), ("bicgstab", 1)])
@pytest.mark.parametrize("n", [33, 8193])
@pytest.mark.parametrize("limit", [1, 2, 5])
@pytest.mark.parametrize("on", [0, 1])
def test_first_iterations_match_oracle(kind, precond, n, limit, on):
    """The iterates themselves, with and without the resident kernels (the
    reference's BiCGSTAB preconditions s alone and does not converge on these
    matrices with Jacobi, so its first iterations are what can be compared:
    at most 5 of them, sums of at most 8,193 terms, 1e-12 of the iterate times
    the growth of a few steps)."""
    lib().emg_test_set_resident(on)
    rp, col, val = resident.tridiagonal(n)
    b = np.random.default_rng(n).standard_normal(n)
    A = HostCsr(rp, col, val)
    x, out = solve(A.h, b, kind, tol=1e-14, max_iter=limit, precond=precond)
    xo, st, it, res = (O.pcg if kind == "cg" else O.bicgstab)(rp, col, val, b, tol=1e-14, max_iter=limit,
                                                              precond=precond)
    assert out.status == st == _abi.EMG_MAX_ITER_REACHED and out.iterations == it == limit
    assert abs(out.residual_norm - res) <= 1e-9 * res
    assert np.linalg.norm(x - xo) <= 1e-9 * np.linalg.norm(xo)


@pytest.mark.parametrize("kind,precond", [("cg", 0), ("cg", 1), ("bicgstab", 0), ("bicgstab", 1)])
@pytest.mark.parametrize("first", ["graph", "resident"])
def test_new_values_on_a_kept_matrix(kind, precond, first):
    """Solve, change the values, solve with the other kernels, and once more."""
    m = mesh.perturbed(mesh.plain_small(8), 0.2, 5)
    l2g = O.dof_build(m.tets, m.dirichlet, gauge=O.GAUGE_REF)["l2g"]
    s = System(m, l2g)
    nu = s.nu.copy()
    oracle = O.pcg if kind == "cg" else O.bicgstab
    for k, scale in enumerate((1.0, 2.5, 0.4)):
        s.nu = nu * scale
        s.assemble()
        lib().emg_test_set_resident(int((first == "resident") == (k % 2 == 0)))
        rp, col, kv, _, rhs = s.export()
        rp = rp.astype(np.int64)
        x, out = solve(s.matrix(0), rhs, kind, tol=1e-10, max_iter=5000, precond=precond)
        xo, st, it, _ = oracle(rp, col, kv, rhs, tol=1e-10, max_iter=5000, precond=precond)
        assert out.status == st
        assert abs(out.iterations - it) <= max(3, 0.15 * it)
        if st == 0:
            r = np.linalg.norm(rhs - O.spmv(rp, col, kv, x)) / np.linalg.norm(rhs)
            assert r <= 1.1e-10
