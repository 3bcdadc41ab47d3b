"""The bounded waits of the front solves and root products, with a poll limit of
zero: direct, FETI-DP and mixed-precision solves, the multiplier operators and
the multiplier right-hand side end with EMG_ERR_TIMEOUT; with the limit restored
an infinite right-hand side is no timeout and the next solve is good."""
import ctypes as C

import numpy as np
import pytest
import torch

from emagddm_b200 import _abi, fetidp, mesh
from tests.helpers import lib

pytestmark = pytest.mark.gpu
TF32 = 16  # EMG_FLAG_FACTOR_TF32


@pytest.fixture
def polls():
    def set_to(n):
        _abi.check(lib().emg_test_set_barrier_spins(n), "emg_test_set_barrier_spins")
    yield set_to
    set_to(-1)


@pytest.mark.parametrize("flags", [0, TF32])
@pytest.mark.parametrize("n", [9, 14])
def test_direct_solve_times_out_and_recovers(polls, n, flags):
    m = mesh.perturbed(mesh.plain_scale(n), 0.2, n)
    ds = fetidp.DirectSolver(m)
    assert ds.factor(flags) == 0, lib().emg_last_error()
    b = np.random.default_rng(n).normal(size=ds.n_dofs)
    polls(0)
    _, rc, out = ds.solve(b)
    assert rc == out.status == _abi.EMG_ERR_TIMEOUT, (rc, out.status)
    polls(-1)
    bad = b.copy()
    bad[5] = np.inf
    _, rc, out = ds.solve(bad)
    assert rc not in (0, _abi.EMG_ERR_TIMEOUT)
    _, rc, out = ds.solve(b)
    assert rc == 0 and out.residual_norm <= 1e-12


@pytest.mark.parametrize("flags", [0, TF32])
@pytest.mark.parametrize("n", [10, 24])
def test_fetidp_solve_times_out_and_recovers(polls, n, flags):
    m = mesh.perturbed(mesh.plain_scale(n), 0.2, n)
    fd = fetidp.FetiDP(m, mesh.jittered_partition(m, 2), 8)
    assert fd.factor(flags) == 0, lib().emg_last_error()
    b = np.random.default_rng(n).normal(size=fd.map.n_dofs)
    polls(0)
    _, rc, out = fd.solve_rhs(b)
    assert rc == out.status == _abi.EMG_ERR_TIMEOUT, (rc, out.status)
    polls(-1)
    bad = b.copy()
    bad[5] = np.inf
    _, rc, out = fd.solve_rhs(bad)
    assert rc not in (0, _abi.EMG_ERR_TIMEOUT)
    _, rc, out = fd.solve_rhs(b, max_iter=5000)
    assert rc == 0 and out.residual_norm <= 1e-10


def test_operators_and_right_hand_side_time_out_and_recover(polls):
    """24^3 in 8: the root products wait for their copies."""
    m = mesh.plain_scale(24)
    fd = fetidp.FetiDP(m, mesh.jittered_partition(m, 2), 8)
    assert fd.factor() == 0, lib().emg_last_error()
    v = torch.tensor(np.random.default_rng(0).normal(size=fd.info()["n_lambda"]), device="cuda")
    y = torch.empty_like(v)

    def apply(op):
        return lib().emg_fetidp_apply(fd.h, op, C.c_void_p(v.data_ptr()), C.c_void_p(y.data_ptr()))

    def rhs():
        return lib().emg_fetidp_lambda_rhs(fd.h, None, C.c_void_p(y.data_ptr()))

    polls(0)
    assert apply(0) == apply(1) == rhs() == _abi.EMG_ERR_TIMEOUT
    polls(-1)
    for call in (lambda: apply(0), lambda: apply(1), rhs):
        assert call() == 0, lib().emg_last_error()
        torch.cuda.synchronize()
        assert torch.isfinite(y).all()
