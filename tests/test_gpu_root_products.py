"""Products with the roots' triangles (L^-T L^-1 w and S_DD w) at root sizes on
both sides of the line between their kernels and with 1 to 8 blocks of 512
columns a row.

The multiplier operator and the deluxe preconditioner are symmetric; in the
products of n <= 4,100 terms with positive definite blocks of condition up to
1e5 the two sides of u.Av = v.Au differ by at most n eps cond < 1e-7 |u||Av|.
The solve reaches a true residual of 1e-10, formed with the assembled sparse
system and, at the smaller sizes, with the oracle's assembly as well (whose
entries agree to 1e-12 of the largest; 1e-9)."""
import ctypes as C

import numpy as np
import pytest
import torch

from emagddm_b200 import _abi, fetidp, mesh
from oracle import oracle as O
from tests.helpers import oracle_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 20, 22, 24, 28, 36, 44, 52])
def test_root_products(n):
    m = mesh.plain_scale(n)
    fd = fetidp.FetiDP(m, mesh.jittered_partition(m, 2), 8)
    L = _abi.lib()
    assert fd.factor() == 0, L.emg_last_error()
    nl = fd.info()["n_lambda"]
    rng = np.random.default_rng(n)
    u, v = (torch.tensor(rng.normal(size=nl), device="cuda") for _ in range(2))
    for op in (0, 1):
        out = []
        for x in (u, v, v):
            y = torch.empty_like(x)
            assert L.emg_fetidp_apply(fd.h, op, C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr())) == 0
            out.append(y)
        assert torch.equal(out[1], out[2])
        a, b = torch.dot(v, out[0]).item(), torch.dot(u, out[1]).item()
        assert abs(a - b) <= 1e-7 * torch.linalg.norm(u).item() * torch.linalg.norm(out[1]).item()
        assert torch.dot(u, out[0]).item() > 0.0
    for precond in (2, 3):
        x, rc, out = fd.solve(tol=1e-10, max_iter=1000, precond=precond)
        assert rc == 0 and out.residual_norm <= 1e-10
        if n <= 24:
            rp, col, kv, _, rhs = oracle_system(m, fd.map.l2g)
            assert np.linalg.norm(rhs - O.spmv(rp, col, kv, x)) <= 1e-9 * np.linalg.norm(rhs)
