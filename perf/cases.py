"""The workloads this library is timed on: what a program that solves gauged
edge-element curl-curl systems on the GPU has it do.

Each case is one call, or the short run of calls, that such a program makes
again and again: products with an assembled matrix, a whole solve from a mesh
on the GPU (numbering, assembly, conjugate gradients), re-assembly for new
materials, a time step of the eddy-current operator, ILU0-preconditioned
solves, a batch of small systems, and the factor-and-solve of the FETI-DP and
direct solvers.  The meshes are this package's unit-cube meshes with every
interior node moved (so no two elements are alike); a seed fixes the node
positions, the materials, the current and any vector.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from emagddm_b200 import _abi, batch, fetidp, mesh

JACOBI, ILU0, PLAIN = _abi.PRECOND_JACOBI, _abi.PRECOND_ILU0, _abi.PRECOND_NONE
DELUXE = 2  # EMG_FETI_PRECOND_DELUXE, the default of FetiDP.solve
DIRECT_TOL, KRYLOV_TOL = 1e-12, 1e-10  # the defaults of DirectSolver.solve; of FetiDP.solve and the small solves
STEP_TOL, INV_DT = 1e-12, 1000.0  # time steps of a millisecond


def listed():
    return [
        # matrix products: the smallest system of the smoke run (latency of one
        # call), and the benchmark's 64^3 matrix (larger than L2)
        {"name": "spmv tet 6", "kind": "spmv", "elem": "tet", "n": 6},
        {"name": "spmv tet 64", "kind": "spmv", "elem": "tet", "n": 64},
        # one-shot solves from a mesh on the GPU: the plain small problem, where
        # launches and host work count, and the plain problem at scale
        {"name": "solve tet 16", "kind": "solve", "elem": "tet", "n": 16},
        {"name": "solve tet 64", "kind": "solve", "elem": "tet", "n": 64},
        # new materials on a kept mesh (a parameter sweep): assembly, then the
        # product with the new matrix (the residual of the last solution)
        {"name": "assemble tet 47", "kind": "assemble", "elem": "tet", "n": 47},
        # a time step with new materials: K and M assembled, K + M/dt formed and
        # solved with BiCGSTAB, on hexahedra
        {"name": "step hex 33", "kind": "step", "elem": "hex", "n": 33, "solver": "bicgstab"},
        # ILU0-preconditioned conjugate gradients with the factor of new values
        {"name": "ilu0 tet 16", "kind": "ilu0", "elem": "tet", "n": 16},
        # many small uneven systems in one call, as in a parameter study
        {"name": "batch 48 of 8..32", "kind": "batch", "count": 48, "nmin": 8, "nmax": 32},
        # FETI-DP with new materials on a kept plan: 8 and 64 uneven subdomains
        {"name": "fetidp tet 16 in 8", "kind": "fetidp", "elem": "tet", "n": 16, "parts": 2, "factor": True},
        {"name": "fetidp tet 64 in 64", "kind": "fetidp", "elem": "tet", "n": 64, "parts": 4, "factor": True},
        # the direct backend: factor and solve, and one more right-hand side on
        # a kept factor
        {"name": "direct tet 33", "kind": "direct", "elem": "tet", "n": 33, "factor": True},
        {"name": "direct rhs tet 24", "kind": "direct", "elem": "tet", "n": 24, "factor": False},
    ]


def _between(rng, lo, hi):
    """A whole number, spread over the logarithm of lo..hi."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["spmv", "solve", "assemble", "step", "ilu0", "batch", "fetidp", "direct"])
    if kind == "spmv":
        return {"kind": kind, "elem": rng.choice(["tet", "tet", "hex", "prism"]), "n": _between(rng, 4, 64)}
    if kind == "solve":
        return {"kind": kind, "elem": rng.choice(["tet", "tet", "hex"]), "n": _between(rng, 6, 64)}
    if kind == "assemble":
        return {"kind": kind, "elem": rng.choice(["tet", "tet", "hex", "prism"]), "n": _between(rng, 6, 64)}
    if kind == "step":
        return {"kind": kind, "elem": rng.choice(["tet", "hex"]), "n": _between(rng, 6, 40),
                "solver": rng.choice(["bicgstab", "cg"])}
    if kind == "ilu0":
        return {"kind": kind, "elem": rng.choice(["tet", "tet", "hex"]), "n": _between(rng, 6, 24)}
    if kind == "batch":
        return {"kind": kind, "count": _between(rng, 8, 64), "nmin": rng.randint(6, 10), "nmax": rng.randint(14, 32)}
    if kind == "fetidp":
        parts = rng.choice([2, 2, 3, 4])
        return {"kind": kind, "elem": rng.choice(["tet", "tet", "hex"]),
                "n": parts * _between(rng, 4 if parts > 2 else 5, 16 if parts < 4 else 12), "parts": parts,
                "factor": rng.random() < 0.6}
    return {"kind": kind, "elem": rng.choice(["tet", "tet", "hex"]), "n": _between(rng, 6, 36),
            "factor": rng.random() < 0.6}


# ---- inputs ------------------------------------------------------------------
def _mesh(case, seed):
    """The plain problem at scale (an iron block, an annular coil) with the
    interior nodes moved by up to a fifth of a cell and materials, conductivity
    and current from the seed; the plain small problem (one material, a box
    source) for the solves up to 20 cells a side, as in this package's small
    configuration."""
    small = case["kind"] == "solve" and case["n"] <= 20
    make = {"tet": (mesh.plain_small, mesh.plain_scale), "hex": (mesh.hex_small, mesh.hex_scale),
            "prism": (mesh.prism_small, mesh.prism_scale)}[case["elem"]][0 if small else 1]
    m = mesh.perturbed(make(case["n"]), 0.2, seed)
    rng = np.random.default_rng([seed, 1])
    m.nu = m.nu * rng.uniform(0.7, 1.4, m.nu.shape)
    m.sigma = rng.uniform(0.5, 5.0, m.nu.shape)
    unit = 1e6 if case["kind"] == "step" else 1.0  # A/mm^2 in a transient problem in SI units
    m.sources = [mesh.Source(s.kind, tuple(unit * rng.uniform(0.5, 1.5) * v for v in s.j), s.p) for s in m.sources]
    return m


def _part(case):
    plain = {"tet": mesh.plain_scale, "hex": mesh.hex_scale}[case["elem"]](case["n"])
    return mesh.jittered_partition(plain, case["parts"]), case["parts"] ** 3


def _vector(seed, n):
    return torch.from_numpy(np.random.default_rng([seed, 2]).standard_normal(n)).cuda()


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _p(t):
    return C.c_void_p(t.data_ptr())


class _Problem:
    """A mesh on the GPU with what the library needs beside it."""

    def __init__(self, m):
        self.m = m
        self.xyz = torch.from_numpy(np.ascontiguousarray(m.xyz, np.float64)).cuda()
        self.elems = torch.from_numpy(np.ascontiguousarray(m.tets, np.int32)).cuda()
        self.material = torch.from_numpy(np.ascontiguousarray(m.material, np.int32)).cuda()
        self.dirichlet = torch.from_numpy(np.ascontiguousarray(m.dirichlet, np.int32)).cuda()
        self.nu = np.ascontiguousarray(m.nu, np.float64)
        self.sigma = np.ascontiguousarray(m.sigma, np.float64)
        self.sources, self.n_sources = _abi.sources_array(m.sources)
        self.l2g = torch.empty((m.n_tets, mesh.EDGES_OF_TYPE[m.elem_type]), dtype=torch.int32, device="cuda")

    def number(self):
        edges, free, dofs = C.c_int64(), C.c_int64(), C.c_int64()
        m = self.m
        _abi.check(_abi.lib().emg_dof_build_device(
            m.elem_type, m.n_nodes, m.n_tets, _p(self.elems), len(m.dirichlet), _p(self.dirichlet), 0,
            _abi.GAUGE_REF, _p(self.l2g), C.byref(edges), C.byref(free), C.byref(dofs), _stream()),
            "emg_dof_build_device")
        return dofs.value


class _System:
    """A matrix pattern on the GPU (emg_system), assembled for given materials."""

    def __init__(self, p, n_dofs):
        self.p, self.n = p, n_dofs
        self.h = C.c_void_p()
        _abi.check(_abi.lib().emg_system_create_typed(
            p.m.elem_type, p.m.n_nodes, _p(p.xyz), p.m.n_tets, _p(p.elems), _p(p.material), _p(p.l2g), n_dofs, 1,
            _stream(), C.byref(self.h)), "emg_system_create_typed")

    def assemble(self, flags=0):
        p = self.p
        _abi.check(_abi.lib().emg_system_assemble(self.h, _abi.ptr(p.nu), _abi.ptr(p.sigma), len(p.nu),
                                                  C.cast(p.sources, C.c_void_p), p.n_sources, flags, _stream()),
                   "emg_system_assemble")

    def solve(self, x, precond):
        cfg, out = _abi.KrylovConfig(KRYLOV_TOL, 50000, precond), _abi.Result()
        _abi.check(_abi.lib().emg_system_solve(self.h, 0, C.byref(cfg), _p(x), 1, _stream(), C.byref(out)),
                   "emg_system_solve")

    def rhs(self):
        """The assembled source vector, where it lies on the GPU."""
        at = _abi.lib().emg_system_rhs_device(self.h)
        view = {"shape": (self.n,), "typestr": "<f8", "data": (int(at), False), "version": 3}
        return torch.as_tensor(type("F", (), {"__cuda_array_interface__": view, "owner": self})(), device="cuda")

    def close(self):
        if self.h:
            _abi.lib().emg_system_destroy(self.h)
            self.h = None

    __del__ = close


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        span = case["nmax"] - case["nmin"] + 1
        sizes = [case["nmin"] + (7 * i) % span for i in range(case["count"])]
        b = batch.build_batch([mesh.random_instance(n, seed + i) for i, n in enumerate(sizes)])
        dev = {k: torch.from_numpy(getattr(b, k)).cuda() for k in ("xyz", "tets", "material", "l2g")}
        return {"kind": kind, "batch": b, "arrays": dev, "x": torch.empty(b.n_rows, dtype=torch.float64, device="cuda")}
    m = _mesh(case, seed)
    if kind in ("fetidp", "direct"):
        solver = fetidp.FetiDP(m, *_part(case)) if kind == "fetidp" else fetidp.DirectSolver(m)
        n = solver.map.n_dofs if kind == "fetidp" else solver.n_dofs
        s = {"kind": kind, "solver": solver, "factor": case["factor"],
             "x": torch.empty(n, dtype=torch.float64, device="cuda")}
        if not case["factor"]:
            _abi.check(solver.factor(), "factor")
            s["b"] = _vector(seed, n)
        return s
    p = _Problem(m)
    if kind == "solve":
        return {"kind": kind, "problem": p}
    n = p.number()
    a = _System(p, n)
    s = {"kind": kind, "system": a, "x": torch.empty(n, dtype=torch.float64, device="cuda")}
    if kind in ("spmv", "assemble"):
        s["x"], s["y"] = _vector(seed, n), torch.empty(n, dtype=torch.float64, device="cuda")
    if kind == "spmv":
        a.assemble()
        s["matrix"] = _abi.lib().emg_system_matrix(a.h, 0)
    if kind == "step":
        s["bicgstab"] = case["solver"] == "bicgstab"
    return s


def run(s):
    L, kind = _abi.lib(), s["kind"]
    if kind == "spmv":
        _abi.check(L.emg_spmv(s["matrix"], _p(s["x"]), _p(s["y"]), _stream()), "emg_spmv")
        return s["y"]
    if kind == "solve":
        p = s["problem"]
        n = p.number()
        x = torch.empty(n, dtype=torch.float64, device="cuda")
        a = _System(p, n)
        a.assemble()
        a.solve(x, JACOBI)
        a.close()
        return {"x": x, "l2g": p.l2g}
    if kind == "assemble":
        a = s["system"]
        a.assemble()
        _abi.check(L.emg_spmv(L.emg_system_matrix(a.h, 0), _p(s["x"]), _p(s["y"]), _stream()), "emg_spmv")
        return {"y": s["y"], "f": a.rhs()}
    if kind == "step":
        a = s["system"]
        a.assemble(_abi.FLAG_MASS)
        op = C.c_void_p()
        _abi.check(L.emg_system_combine(a.h, 1.0, INV_DT, C.byref(op)), "emg_system_combine")
        cfg, out = _abi.KrylovConfig(STEP_TOL, 20000, PLAIN if s["bicgstab"] else JACOBI), _abi.Result()
        solve = L.emg_bicgstab_solve_device if s["bicgstab"] else L.emg_cg_solve_device
        rc = solve(op, C.c_void_p(L.emg_system_rhs_device(a.h)), _p(s["x"]), C.byref(cfg), _stream(), C.byref(out))
        L.emg_csr_destroy(op)
        _abi.check(rc, "solve")
        return s["x"]
    if kind == "ilu0":
        a = s["system"]
        a.assemble()
        a.solve(s["x"], ILU0)
        return s["x"]
    if kind == "batch":
        d = s["arrays"]
        system = batch.BatchSystem(s["batch"], _stream(), {k: _p(t) for k, t in d.items()})
        rc, _ = system.solve(s["x"].data_ptr(), tol=KRYLOV_TOL, stream=_stream())
        _abi.check(rc, "emg_batch_cg_solve_device")
        return s["x"]
    solver, x, out = s["solver"], s["x"], _abi.Result()
    if s["factor"]:
        _abi.check(solver.factor(), "factor")
    b = _p(s["b"]) if "b" in s else None
    if kind == "fetidp":
        cfg = _abi.KrylovConfig(KRYLOV_TOL, 2000, DELUXE)
        if b is None:
            rc = L.emg_fetidp_solve(solver.h, C.byref(cfg), _p(x), 1, C.byref(out))
        else:
            rc = L.emg_fetidp_solve_rhs(solver.h, C.byref(cfg), b, _p(x), 1, C.byref(out))
    else:
        cfg = _abi.KrylovConfig(DIRECT_TOL, 6, 0)
        rc = L.emg_direct_solve(solver.h, C.byref(cfg), b, _p(x), 1, C.byref(out))
    _abi.check(rc, "solve")
    return x


# ---- the work of a pass ------------------------------------------------------
# Rows and entries of the `ref`-gauged matrix on n^3 cells (exact for n >= 5).
_ROWS = {"tet": (6, -9, 3, 0), "hex": (2, -4, 2, 0), "prism": (3, -5, 2, 0)}
_ENTRIES = {"tet": (78, -201, 171, -48), "hex": (42, -148, 154, -40), "prism": (45, -129, 102, -20)}
_PER_CELL = {"tet": (6, 4, 6), "hex": (1, 8, 12), "prism": (2, 6, 9)}  # elements; nodes and edges of one
_FLOPS = {"tet": 400.0, "hex": 20000.0, "prism": 9000.0}  # of one element's matrix


def _sizes(elem, n):
    cubic = lambda c: float(max(1, ((c[0] * n + c[1]) * n + c[2]) * n + c[3]))  # noqa: E731
    per, nodes, edges = _PER_CELL[elem]
    return cubic(_ROWS[elem]), cubic(_ENTRIES[elem]), per * n ** 3, nodes, edges


def _matrix_pass(rows, entries):
    return 12.0 * entries + 20.0 * rows, 2.0 * entries


def _assembly(elem, n, mass):
    rows, entries, elems, nodes, edges = _sizes(elem, n)
    read = elems * (4 * nodes + 4 + 4 * edges) + 24.0 * (n + 1) ** 3
    return read + (16 if mass else 8) * entries + 8 * rows, elems * _FLOPS[elem] * (2 if mass else 1)


def _krylov(rows, entries, iterations, products=1):
    """Iterations that read the matrix once a product and each of x, r, p once
    (and write it)."""
    b, f = _matrix_pass(rows, entries)
    return iterations * (products * b + 48.0 * rows), iterations * (products * f + 12.0 * rows)


def work(case):
    kind, b, f = case["kind"], 0.0, 0.0
    if kind == "batch":
        span = case["nmax"] - case["nmin"] + 1
        for i in range(case["count"]):
            n = case["nmin"] + (7 * i) % span
            rows, entries = _sizes("tet", n)[:2]
            for x, y in (_assembly("tet", n, False), _krylov(rows, entries, 28 * n)):
                b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    elem, n = case["elem"], case["n"]
    rows, entries = _sizes(elem, n)[:2]
    if kind == "spmv":
        b, f = _matrix_pass(rows, entries)
    elif kind == "assemble":
        (b, f), (x, y) = _assembly(elem, n, False), _matrix_pass(rows, entries)
        b, f = b + x, f + y
    elif kind in ("solve", "step", "ilu0"):
        b, f = _assembly(elem, n, kind == "step")
        # iterations seen on these meshes; ILU0 reads the factor beside the matrix
        count = {"solve": 28 * n, "step": 60, "ilu0": 12 * n}[kind]
        products = 2 if kind == "ilu0" or case.get("solver") == "bicgstab" else 1
        x, y = _krylov(rows, entries, count, products)
        b, f = b + x, f + y
    elif kind == "fetidp":
        # the multifrontal factor of a subdomain of m^3 cells (its entries ~ m^4,
        # operations ~ m^6), and about 40 multiplier iterations over its dense blocks
        m, k = n / case["parts"], case["parts"] ** 3
        size = {"tet": 1.0, "hex": 0.2}[elem]
        if case["factor"]:
            b, f = 1900.0 * size * k * m ** 4, 1200.0 * size * k * m ** 6
        b += (40 * 1290.0 + 4 * 1900.0) * size * k * m ** 4
        f += 2 * b / 8
    else:
        size = {"tet": 1.0, "hex": 0.2}[elem]
        if case["factor"]:
            b, f = 1200.0 * size * 8 * n ** 4 / 8, 178.0 * size * n ** 6
        b += 2 * 1200.0 * size * n ** 4
        f += 2 * b / 8
    return {"bytes": float(b), "flops": float(f)}


# ---- the same results in plain torch -----------------------------------------
_TET_EDGES = ((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3))
_HEX_EDGES = ((0, 1), (1, 2), (2, 3), (3, 0), (4, 5), (5, 6), (6, 7), (7, 4), (0, 4), (1, 5), (2, 6), (3, 7))
_CORNERS = ((-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1))


def _inside(s, x):
    """Which points lie in the open source region s."""
    p = s.p
    if s.kind == mesh.SRC_BOX:
        return ((x[..., 0] > p[0]) & (x[..., 0] < p[1]) & (x[..., 1] > p[2]) & (x[..., 1] < p[3])
                & (x[..., 2] > p[4]) & (x[..., 2] < p[5]))
    r = torch.sqrt((x[..., 0] - p[0]) ** 2 + (x[..., 1] - p[1]) ** 2)
    return (r > p[2]) & (r < p[3]) & (x[..., 2] > p[4]) & (x[..., 2] < p[5])


def _elements(m, tet_source=None):
    """K_e, M_e and F_e of every element, edges oriented from the lower node."""
    X = torch.from_numpy(m.xyz).cuda()[torch.from_numpy(m.tets.astype(np.int64)).cuda()]
    mat = torch.from_numpy(np.asarray(m.material, np.int64)).cuda()
    nu, sg = torch.from_numpy(np.asarray(m.nu)).cuda()[mat], torch.from_numpy(np.asarray(m.sigma)).cuda()[mat]
    tet = m.tets.shape[1] == 4
    edges = _TET_EDGES if tet else _HEX_EDGES
    E, T = len(edges), X.shape[0]
    K, M = (torch.zeros(T, E, E, dtype=torch.float64, device="cuda") for _ in range(2))
    F = torch.zeros(T, E, dtype=torch.float64, device="cuda")
    if tet:
        J = (X[:, 1:] - X[:, :1]).transpose(1, 2)
        a, b = (5 + 3 * math.sqrt(5)) / 20, (5 - math.sqrt(5)) / 20
        points = [([a if k == q else b for k in range(4)], 1 / 24) for q in range(4)]
    else:
        g = 1 / math.sqrt(3)
        points = [((x, y, z), 1.0) for x in (-g, g) for y in (-g, g) for z in (-g, g)]
    for at, w in points:
        if tet:
            G = torch.linalg.inv(J)                                  # rows: gradients of lambda_1..3
            grad = torch.cat([-G.sum(1, keepdim=True), G], 1)
            W = torch.stack([at[i] * grad[:, j] - at[j] * grad[:, i] for i, j in edges], 1)
            curl = torch.stack([2 * torch.linalg.cross(grad[:, i], grad[:, j]) for i, j in edges], 1)
            pos = sum(at[k] * X[:, k] for k in range(4))
            det = torch.linalg.det(J).abs()
        else:
            c = torch.tensor(_CORNERS, dtype=torch.float64, device="cuda")
            t = torch.tensor(at, dtype=torch.float64, device="cuda")
            l = 1 + c * t
            N = l.prod(1) / 8
            dN = torch.stack([c[:, d] * l[:, (d + 1) % 3] * l[:, (d + 2) % 3] / 8 for d in range(3)], 1)
            J = torch.einsum("tna,nb->tab", X, dN)
            det = torch.linalg.det(J)
            inv = torch.linalg.inv(J)
            pos = torch.einsum("tna,n->ta", X, N)
            Wr, Cr = torch.zeros(12, 3, dtype=torch.float64), torch.zeros(12, 3, dtype=torch.float64)
            for k, (i, j) in enumerate(edges):
                d = next(q for q in range(3) if _CORNERS[i][q] != _CORNERS[j][q])
                u, v = (d + 1) % 3, (d + 2) % 3
                s, cu, cv = (_CORNERS[j][d] - _CORNERS[i][d]) / 2, _CORNERS[i][u], _CORNERS[i][v]
                Wr[k, d] = 0.5 * s * (1 + cu * at[u]) * (1 + cv * at[v])
                Cr[k, u] = 0.5 * s * cv * (1 + cu * at[u])
                Cr[k, v] = -0.5 * s * cu * (1 + cv * at[v])
            W = torch.einsum("tba,kb->tka", inv, Wr.cuda())
            curl = torch.einsum("tab,kb->tka", J, Cr.cuda()) / det[:, None, None]
        K += (nu * w * det)[:, None, None] * (curl @ curl.transpose(1, 2))
        M += (sg * w * det)[:, None, None] * (W @ W.transpose(1, 2))
        for q, s in enumerate(m.sources):
            on = _inside(s, pos)
            if tet_source is not None:
                on = on & (tet_source == q)
            j = torch.tensor(s.j, dtype=torch.float64, device="cuda")
            F += torch.where(on, w * det, torch.zeros_like(det))[:, None] * (W @ j)
    node = torch.from_numpy(m.tets.astype(np.int64)).cuda()
    sign = torch.stack([torch.where(node[:, i] < node[:, j], 1.0, -1.0).double() for i, j in edges], 1)
    return K * sign[:, :, None] * sign[:, None, :], M * sign[:, :, None] * sign[:, None, :], F * sign


class _Plain:
    """The system in 64 bits from the element matrices, matrix-free."""

    def __init__(self, m, l2g, n, inv_dt=None, blocks=None, tet_source=None):
        self.A, M, F = _elements(m, tet_source)
        if inv_dt is not None:
            self.A = self.A + inv_dt * M
        g = torch.as_tensor(l2g).cuda().long()
        self.n, self.at = n, torch.where(g < 0, n, g)
        self.f = self._gather(F)
        self.blocks = blocks  # the system that each row belongs to, where there are several

    def _gather(self, v):
        return torch.zeros(self.n + 1, dtype=torch.float64, device="cuda").index_add_(
            0, self.at.reshape(-1), v.reshape(-1))[:-1]

    def mul(self, x):
        e = torch.cat([x, x.new_zeros(1)])[self.at]
        return self._gather(torch.bmm(self.A, e[:, :, None])[:, :, 0])

    def dense(self):
        E = self.at.shape[1]
        D = torch.zeros((self.n + 1) * (self.n + 1), dtype=torch.float64, device="cuda")
        at = self.at[:, :, None].expand(-1, E, E) * (self.n + 1) + self.at[:, None, :].expand(-1, E, E)
        D.index_add_(0, at.reshape(-1), self.A.reshape(-1))
        return D.view(self.n + 1, self.n + 1)[:-1, :-1]

    def solve(self, b, most=12000):
        if self.n <= 24000 and self.blocks is None:
            L = torch.linalg.cholesky(self.dense())
            x = torch.cholesky_solve(b[:, None], L)[:, 0]
            return x + torch.cholesky_solve((b - self.mul(x))[:, None], L)[:, 0]
        d = self._gather(torch.diagonal(self.A, dim1=1, dim2=2))
        nb = 1 if self.blocks is None else int(self.blocks[-1]) + 1
        dot = ((lambda u, v: torch.dot(u, v)[None]) if nb == 1 else
               (lambda u, v: torch.zeros(nb, dtype=torch.float64, device="cuda").index_add_(0, self.blocks, u * v)))
        spread = (lambda s: s) if nb == 1 else (lambda s: s[self.blocks])
        x, size = torch.zeros_like(b), torch.clamp(dot(b, b), min=1e-300)
        for _ in range(2):  # conjugate gradients, started again once from the true residual
            r = b - self.mul(x)
            z = r / d
            p, rz = z.clone(), dot(r, z)
            for k in range(most):
                q = self.mul(p)
                alpha = torch.where(rz > 0, rz / torch.clamp(dot(p, q), min=1e-300), 0.0)
                x, r = x + spread(alpha) * p, r - spread(alpha) * q
                z = r / d
                new = dot(r, z)
                p, rz = z + spread(torch.where(rz > 0, new / torch.clamp(rz, min=1e-300), 0.0)) * p, new
                if k % 50 == 0 and float((dot(r, r) / size).max()) < 1e-28:
                    break
            else:
                return None
        return x


def exact(case, seed):
    """run()'s results in plain torch; the DOF map is an input, as in prepare().
    None for prisms, and for FETI-DP and direct systems too large for a dense
    factor (their gauge makes plain conjugate gradients slow)."""
    kind = case["kind"]
    if kind == "batch":
        b = prepare(case, seed)["batch"]
        m = mesh.CubeMesh(n=0, xyz=b.xyz, tets=b.tets, material=b.material, dirichlet=None, nu=b.nu, sigma=b.sigma,
                          sources=b.sources)
        rows = torch.from_numpy(np.repeat(np.arange(len(b.instances)), np.diff(b.block_row_ptr))).cuda()
        if len(b.sources) > 64 or m.n_tets > 4_000_000:
            return None
        p = _Plain(m, b.l2g, b.n_rows, blocks=rows, tet_source=torch.from_numpy(b.tet_source).cuda())
        return p.solve(p.f, 3000)
    if case["elem"] == "prism":
        return None
    m = _mesh(case, seed)
    if kind == "fetidp":
        pm = fetidp.partitioned_dofmap(m, *_part(case))
        if pm.n_dofs > 24000:
            return None
        p = _Plain(m, pm.l2g, pm.n_dofs)
        return p.solve(p.f if case["factor"] else _vector(seed, p.n))
    problem = _Problem(m)
    n = problem.number()
    p = _Plain(m, problem.l2g, n, inv_dt=INV_DT if kind == "step" else None)
    if kind == "spmv":
        return p.mul(_vector(seed, n))
    if kind == "assemble":
        return {"y": p.mul(_vector(seed, n)), "f": p.f}
    if kind == "solve":
        return {"x": p.solve(p.f), "l2g": None}
    return p.solve(_vector(seed, n) if kind == "direct" and not case["factor"] else p.f)
