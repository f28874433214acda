"""Performance cases of the framework: what its users run, over the sizes they run it at.

Each case goes through the public Python binding of the C-ABI (`System`, `serve.Server`): the
inputs a caller holds are host arrays (meshes, coefficients, loads), and the results come back
as host arrays, as the ABI takes and gives them.  A context with a registered mesh and pattern
is what a caller keeps between solves, so it is made in prepare(); the coefficients of a pass
are uploaded in the pass.

The kinds, and what they stand for:

  poisson     heat::Laplace with a random conductivity per element and a nodal source: new
              coefficients, assembly, CG, nodal values.  Q1 / Q2 quadrilaterals and P2
              tetrahedra (jittered), mixed precision (the framework's main path) or FP64 (the
              reference's arithmetic).
  elasticity  small-strain elasticity on trilinear hexahedra, one face clamped, a traction on
              the opposite one, two decades of stiffness contrast: mixed or FP64.  `distort`
              moves the interior nodes (no element a parallelepiped).
  batch       many independent Q1 / Q2 Poisson problems of different sizes in one context.
  newton      a compressible neo-Hookean block pulled in load steps: a caller's own Newton loop
              with FP32 tangents, FP32 CG and FP64 residuals.
  served      the same problems submitted to the native server, mixed precision.
  heat        nonlinear heat conduction, Newton with the non-symmetric BiCGSTAB solver.
  setup       a new mesh: DOF numbering, constraints, sparsity pattern (integers only).
  tangent     the neo-Hookean tangent and residual at a displacement, exported as CSR to a
              caller that has a solver of its own.

exact() restates each problem in FP64 with plain torch: element integrals by the textbook
formulas, sparse products, CG / BiCGSTAB / Newton to convergence.
"""
import ctypes
import math

import numpy as np
import torch

from insilico_gb300 import _abi as A
from insilico_gb300 import serve as SV
from insilico_gb300 import workloads as W
from insilico_gb300.system import System


# ---------------------------------------------------------------------------
# the cases
def _poisson(shape, degree, nx, ny, nz, precision):
    return {"kind": "poisson", "shape": shape, "degree": degree, "nx": nx, "ny": ny, "nz": nz, "precision": precision}


def _elasticity(nx, ny, nz, precision, distort):
    return {"kind": "elasticity", "nx": nx, "ny": ny, "nz": nz, "precision": precision, "distort": distort}


def listed():
    return [
        # the smallest scalar solve in earnest: a 64 x 64 Poisson problem inside somebody's loop; latency
        {"name": "poisson_q1_64x64_mixed", **_poisson("quad", 1, 64, 64, 0, "mixed")},
        # the reference's arithmetic on an odd quadratic mesh: a user who checks against it
        {"name": "poisson_q2_121x77_fp64", **_poisson("quad", 2, 121, 77, 0, "fp64")},
        # 3-D heat conduction on quadratic tetrahedra, unstructured matrix, about half a million DOFs
        {"name": "poisson_p2tet_40_mixed", **_poisson("tet", 2, 40, 40, 40, "mixed")},
        # a small ragged component: latency and launches
        {"name": "elasticity_9x7x5_mixed", **_elasticity(9, 7, 5, "mixed", False)},
        # a mid-size part with a distorted mesh, in the reference's arithmetic
        {"name": "elasticity_23x19x17_fp64", **_elasticity(23, 19, 17, "fp64", True)},
        # the large solve: 811,200 DOFs, the benchmark's own size
        {"name": "elasticity_64_mixed", **_elasticity(64, 64, 64, "mixed", False)},
        # a parameter study: many independent quadratic problems of mixed sizes at once
        {"name": "batch_q2_24_mixed", "kind": "batch", "degree": 2, "count": 24, "side_min": 8, "side_max": 96,
         "precision": "mixed"},
        # a nonlinear analysis of one part, the caller's own Newton loop
        {"name": "newton_20_fp32", "kind": "newton", "side": 20, "load_steps": 3},
        # several users' nonlinear parts on one GPU through the server
        {"name": "served_6_mixed", "kind": "served", "count": 6, "side_min": 8, "side_max": 22, "load_steps": 3},
        # nonlinear heat conduction, non-symmetric tangent
        {"name": "heat_q2_61x47", "kind": "heat", "nx": 61, "ny": 47},
        # a new mesh every time (remeshing): numbering and pattern
        {"name": "setup_p2tet_17x13x11", "kind": "setup", "nx": 17, "ny": 13, "nz": 11},
        # tangent and residual handed to another solver
        {"name": "tangent_hex_19x13x12_fp64", "kind": "tangent", "nx": 19, "ny": 13, "nz": 12},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["poisson", "poisson", "poisson", "elasticity", "elasticity", "elasticity", "batch", "newton",
                       "served", "heat", "setup", "tangent"])
    if kind == "poisson":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        if rng.random() < 0.5:
            degree = rng.choice([1, 2])
            nx = _log_int(rng, 16, 320 // degree)
            ny = max(8, min(320 // degree, int(nx * rng.uniform(0.6, 1.5))))
            return _poisson("quad", degree, nx, ny, 0, precision)
        return _poisson("tet", 2, *_around(rng, _log_int(rng, 6, 38), 4, 40), precision)
    if kind == "elasticity":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        n = _log_int(rng, 5, 58 if precision == "mixed" else 36)
        return _elasticity(*_around(rng, n, 3, 64), precision, rng.random() < 0.5)
    if kind == "batch":
        lo = _log_int(rng, 6, 24)
        return {"kind": "batch", "degree": rng.choice([1, 2]), "count": _log_int(rng, 3, 40), "side_min": lo,
                "side_max": lo + _log_int(rng, 4, 80), "precision": rng.choice(["mixed", "mixed", "fp64"])}
    if kind == "newton":
        return {"kind": "newton", "side": _log_int(rng, 6, 30), "load_steps": rng.choice([3, 5])}
    if kind == "served":
        lo = _log_int(rng, 6, 12)
        return {"kind": "served", "count": _log_int(rng, 2, 9), "side_min": lo, "side_max": lo + _log_int(rng, 2, 13),
                "load_steps": rng.choice([3, 5])}
    if kind == "heat":
        nx = _log_int(rng, 12, 90)
        return {"kind": "heat", "nx": nx, "ny": max(8, int(nx * rng.uniform(0.5, 1.2)))}
    nx, ny, nz = _around(rng, _log_int(rng, 5, 22), 3, 26)
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz}


def _around(rng, n, lo, hi):
    return [max(lo, min(hi, int(n * rng.uniform(0.75, 1.1)))) for _ in range(3)]


# tolerances: the linear solves' is the binding's default, relative to the right-hand side
TOL = 1e-10
TOL_HEAT = 1e-9
TOL_NEWTON_LIN = 1e-6      # FP32 tangent: inexact Newton steps
TOL_NEWTON = 1e-16         # ||R|| / N, absolute
MAX_NEWTON = 15
TOL_HEAT_NEWTON = 1e-13
PULL = 0.3


# ---------------------------------------------------------------------------
# meshes and coefficients (numpy; the same for both sides and for exact())
def _grid(n):
    """Nodes of a unit square / cube with n[d] cells per direction, first coordinate fastest."""
    ax = [np.arange(m + 1) / m for m in n]
    g = np.meshgrid(*ax[::-1], indexing="ij")
    return np.ascontiguousarray(np.stack([a.ravel() for a in g[::-1]], axis=1))


def _cells(n):
    """Lexicographic corner ids of every cell, first coordinate fastest."""
    idx = np.meshgrid(*[np.arange(m) for m in n[::-1]], indexing="ij")[::-1]
    stride, s = [], 1
    for m in n:
        stride.append(s)
        s *= m + 1
    base = sum(i.ravel() * st for i, st in zip(idx, stride))
    corners = [sum(((c >> d) & 1) * stride[d] for d in range(len(n))) for c in range(1 << len(n))]
    return base[:, None] + np.array(corners)[None, :]


_QUAD = [0, 1, 3, 2]
_HEX = [0, 1, 3, 2, 4, 5, 7, 6]
# six tetrahedra of a hexahedron (corners in lexicographic order)
_TETS = np.array(_HEX)[np.array([[0, 1, 3, 4], [1, 3, 4, 5], [3, 4, 5, 7], [1, 3, 5, 2], [3, 5, 2, 7], [5, 2, 7, 6]])]


def _mesh(shape, nx, ny, nz=0, jitter=0.0, rng=None):
    n = (nx, ny) if shape == "quad" else (nx, ny, nz)
    X, lex = _grid(n), _cells(n)
    conn = lex[:, _QUAD] if shape == "quad" else lex[:, _HEX] if shape == "hex" else lex[:, _TETS].reshape(-1, 4)
    if jitter:
        h = 1.0 / np.array(n)
        inside = np.all((X > 1e-9) & (X < 1 - 1e-9), axis=1)
        J = rng.uniform(-jitter, jitter, X.shape) * h * inside[:, None]
        if shape == "tet":  # nodes of a tetrahedron that the jitter would turn inside out stay on the grid
            for _ in range(20):
                Y = X + J
                a, b, c, d = (Y[conn[:, i]] for i in range(4))
                bad = np.einsum("ij,ij->i", np.cross(b - a, c - a), d - a) <= 0.05 * np.prod(h)
                if not bad.any():
                    break
                J[np.unique(conn[bad])] = 0.0
        X = X + J
    return np.ascontiguousarray(X), np.ascontiguousarray(conn, dtype=np.int64)


def _rng(seed, stream=0):
    return np.random.Generator(np.random.Philox(np.random.SeedSequence([int(seed) & (2**63 - 1), stream])))


def _poisson_data(case, seed):
    g = _rng(seed)
    tet = case["shape"] == "tet"
    X, conn = _mesh(case["shape"], case["nx"], case["ny"], case["nz"], 0.2 if tet else 0.0, g)
    kappa = np.exp(g.normal(0.0, 1.0 if tet else 0.5, len(conn)))
    return X, conn, kappa, g.uniform(0.0, 1.0, (len(X), 1))


def _elasticity_data(case, seed):
    g = _rng(seed)
    X, conn = _mesh("hex", case["nx"], case["ny"], case["nz"], 0.1 if case["distort"] else 0.0, g)
    E, nu = 10.0 ** g.uniform(3.0, 5.0, len(conn)), g.uniform(0.2, 0.45, len(conn))
    lam, mu = E * nu / (1.0 + nu) / (1.0 - 2.0 * nu), E / 2.0 / (1.0 + nu)
    return X, conn, lam, mu, g.uniform(0.5, 1.5, 3)


def _batch_data(case, seed):
    sides = np.unique(np.round(np.geomspace(case["side_min"], case["side_max"], case["count"])).astype(int))
    sides = np.resize(sides, case["count"])
    out = []
    for k, s in enumerate(sides):
        g = _rng(seed, 1 + k)
        X, conn = _mesh("quad", int(s), int(s))
        out.append((X, conn, np.exp(g.normal(0.0, 0.5, len(conn))), g.uniform(0.0, 1.0, (len(X), 1))))
    return out


def _newton_data(case, seed):
    g = _rng(seed)
    X, conn = _mesh("hex", case["side"], case["side"], case["side"])
    mu = 10.0 ** g.uniform(-1.0, 1.0) * np.exp(g.normal(0.0, 0.2, len(conn)))
    return X, conn, (10.0 - 2.0 / 3.0) * mu, mu


def _served_data(case, seed):
    g = _rng(seed)
    sides = np.round(np.geomspace(case["side_min"], case["side_max"], case["count"])).astype(int)
    return [(int(s), float(10.0 ** g.uniform(-1.0, 1.0))) for s in sides]


def _tangent_data(case, seed):
    g = _rng(seed)
    X, conn = _mesh("hex", case["nx"], case["ny"], case["nz"], 0.1, g)
    mu = np.exp(g.normal(0.0, 0.3, len(conn)))
    u = 0.02 * np.sin(3.0 * X[:, [1, 2, 0]] + g.uniform(0.0, 6.0, 3)) * X[:, :1]
    return X, conn, 3.0 * mu, mu, u


def _heat_param(seed, ne):
    return np.full(ne, 1.5 + 1.5 * _rng(seed).random())


# ---------------------------------------------------------------------------
# prepare / run
def _all_boundary(x):
    return np.ones((len(x), 1), dtype=bool), 0.0


def _clamp(x):
    return np.repeat((np.abs(x[:, 0]) < 1e-9)[:, None], 3, axis=1), 0.0


def _pulled(first):
    def f(x):
        left, right = np.abs(x[:, 0]) < 1e-9, np.abs(x[:, 0] - 1.0) < 1e-9
        mask, vals = np.repeat(left[:, None], 3, axis=1), np.zeros((len(x), 3))
        mask[right, 0] = True
        vals[right, 0] = first
        return mask, vals
    return f


_SHAPE = {"quad": A.QUAD, "tet": A.TET, "hex": A.HEX}


def _context(shape, X, conn, degree, ncomp, dirichlet):
    S = System()
    S.upload_mesh(shape, X, conn)
    S.create_field(degree, ncomp)
    S.constrain_boundary(dirichlet)
    S.number_dofs()
    S.register_pattern()
    return S


def _qdeg(case):
    return 2 if case["shape"] == "tet" or case["degree"] == 1 else 4


def prepare(case, seed):
    kind = case["kind"]
    if kind == "poisson":
        X, conn, kappa, f = _poisson_data(case, seed)
        S = _context(_SHAPE[case["shape"]], X, conn, case["degree"], 1, _all_boundary)
        S.set_body_force_nodal(f)
        return {"kind": kind, "S": S, "kappa": kappa, "qdeg": _qdeg(case), "precision": case["precision"], "tol": TOL}
    if kind == "elasticity":
        X, conn, lam, mu, t = _elasticity_data(case, seed)
        S = _context(A.HEX, X, conn, 1, 3, _clamp)
        e, f = S.boundary_faces()
        e, f = W.faces_on_plane(A.HEX, X, conn, e, f, 0, 1.0)
        S.set_neumann(e, f, t, 2)
        return {"kind": kind, "S": S, "lam": lam, "mu": mu, "precision": case["precision"]}
    if kind == "batch":
        data = _batch_data(case, seed)
        S = System()
        S.upload_batch(A.QUAD, [(X, c) for X, c, _, _ in data])
        S.create_field(case["degree"], 1)
        S.constrain_boundary(_all_boundary)
        S.number_dofs()
        S.register_pattern()
        S.set_body_force_nodal(np.concatenate([d[3] for d in data]))
        return {"kind": "poisson", "S": S, "kappa": np.concatenate([d[2] for d in data]),
                "qdeg": 2 if case["degree"] == 1 else 4, "precision": case["precision"], "tol": TOL}
    if kind == "newton":
        X, conn, lam, mu = _newton_data(case, seed)
        S = _context(A.HEX, X, conn, 1, 3, _pulled(PULL / case["load_steps"]))
        S.set_hyperelastic("neohooke", lam, mu, 3)
        return {"kind": kind, "S": S, "steps": case["load_steps"], "zero": np.zeros(len(X) * 3)}
    if kind == "served":
        reqs = []
        for k, (side, mu) in enumerate(_served_data(case, seed)):
            r = SV.Request(k, side=side, mu=mu, load_steps=case["load_steps"], pull=PULL)
            reqs.append((r, SV.request_arrays(r)))
        srv = SV.Server(precision=A.PREC_MIXED, max_batch=1, max_batches=8, reserve_bytes=1 << 30, lin_tol=TOL)
        return {"kind": kind, "server": srv, "requests": reqs}
    if kind == "heat":
        X, conn = _mesh("quad", case["nx"], case["ny"])
        S = System()
        S.upload_mesh(A.QUAD, X, conn)
        S.create_field(2, 1)

        def bc(x):
            left, right = np.abs(x[:, 0]) < 1e-9, np.abs(x[:, 0] - 1.0) < 1e-9
            return (left | right)[:, None], np.where(right, 1.0, 0.0)[:, None]
        S.constrain_boundary(bc)
        n = S.number_dofs()
        S.register_pattern()
        S.set_heat_static("fenics", _heat_param(seed, len(conn)), 5)
        return {"kind": kind, "S": S, "n": n, "zero": np.zeros(S.ndofobj)}
    if kind == "setup":
        X, conn = _mesh("tet", case["nx"], case["ny"], case["nz"], 0.2, _rng(seed))
        order = _rng(seed, 1).permutation(len(conn))  # a mesh generator's element order
        return {"kind": kind, "X": X, "conn": np.ascontiguousarray(conn[order])}
    X, conn, lam, mu, u = _tangent_data(case, seed)
    S = _context(A.HEX, X, conn, 1, 3, _clamp)
    S.set_hyperelastic("neohooke", lam, mu, 3)
    return {"kind": "tangent", "S": S, "u": u.ravel()}


_PREC = {"mixed": (A.PREC_MIXED, A.SOLVE_CG_FP32_IR), "fp64": (A.PREC_FP64, A.SOLVE_CG_FP64)}


def run(state):
    kind = state["kind"]
    if kind == "setup":
        S = _context(A.TET, state["X"], state["conn"], 2, 1, _all_boundary)
        out = {"dof_index": S.dof_index(), "elem_dofobj": S.elem_dofobj()}
        out["rowptr"], out["colind"], _ = S.csr(values=False)
        S.close()
        return out
    if kind == "served":
        srv, reqs = state["server"], state["requests"]
        tickets = [srv.submit(r, a) for r, a in reqs]
        for t in tickets:
            st = srv.L.isl_serve_wait(srv.h, t, 600.0, ctypes.byref(ctypes.c_int()))
            if st != A.ISL_OK:
                raise A.IslError(st, "isl_serve_wait")
        done = [srv.collect(t, r, len(a["X"])) for t, (r, a) in zip(tickets, reqs)]
        for r in done:
            if r.status != A.ISL_OK:
                raise A.IslError(r.status, r.error)
        return {f"u{r.rid}": r.u for r in done}
    S = state["S"]
    if kind == "poisson":
        prec, method = _PREC[state["precision"]]
        S.set_laplace(state["kappa"], state["qdeg"])
        S.assemble(prec)
        S.solve(method, tol=state["tol"])
        S.distribute()
        return S.values()
    if kind == "elasticity":
        prec, method = _PREC[state["precision"]]
        S.set_hyperelastic("stvenant", state["lam"], state["mu"], 3)
        S.assemble(prec)
        S.solve(method, tol=TOL)
        return S.solution()  # a linear analysis: the context stays at the undeformed state
    if kind == "newton":
        S.set_values(state["zero"])
        for step in range(state["steps"]):
            S.scale_constraints(1.0 if step == 0 else (step + 1) / step)
            for _ in range(MAX_NEWTON):
                S.assemble(A.PREC_FP32, incremental=True, with_residual=True)
                if S.norm() < TOL_NEWTON:
                    break
                S.solve(A.SOLVE_CG_FP32_IR, tol=TOL_NEWTON_LIN)
                S.distribute(add=True)
        S.scale_constraints(1.0 / state["steps"])
        return S.values()
    if kind == "heat":
        S.set_values(state["zero"])
        W.heat_newton(S, state["n"], max_iter=12, tolerance=TOL_HEAT_NEWTON, lin_tol=TOL_HEAT)
        return S.values()
    S.set_values(state["u"])
    S.assemble(A.PREC_FP64, incremental=True, with_residual=True)
    rp, ci, v = S.csr()
    return {"rowptr": rp, "colind": ci, "values": v, "rhs": S.rhs()}


# ---------------------------------------------------------------------------
# work: bytes and operations that a pass cannot do without.  A solve is counted as one pass over
# its inputs and outputs (mesh, coefficients, the solution) plus the assembly of the matrix and
# one product with it: how often the matrix is read beyond that is the algorithm's affair.
def _sizes(case):
    kind = case["kind"]
    if kind == "poisson" or kind == "setup":
        shape, deg = (case["shape"], case["degree"]) if kind == "poisson" else ("tet", 2)
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        if shape == "quad":
            return nx * ny, (nx + 1) * (ny + 1), 4, (deg * nx + 1) * (deg * ny + 1), {1: 9, 2: 16}[deg], 2, 1, (deg + 1) ** 2
        return 6 * nx * ny * nz, (nx + 1) * (ny + 1) * (nz + 1), 4, (2 * nx + 1) * (2 * ny + 1) * (2 * nz + 1), 28, 3, 1, 10
    if kind == "heat":
        nx, ny = case["nx"], case["ny"]
        return nx * ny, (nx + 1) * (ny + 1), 4, (2 * nx + 1) * (2 * ny + 1), 16, 2, 1, 9
    nx, ny, nz = (case["side"],) * 3 if kind in ("newton", "one") else (case["nx"], case["ny"], case["nz"])
    nn = (nx + 1) * (ny + 1) * (nz + 1)
    return nx * ny * nz, nn, 8, 3 * nn, 81, 3, 3, 24


def _one(case, setup=False):
    ne, nn, nv, nd, row, dim, nc, nl = _sizes(case)
    nnz = row * nd
    by = nn * dim * 8 + ne * nv * 4 + nd * 8          # mesh and result
    if setup:
        return by + ne * nl * 8 + nd * 8 + nnz * 8, 0.0
    by += ne * 16 + nd * 8 + nnz * 8 + nnz * 12       # coefficients, right-hand side, matrix written and read once
    return by, 2.0 * nnz + ne * nl * nl * 40.0


def work(case):
    kind = case["kind"]
    if kind == "batch":
        tot = [0.0, 0.0]
        for s in np.resize(np.unique(np.round(np.geomspace(case["side_min"], case["side_max"], case["count"])).astype(int)), case["count"]):
            b, f = _one(_poisson("quad", case["degree"], int(s), int(s), 0, ""))
            tot = [tot[0] + b, tot[1] + f]
        return {"bytes": tot[0], "flops": tot[1]}
    if kind == "served":
        tot = [0.0, 0.0]
        for s in np.round(np.geomspace(case["side_min"], case["side_max"], case["count"])).astype(int):
            b, f = _one({"kind": "one", "side": int(s)})
            tot = [tot[0] + b * case["load_steps"], tot[1] + f * case["load_steps"]]
        return {"bytes": tot[0], "flops": tot[1]}
    b, f = _one(case, kind == "setup")
    if kind == "newton":
        b, f = b * case["load_steps"], f * case["load_steps"]
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# exact: the same problems in FP64 torch
_F64 = torch.float64


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    return (x + 1) / 2, w / 2


def _cube_rule(dim, n):
    x, w = _gauss(n)
    pts = np.array(np.meshgrid(*[x] * dim, indexing="ij")).reshape(dim, -1).T
    wts = np.prod(np.array(np.meshgrid(*[w] * dim, indexing="ij")).reshape(dim, -1), axis=0)
    return pts, wts


_TET_RULE = (np.array([[0.1381966011250105] * 3] + [[0.5854101966249685 if i == d else 0.1381966011250105 for i in range(3)]
                                                   for d in range(3)]), np.full(4, 1.0 / 24.0))


def _lag(k, x):
    return ([1 - x, x], [-np.ones_like(x), np.ones_like(x)]) if k == 1 else \
        ([(1 - x) * (1 - 2 * x), 4 * x * (1 - x), x * (2 * x - 1)], [4 * x - 3, 4 - 8 * x, 4 * x - 1])


def _basis(shape, k, x):
    """Values [nq, nf] and reference gradients [nq, nf, dim], vertices, edges, cell in local order."""
    if shape == "tet":
        b = [1 - x.sum(1), x[:, 0], x[:, 1], x[:, 2]]
        db = np.array([[-1, -1, -1], [1, 0, 0], [0, 1, 0], [0, 0, 1]], float)
        if k == 1:
            return np.stack(b, 1), np.repeat(db[None], len(x), 0)
        v = [c * (2 * c - 1) for c in b]
        g = [(4 * c - 1)[:, None] * db[i] for i, c in enumerate(b)]
        for i, j in _TET_EDGES:
            v.append(4 * b[i] * b[j])
            g.append(4 * (b[i][:, None] * db[j] + b[j][:, None] * db[i]))
        return np.stack(v, 1), np.stack(g, 1)
    dim = x.shape[1]
    V, D = zip(*[_lag(k, x[:, d]) for d in range(dim)])
    if shape == "hex":
        pos = [(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)]
    else:
        pos = [(0, 0), (k, 0), (k, k), (0, k)] + ([(1, 0), (2, 1), (1, 2), (0, 1), (1, 1)] if k == 2 else [])
    v = [np.prod([V[d][p[d]] for d in range(dim)], axis=0) for p in pos]
    g = [np.stack([np.prod([(D if d == a else V)[d][p[d]] for d in range(dim)], axis=0) for a in range(dim)], 1) for p in pos]
    return np.stack(v, 1), np.stack(g, 1)


_TET_EDGES = [(0, 1), (1, 2), (2, 0), (3, 0), (3, 1), (3, 2)]
_QUAD_EDGES = [(0, 1), (1, 2), (2, 3), (3, 0)]


def _first_visit(keys):
    """Ids of equal keys in order of first appearance."""
    _, first, inv = np.unique(keys, return_index=True, return_inverse=True)
    rank = np.empty(len(first), np.int64)
    rank[np.argsort(first, kind="stable")] = np.arange(len(first))
    return rank[inv.ravel()], len(first)


def _dofs(shape, k, conn):
    """DOF ids per element: the nodes (degree 1), else vertices, edges, cells in first-visit order."""
    if k == 1:
        return conn, int(conn.max()) + 1
    edges = np.array(_TET_EDGES if shape == "tet" else _QUAD_EDGES)
    v, nv = _first_visit(conn.ravel())
    e = np.sort(conn[:, edges], axis=2)
    e, n1 = _first_visit((e[..., 0] * (int(conn.max()) + 1) + e[..., 1]).ravel())
    cols = [v.reshape(conn.shape), e.reshape(len(conn), -1) + nv]
    n = nv + n1
    if shape == "quad":
        cols.append(n + np.arange(len(conn))[:, None])
        n += len(conn)
    return np.concatenate(cols, axis=1), n


def _boundary_dofs(shape, k, X, conn, dofs, n, pick):
    """DOFs whose support point satisfies pick(x)."""
    pts = np.empty((n, X.shape[1]))
    pts[dofs[:, :conn.shape[1]]] = X[conn]
    if k == 2:
        edges = np.array(_TET_EDGES if shape == "tet" else _QUAD_EDGES)
        pts[dofs[:, conn.shape[1]:conn.shape[1] + len(edges)]] = X[conn[:, edges]].mean(axis=2)
        if shape == "quad":
            pts[dofs[:, -1]] = X[conn].mean(axis=1)
    return pick(pts)


class _Geo:
    """Quadrature on every element: per point the weights detJ w [ne], values and physical gradients."""

    def __init__(self, shape, k, X, conn, rule):
        self.dev = _dev()
        self.X = torch.tensor(X, dtype=_F64, device=self.dev)
        self.xe = self.X[torch.tensor(conn, device=self.dev)]
        pts, self.w = rule
        self.phi, self.dphi = _basis(shape, k, pts)
        self.N, self.dN = _basis(shape, 1, pts)

    def point(self, q):
        J = torch.einsum("eai,aj->eij", self.xe, torch.tensor(self.dN[q], device=self.dev))
        det = torch.linalg.det(J)
        g = torch.einsum("aj,eji->eai", torch.tensor(self.dphi[q], device=self.dev), torch.linalg.inv(J))
        return det * self.w[q], torch.tensor(self.phi[q], device=self.dev), g, torch.tensor(self.N[q], device=self.dev)


def _matrix(Ke, dofs, active, n):
    """CSR matrix over the active DOFs (a map to equations, -1 off) of the element matrices."""
    eq = torch.tensor(active, device=Ke.device)[torch.tensor(dofs, device=Ke.device)]
    m = eq.shape[1]
    r, c = eq[:, :, None].expand(-1, m, m).reshape(-1), eq[:, None, :].expand(-1, m, m).reshape(-1)
    on = (r >= 0) & (c >= 0)
    M = torch.sparse_coo_tensor(torch.stack([r[on], c[on]]), Ke.reshape(-1)[on], (n, n)).coalesce()
    i = M.indices()
    rp = torch.zeros(n + 1, dtype=torch.int64, device=Ke.device)
    rp[1:] = torch.cumsum(torch.bincount(i[0], minlength=n), 0)
    return torch.sparse_csr_tensor(rp, i[1], M.values(), (n, n))


def _gather(Fe, dofs, n):
    out = torch.zeros(n, dtype=_F64, device=Fe.device)
    return out.index_add_(0, torch.tensor(dofs, device=Fe.device).reshape(-1), Fe.reshape(-1))


def _equations(fixed):
    eq = np.cumsum(~fixed) - 1
    eq[fixed] = -1
    return eq, int((~fixed).sum())


def _diag(K):
    rp, ci, v = K.crow_indices(), K.col_indices(), K.values()
    rows = torch.repeat_interleave(torch.arange(len(rp) - 1, device=v.device), rp[1:] - rp[:-1])
    on = rows == ci
    d = torch.zeros(len(rp) - 1, dtype=_F64, device=v.device)
    d[rows[on]] = v[on]
    return d


def _cg(K, b, rounds=3, tol=1e-13, most=20000):
    """Jacobi CG, restarted from the true residual."""
    d = 1.0 / _diag(K)
    x, bn = torch.zeros_like(b), float(torch.linalg.vector_norm(b))
    if bn == 0:
        return x
    for _ in range(rounds):
        r = b - K @ x
        goal, y = max(tol * bn, 1e-7 * float(torch.linalg.vector_norm(r))), torch.zeros_like(b)
        z = d * r
        p, rz = z.clone(), torch.dot(r, z)
        for it in range(most):
            q = K @ p
            a = rz / torch.dot(p, q)
            y += a * p
            r = r - a * q
            z = d * r
            new = torch.dot(r, z)
            p = z + (new / rz) * p
            rz = new
            if it % 16 == 15 and not float(torch.linalg.vector_norm(r)) > goal:
                break
        x = x + y
        if float(torch.linalg.vector_norm(b - K @ x)) < tol * bn:
            break
    return x


def _bicgstab(K, b, tol=1e-13, rounds=4, most=4000):
    d = 1.0 / _diag(K)
    x, bn = torch.zeros_like(b), float(torch.linalg.vector_norm(b))
    for _ in range(rounds):
        r = b - K @ x
        goal = max(tol * bn, 1e-6 * float(torch.linalg.vector_norm(r)))
        r0, p, best, best_x = r.clone(), r.clone(), math.inf, x
        y, rho = x.clone(), torch.dot(r, r)
        for it in range(most):
            v = K @ (d * p)
            a = rho / torch.dot(r0, v)
            s = r - a * v
            t = K @ (d * s)
            w = torch.dot(t, s) / torch.dot(t, t)
            y = y + a * (d * p) + w * (d * s)
            r = s - w * t
            new = torch.dot(r0, r)
            p = r + (new / rho) * (a / w) * (p - w * v)
            rho = new
            if it % 16 == 15:
                now = float(torch.linalg.vector_norm(r))
                if not math.isfinite(now):
                    break
                if now < best:
                    best, best_x = now, y
                if now < goal:
                    break
        x = best_x
        if float(torch.linalg.vector_norm(b - K @ x)) < tol * bn:
            break
    return x


def _exact_poisson(shape, k, X, conn, kappa, f, rule):
    dofs, n = _dofs(shape, k, conn)
    G = _Geo(shape, k, X, conn, rule)
    kap, fe = torch.tensor(kappa, device=G.dev), torch.tensor(f[:, 0][conn], device=G.dev)
    Ke, Fe = 0.0, 0.0
    for q in range(len(G.w)):
        w, phi, g, N = G.point(q)
        Ke = Ke + torch.einsum("e,eai,ebi->eab", w * kap, g, g)
        Fe = Fe + (w * (fe @ N))[:, None] * phi
    fixed = _boundary_dofs(shape, k, X, conn, dofs, n, lambda x: np.any((x < 1e-9) | (x > 1 - 1e-9), axis=1))
    eq, m = _equations(fixed)
    u = torch.zeros(n, dtype=_F64, device=G.dev)
    if m:
        act = torch.tensor(np.nonzero(~fixed)[0], device=G.dev)
        u[act] = _cg(_matrix(Ke, dofs, eq, m), _gather(Fe, dofs, n)[act])
    return u.cpu().numpy()


def _vector_dofs(conn):
    return (conn[:, :, None] * 3 + np.arange(3)).reshape(len(conn), -1)


def _exact_elasticity(case, seed):
    X, conn, lam, mu, t = _elasticity_data(case, seed)
    G = _Geo("hex", 1, X, conn, _cube_rule(3, 2))
    L, M, I = torch.tensor(lam, device=G.dev), torch.tensor(mu, device=G.dev), torch.eye(3, dtype=_F64, device=G.dev)
    Ke = 0.0
    for q in range(8):
        w, _, g, _ = G.point(q)
        Ke = Ke + torch.einsum("e,eai,ebk->eaibk", w * L, g, g) + torch.einsum("e,eak,ebi->eaibk", w * M, g, g) + \
            torch.einsum("e,eaj,ebj,ik->eaibk", w * M, g, g, I)
    # the traction on x = 1: a quarter of each rectangle's area to each corner (distorted meshes keep their boundary nodes)
    load = np.zeros((len(X), 3))
    right = np.nonzero(np.abs(X[:, 0] - 1) < 1e-9)[0]
    wy, wz = (np.where((X[right, d] < 1e-9) | (X[right, d] > 1 - 1e-9), 0.5, 1.0) / m for d, m in ((1, case["ny"]), (2, case["nz"])))
    load[right] = (wy * wz)[:, None] * t
    fixed = np.repeat(np.abs(X[:, 0]) < 1e-9, 3)
    eq, m = _equations(fixed)
    K = _matrix(Ke.reshape(len(conn), 24, 24), _vector_dofs(conn), eq, m)
    del Ke
    return _cg(K, torch.tensor(load.ravel()[~fixed], device=G.dev)).cpu().numpy()


def _neohooke(G, conn, lam, mu, u):
    """Element tangents [ne, 24, 24] and internal forces [ne, 24] at the displacement u [nn, 3]."""
    ue = u[torch.tensor(conn, device=G.dev)]
    I = torch.eye(3, dtype=_F64, device=G.dev)
    Ke, Fe = 0.0, 0.0
    for q in range(8):
        w, _, g, _ = G.point(q)
        F = I + torch.einsum("eai,eaj->eij", ue, g)
        C = torch.einsum("eki,ekj->eij", F, F)
        Ci, lj = torch.linalg.inv(C), torch.log(torch.linalg.det(F))
        S = (lam * lj - mu)[:, None, None] * Ci + mu[:, None, None] * I
        f2 = mu - lam * lj
        B = torch.einsum("eiA,eaB->eaiAB", F, g)          # delta E = sym(B)
        Bs = 0.5 * (B + B.transpose(3, 4))
        CB = torch.einsum("eAB,eCD,ebkCD->ebkAB", Ci, Ci, Bs) * lam[:, None, None, None, None] + \
            2.0 * f2[:, None, None, None, None] * torch.einsum("eAC,ebkCD,eDB->ebkAB", Ci, Bs, Ci)
        Ke = Ke + torch.einsum("e,eaiAB,ebkAB->eaibk", w, Bs, CB) + torch.einsum("e,eaA,eAB,ebB,ik->eaibk", w, g, S, g, I)
        Fe = Fe + torch.einsum("e,eiA,eAB,eaB->eai", w, F, S, g)
    return Ke.reshape(len(conn), 24, 24), Fe.reshape(len(conn), 24)


def _exact_newton(X, conn, lam, mu, steps):
    G = _Geo("hex", 1, X, conn, _cube_rule(3, 2))
    L, M = torch.tensor(lam, device=G.dev), torch.tensor(mu, device=G.dev)
    left, right = np.abs(X[:, 0]) < 1e-9, np.abs(X[:, 0] - 1) < 1e-9
    fixed = np.repeat(left[:, None], 3, axis=1)
    fixed[right, 0] = True
    eq, m = _equations(fixed.ravel())
    dofs = _vector_dofs(conn)
    act = torch.tensor(np.nonzero(eq >= 0)[0], device=G.dev)
    off = torch.tensor(np.nonzero(fixed.ravel())[0], device=G.dev)
    R = torch.tensor(right, device=G.dev)
    u = torch.zeros(len(X), 3, dtype=_F64, device=G.dev)
    d_dofs = torch.tensor(dofs, device=G.dev)
    for step in range(steps):
        du = torch.zeros_like(u)
        du[R, 0] = PULL * (step + 1) / steps - u[R, 0]
        for it in range(14):
            Ke, Fe = _neohooke(G, conn, L, M, u)
            Fe = Fe + torch.einsum("eab,eb->ea", Ke, du.reshape(-1)[d_dofs])  # the prescribed increment, first iteration
            r = -_gather(Fe, dofs, 3 * len(X))[act]
            if it and float(torch.linalg.vector_norm(r)) < 1e-13 * float(mu.mean()):
                break
            v = u.reshape(-1).clone()
            x = _cg(_matrix(Ke, dofs, eq, m), r, rounds=1, tol=1e-11)
            v[act] += x
            v[off] += du.reshape(-1)[off]
            u, du = v.reshape(-1, 3), torch.zeros_like(u)
            if it and float(torch.linalg.vector_norm(x)) < 1e-13 * float(torch.linalg.vector_norm(v)):
                break
    return u.reshape(-1).cpu().numpy()


def _exact_heat(case, seed):
    X, conn = _mesh("quad", case["nx"], case["ny"])
    m = float(_heat_param(seed, 1)[0])
    dofs, n = _dofs("quad", 2, conn)
    G = _Geo("quad", 2, X, conn, _cube_rule(2, 3))
    d = torch.tensor(dofs, device=G.dev)
    fixed = _boundary_dofs("quad", 2, X, conn, dofs, n, lambda x: (x[:, 0] < 1e-9) | (x[:, 0] > 1 - 1e-9))
    one = _boundary_dofs("quad", 2, X, conn, dofs, n, lambda x: x[:, 0] > 1 - 1e-9)
    eq, neq = _equations(fixed)
    act = torch.tensor(np.nonzero(~fixed)[0], device=G.dev)
    u = torch.zeros(n, dtype=_F64, device=G.dev)
    du = torch.tensor(np.where(one, 1.0, 0.0), device=G.dev)
    for it in range(14):
        Ke, Fe, ue = 0.0, 0.0, u[d]
        for q in range(9):
            w, phi, g, _ = G.point(q)
            uq, gu = ue @ phi, torch.einsum("ea,eai->ei", ue, g)
            k, dk = (1 + uq) ** m, m * (1 + uq) ** (m - 1)
            gg = torch.einsum("eai,ei->ea", g, gu)
            Ke = Ke + torch.einsum("e,eai,ebi->eab", w * k, g, g) + (w * dk)[:, None, None] * gg[:, :, None] * phi
            Fe = Fe + (w * k)[:, None] * gg
        Fe = Fe + torch.einsum("eab,eb->ea", Ke, du[d])
        r = -_gather(Fe, dofs, n)[act]
        if it and float(torch.linalg.vector_norm(r)) < 1e-13:
            break
        x = _bicgstab(_matrix(Ke, dofs, eq, neq), r)
        u[act] += x
        u, du = u + du, torch.zeros_like(du)
    return u.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "poisson":
        X, conn, kappa, f = _poisson_data(case, seed)
        rule = _TET_RULE if case["shape"] == "tet" else _cube_rule(2, 2 if case["degree"] == 1 else 3)
        return _exact_poisson(case["shape"], case["degree"], X, conn, kappa, f, rule)
    if kind == "elasticity":
        return _exact_elasticity(case, seed)
    if kind == "batch":
        rule = _cube_rule(2, 2 if case["degree"] == 1 else 3)
        return np.concatenate([_exact_poisson("quad", case["degree"], X, c, k, f, rule) for X, c, k, f in _batch_data(case, seed)])
    if kind == "newton":
        X, conn, lam, mu = _newton_data(case, seed)
        return _exact_newton(X, conn, lam, mu, case["load_steps"])
    if kind == "served":
        out = {}
        for k, (side, mu) in enumerate(_served_data(case, seed)):
            X, conn = _mesh("hex", side, side, side)
            one = np.ones(len(conn))
            out[f"u{k}"] = _exact_newton(X, conn, (10.0 - 2.0 / 3.0) * mu * one, mu * one, case["load_steps"])
        return out
    if kind == "heat":
        return _exact_heat(case, seed)
    if kind == "setup":
        return None
    X, conn, lam, mu, u = _tangent_data(case, seed)
    G = _Geo("hex", 1, X, conn, _cube_rule(3, 2))
    U = torch.tensor(u, device=G.dev)
    Ke, Fe = _neohooke(G, conn, torch.tensor(lam, device=G.dev), torch.tensor(mu, device=G.dev), U)
    dofs, fixed = _vector_dofs(conn), np.repeat(np.abs(X[:, 0]) < 1e-9, 3)
    eq, m = _equations(fixed)
    # the clamped face is held at zero, where u is zero too: nothing is lifted
    K = _matrix(Ke, dofs, eq, m)
    rhs = -_gather(Fe, dofs, 3 * len(X))[torch.tensor(~fixed, device=G.dev)]
    return {"rowptr": None, "colind": None, "values": K.values().cpu().numpy(), "rhs": rhs.cpu().numpy()}
