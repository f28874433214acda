"""The grid barriers of the solves that run in one cooperative launch: armed so
that they cannot complete, the bounded wait runs out, the solve returns
ISL_ERR_TIMEOUT, and the next solve on the context is bitwise the one before."""
import numpy as np
import pytest

from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W
from insilico_gb300.system import System

pytestmark = pytest.mark.gpu


def _cg():
    p = W.config("c1", n=33)
    p.fedeg, p.qdeg = 2, 4
    S = W.setup_system(p)
    S.assemble(A.PREC_FP64)
    return S, A.SOLVE_CG_FP64


def _bicgstab():
    X, conn = W.unit_cube("quad", 17, 13)
    S = System()
    W.heat_setup(S, X, conn, m=2.0)
    S.set_values(np.linspace(0.1, 0.9, S.ndofobj))
    S.assemble(A.PREC_FP64, incremental=True, with_residual=True)
    return S, A.SOLVE_BICGSTAB


def _batch():
    """150 and Q2: 89,401 equations, about 251 KB of shared memory per CTA of a cluster, so a grid"""
    data = [W.unit_cube("quad", s, s) for s in (12, 150)]
    S = System()
    S.upload_batch(A.QUAD, data)
    S.create_field(2, 1)
    S.constrain_boundary(lambda x: (np.ones((len(x), 1), dtype=bool), 0.0))
    S.number_dofs()
    S.register_pattern()
    S.set_laplace(np.random.default_rng(1).uniform(0.5, 2.0, sum(len(c) for _, c in data)), 4)
    S.set_body_force_nodal(np.ones((sum(len(x) for x, _ in data), 1)))
    S.assemble(A.PREC_MIXED)
    return S, A.SOLVE_CG_FP32_IR


def _grid():
    S = W.setup_system(W.config("c2", n=13))
    S.assemble(A.PREC_MIXED)
    return S, A.SOLVE_CG_FP32_IR


CASES = {"FP64 CG": _cg, "FP64 BiCGSTAB": _bicgstab, "mixed, one grid": _grid, "batch with a grid instance": _batch}


@pytest.mark.parametrize("name", CASES)
def test_barrier_timeout_reports_status(name):
    S, method = CASES[name]()
    it, _, _ = S.solve(method, tol=1e-10)
    x = S.solution()
    S.set_option(A.OPT_BARRIER_TEST, 1)
    _, _, st = S.solve(method, tol=1e-10, check=False)
    assert st == A.ISL_ERR_TIMEOUT
    it2, _, st = S.solve(method, tol=1e-10)
    assert st == A.ISL_OK and it2 == it and np.array_equal(S.solution(), x)
    S.close()


@pytest.mark.parametrize("name", CASES)
def test_barrier_counter_wraps(name):
    """the barrier's 32-bit counter starts 64 arrivals below its wrap"""
    S, method = CASES[name]()
    it, _, _ = S.solve(method, tol=1e-10)
    x = S.solution()
    S.set_option(A.OPT_BARRIER_TEST, 2)
    it2, _, st = S.solve(method, tol=1e-10, check=False)
    assert st == A.ISL_OK and it2 == it and np.array_equal(S.solution(), x)
    S.close()
