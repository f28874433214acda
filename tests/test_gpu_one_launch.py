"""FP64 CG and BiCGSTAB of small systems in one cooperative launch against the
graph of separate kernels: the same recurrences with FP64 sums in another
order, so the same iteration count within 2 %, and solutions that agree to
1e-9 relative at a residual tolerance of 1e-12 (the bar of the FP64 solves)."""
import numpy as np
import pytest

from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _quad(n, deg):
    p = W.config("c1", n=n)
    p.fedeg, p.qdeg = deg, 2 * deg
    return p


CASES = {"quad Q1 2 (1 equation)": lambda: _quad(2, 1), "quad Q1 6 (25, one CTA)": lambda: _quad(6, 1),
         "quad Q1 20 (361)": lambda: _quad(20, 1), "quad Q2 33": lambda: _quad(33, 2),
         "quad Q1 255 (64,516, the largest range)": lambda: _quad(255, 1), "hex 5": lambda: W.config("c2", n=5),
         "hex 16 (81 entries a row)": lambda: W.config("c2", n=16), "tet P2 9": lambda: W.config("c3", n=9),
         "tet P2 15 (columns spread over the numbering)": lambda: W.config("c3", n=15)}


@pytest.mark.parametrize("name", CASES)
def test_cg_matches_the_graph_path(name):
    S = W.setup_system(CASES[name]())
    S.assemble(A.PREC_FP64)
    out = {}
    for persist in (1, 0):
        S.set_option(A.OPT_PERSISTENT, persist)
        l0 = S.launch_count()
        it, rel, _ = S.solve(A.SOLVE_CG_FP64, tol=1e-12)
        launches, x = S.launch_count() - l0, S.solution()
        it2, _, _ = S.solve(A.SOLVE_CG_FP64, tol=1e-12)
        assert it2 == it and np.array_equal(S.solution(), x) and rel <= 1e-12
        out[persist] = (it, x, launches)
    assert abs(out[1][0] - out[0][0]) <= max(2, out[0][0] // 50)
    assert np.linalg.norm(out[1][1] - out[0][1]) <= 1e-9 * np.linalg.norm(out[0][1])
    S.set_option(A.OPT_PERSISTENT, 1)
    it, _, st = S.solve(A.SOLVE_CG_FP64, tol=1e-30, max_iter=1, check=False)
    assert it == 1 and st in (A.ISL_OK, A.ISL_ERR_NOT_CONVERGED)
    S.close()


def test_cg_takes_one_launch():
    S = W.setup_system(_quad(33, 2))
    S.assemble(A.PREC_FP64)
    l0 = S.launch_count()
    S.solve(A.SOLVE_CG_FP64, tol=1e-12)
    assert S.launch_count() - l0 == 1
    S.close()


@pytest.mark.parametrize("nx,ny", [(3, 2), (17, 13), (40, 40)])
def test_bicgstab_matches_the_graph_path(nx, ny):
    X, conn = W.unit_cube("quad", nx, ny)
    from insilico_gb300.system import System
    S = System()
    W.heat_setup(S, X, conn, m=2.0)
    # the tangent at a nonzero state is not symmetric
    S.set_values(np.linspace(0.1, 0.9, S.ndofobj))
    S.assemble(A.PREC_FP64, incremental=True, with_residual=True)
    out = {}
    for persist in (1, 0):
        S.set_option(A.OPT_PERSISTENT, persist)
        it, rel, _ = S.solve(A.SOLVE_BICGSTAB, tol=1e-12)
        x = S.solution()
        it2, _, _ = S.solve(A.SOLVE_BICGSTAB, tol=1e-12)
        assert it2 == it and np.array_equal(S.solution(), x) and rel <= 1e-12
        out[persist] = x
    assert np.linalg.norm(out[1] - out[0]) <= 1e-9 * np.linalg.norm(out[0])
    S.close()


def test_zero_right_hand_side():
    p = _quad(20, 1)
    p.body = np.zeros_like(p.body)
    S = W.setup_system(p)
    S.assemble(A.PREC_FP64)
    for method in (A.SOLVE_CG_FP64, A.SOLVE_BICGSTAB):
        it, _, st = S.solve(method, tol=1e-12)
        assert st == A.ISL_OK and it == 0 and not S.solution().any()
    S.close()
