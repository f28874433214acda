"""Two-level preconditioned mixed CG: same solutions as the one-level and the
FP64 solves (1e-8 relative at a residual tolerance of 1e-12, the bar of the
other solver tests), far fewer iterations, bitwise reproducible."""
import numpy as np
import pytest

from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _distorted(n):
    p = W.config("c2", n=n)
    g = np.random.default_rng(5)
    inside = np.all((p.X > 1e-9) & (p.X < 1 - 1e-9), axis=1)
    p.X = p.X + 0.08 / n * g.uniform(-1.0, 1.0, p.X.shape) * inside[:, None]
    return p


def _graded(n):
    """boxes that shrink towards x = 0: equal-width aggregates would hold most nodes in one"""
    p = W.config("c2", n=n)
    p.X = p.X.copy()
    p.X[:, 0] = p.X[:, 0] ** 3
    p.neumann_plane = (0, 1.0, np.array([1.0, 0.0, 0.0]))
    return p


def _thin(n):
    p = W.config("c2", n=n)
    p.X = p.X * np.array([1.0, 1.0, 0.05])
    return p


def _pulled(n):
    p = W.config("c2", n=n)

    def diri(x):
        m = np.repeat((np.abs(x[:, 0]) < 1e-9)[:, None], 3, axis=1)
        v = np.zeros(m.shape)
        right = np.abs(x[:, 0] - 1.0) < 1e-9
        m[right, 0] = True
        v[right, 0] = 0.01
        return m, v
    p.dirichlet, p.neumann_plane = diri, None
    return p


def _quad(n, deg):
    p = W.config("c1", n=n)
    p.fedeg, p.qdeg = deg, 2 * deg
    return p


def _plane_strain(n):
    X, conn = W.unit_cube("quad", n, n)
    g = np.random.default_rng(7)
    lam, mu = W.lame(10.0 ** g.uniform(2.0, 3.0, len(conn)), 0.3)

    def diri(x):
        return np.repeat((np.abs(x[:, 0]) < 1e-9)[:, None], 2, axis=1), 0.0
    return W.Problem("plane strain", A.QUAD, X, conn, 1, 2, "hyperelastic", 3, lam=lam, mu=mu, material="stvenant",
                     body=np.tile([0.0, -1.0], (len(X), 1)), dirichlet=diri)


def _box(nx, ny, nz):
    p = W.config("c2", n=4)
    p.X, p.conn = W.unit_cube("hex", nx, ny, nz)
    g = np.random.default_rng(9)
    p.lam, p.mu = W.lame(10.0 ** g.uniform(3.0, 5.0, len(p.conn)), 0.3)
    return p


CASES = {"hex 5x4x3 (100 nodes)": lambda: _box(5, 4, 3), "hex 9x7x5": lambda: _box(9, 7, 5), "hex 12 (1,872 nodes)": lambda: W.config("c2", n=12), "hex distorted 13": lambda: _distorted(13),
         "hex 21 (more aggregates than one inversion tile)": lambda: W.config("c2", n=21),
         "hex graded 12": lambda: _graded(12), "hex padded 13": lambda: _pulled(13),
         "quad Q1 47 (2,116 equations)": lambda: _quad(47, 1), "quad Q2 40": lambda: _quad(40, 2),
         "quad Q1 160 (sliced ELL)": lambda: _quad(160, 1), "tet P2 9": lambda: W.config("c3", n=9),
         "tet P2 15 (sliced ELL)": lambda: W.config("c3", n=15), "plane strain 40": lambda: _plane_strain(40)}


TOL = {"plane strain 40": 1e-11}


@pytest.mark.parametrize("name", CASES)
def test_same_solution_in_fewer_iterations(name):
    tol = TOL.get(name, 1e-12)
    S = W.setup_system(CASES[name]())
    assert S.get_option(A.OPT_TWO_LEVEL) == 1
    S.assemble(A.PREC_MIXED)
    S.solve(A.SOLVE_CG_FP64, tol=1e-13)
    x64 = S.solution()
    it, rel, _ = S.solve(A.SOLVE_CG_FP32_IR, tol=tol)
    x = S.solution()
    it2, _, _ = S.solve(A.SOLVE_CG_FP32_IR, tol=tol)
    assert it2 == it and np.array_equal(S.solution(), x)
    assert rel <= tol and np.linalg.norm(x - x64) <= 1e-8 * np.linalg.norm(x64)
    # the graph of separate kernels (the default solves these in one launch, but for the largest)
    S.set_option(A.OPT_PERSISTENT, 0)
    small = S.get_option(A.OPT_BLOCKED) and S.neq < 3 * 1280  # one-level on the graph path
    itg, rel, _ = S.solve(A.SOLVE_CG_FP32_IR, tol=tol)
    xg = S.solution()
    assert rel <= tol and np.linalg.norm(xg - x64) <= 1e-8 * np.linalg.norm(x64)
    assert small or abs(itg - it) <= max(3, it // 10)
    S.solve(A.SOLVE_CG_FP32_IR, tol=tol)
    assert np.array_equal(S.solution(), xg)
    S.set_option(A.OPT_PERSISTENT, 1)
    S.set_option(A.OPT_TWO_LEVEL, 0)
    one, _, _ = S.solve(A.SOLVE_CG_FP32_IR, tol=tol)
    assert np.linalg.norm(S.solution() - x64) <= 1e-8 * np.linalg.norm(x64)
    assert it <= 0.85 * one
    # FP32 tangent only: the iterated residual decides
    S.set_option(A.OPT_TWO_LEVEL, 1)
    S.assemble(A.PREC_FP32)
    it32, rel32, _ = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-6)
    assert rel32 <= 1e-6 and 0 < it32 < one
    S.close()


def test_thin_plate_solves_to_the_same_tolerance():
    """a plate 20 times thinner than wide (stretched elements): the aggregates span
    its thickness; the true residual decides, however many iterations that takes"""
    S = W.setup_system(_thin(12))
    S.assemble(A.PREC_MIXED)
    _, rel, _ = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-8)
    assert rel <= 1e-8
    S.close()


def test_tolerance_at_the_fp64_limit_falls_back_to_one_level():
    """plane strain at 1e-12, just above what FP64 residuals of this system can
    reach: where the two-level iteration stagnates the one-level one takes over"""
    S = W.setup_system(_plane_strain(40))
    S.assemble(A.PREC_MIXED)
    _, rel, _ = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-12)
    assert rel <= 1e-12
    S.close()


def test_iteration_limit_zero_load_and_new_mesh():
    p = W.config("c1", n=60)
    S = W.setup_system(p)
    S.assemble(A.PREC_MIXED)
    it, rel, st = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-12, max_iter=5, check=False)
    assert st == A.ISL_ERR_NOT_CONVERGED and it == 5 and rel > 1e-12
    S.set_body_force_nodal(np.zeros((len(p.X), 1)))
    S.assemble(A.PREC_MIXED)
    it, rel, st = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-12)
    assert st == A.ISL_OK and it == 0 and not S.solution().any()
    # the context takes another mesh: new aggregates, new capture
    q = W.config("c2", n=13)
    W.setup_system(q, S)
    S.assemble(A.PREC_MIXED)
    S.solve(A.SOLVE_CG_FP64, tol=1e-13)
    x64 = S.solution()
    S.solve(A.SOLVE_CG_FP32_IR, tol=1e-12)
    assert np.linalg.norm(S.solution() - x64) <= 1e-8 * np.linalg.norm(x64)
    S.close()


def test_grid_barrier_timeout_reports_status():
    """the one-launch grid solve with its barrier armed so that it cannot
    complete: the bounded wait runs out, the solve returns ISL_ERR_TIMEOUT, and
    the next solve on the context is bitwise the one before"""
    S = W.setup_system(W.config("c2", n=13))
    S.assemble(A.PREC_MIXED)
    it, _, _ = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-10)
    x = S.solution()
    S.set_option(A.OPT_BARRIER_TEST, 1)
    _, _, st = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-10, check=False)
    assert st == A.ISL_ERR_TIMEOUT
    it2, _, st = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-10)
    assert st == A.ISL_OK and it2 == it and np.array_equal(S.solution(), x)
    S.close()
