"""High contrast between two halves of a mesh: the coarse inverse stays definite,
so the two-level iteration itself reaches the tolerance.  (Where it breaks down
the one-level solve runs, and the number of iterations is that solve's.)"""
import numpy as np
import pytest

from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W
from insilico_gb300.system import System

pytestmark = pytest.mark.gpu


def _halves(p, contrast):
    x = p.X[p.conn].mean(axis=1)[:, 0]
    soft = np.where(x > 0.5, contrast, 1.0)
    if p.kernel == "laplace":
        p.kappa = soft
    else:
        p.lam, p.mu = W.lame(soft, 0.3)
    return p


def _iterations(config, n, contrast, persist):
    S = W.setup_system(_halves(W.config(config, n=n), contrast))
    S.set_option(A.OPT_PERSISTENT, persist)
    S.assemble(A.PREC_MIXED)
    two, rel, _ = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-8)
    S.set_option(A.OPT_TWO_LEVEL, 0)
    one, rel1, _ = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-8)
    S.close()
    assert rel <= 1e-8 and rel1 <= 1e-8
    return two, one


@pytest.mark.parametrize("persist", [1, 0])
@pytest.mark.parametrize("config,n", [("c1", 64), ("c2", 16), ("c3", 12)], ids=["quad Q1", "hex", "tet P2"])
def test_contrast_inside_the_aggregates(config, n, persist):
    """1e6: aggregates across the interface give the coarse matrix a condition of
    some 1e5, which the FP32 inversion has to survive"""
    two, one = _iterations(config, n, 1e-6, persist)
    assert two < one


@pytest.mark.parametrize("persist", [1, 0])
@pytest.mark.parametrize("config,n", [("c1", 160), ("c2", 16), ("c3", 12)], ids=["quad Q1", "hex", "tet P2"])
@pytest.mark.parametrize("contrast", [1e-8, 1e-9])
def test_couplings_of_the_soft_half(config, n, contrast, persist):
    """a soft region's couplings, beside diagonal entries 1e8 and 1e9 times theirs"""
    two, one = _iterations(config, n, contrast, persist)
    assert two < one


def test_couplings_of_the_soft_half_of_an_instance():
    X, conn = W.unit_cube("quad", 160, 160)
    kappa = W.config("c1", n=160).kappa
    soft = np.where(X[conn].mean(axis=1)[:, 0] > 0.5, 1e-8, 1.0)
    S = System()
    S.upload_batch(A.QUAD, [(X, conn), (X, conn)])
    S.create_field(1, 1)
    S.constrain_boundary(lambda x: (np.ones((len(x), 1), dtype=bool), 0.0))
    S.number_dofs()
    S.register_pattern()
    S.set_laplace(np.concatenate([soft, kappa]), 2)
    S.set_body_force_nodal(np.tile(W.config("c1", n=160).body, (2, 1)))
    S.assemble(A.PREC_MIXED)
    S.solve(A.SOLVE_CG_FP32_IR, tol=1e-8)
    two, rel = S.batch_stats()
    S.set_option(A.OPT_TWO_LEVEL, 0)
    S.solve(A.SOLVE_CG_FP32_IR, tol=1e-8)
    one, _ = S.batch_stats()
    S.close()
    assert np.all(rel <= 1e-8) and np.all(two < one)


def test_a_solve_beyond_fp32_directions_is_given_up_early():
    """a plate 20 times thinner than wide, 16^3 cells (13,872 equations): neither
    iteration reaches 1e-10; the two-level one gives up after 1,000 iterations
    without a reliable update (graphs of 8 iterations, at most 32 kernels each; the
    last update is at about iteration 200), and the solve ends as the one-level one"""
    p = W.config("c2", n=16)
    p.X = p.X * np.array([1.0, 1.0, 0.05])
    S = W.setup_system(p)
    S.set_option(A.OPT_PERSISTENT, 0)
    S.assemble(A.PREC_MIXED)
    out = {}
    for two_level in (0, 1):
        S.set_option(A.OPT_TWO_LEVEL, two_level)
        S.solve(A.SOLVE_CG_FP32_IR, tol=1e-10, check=False)
        l0 = S.launch_count()
        it, rel, st = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-10, check=False)
        out[two_level] = S.launch_count() - l0, it, rel, st, S.solution()
    S.close()
    assert out[0][3] == out[1][3] == A.ISL_ERR_NOT_CONVERGED
    assert out[0][1:3] == out[1][1:3] and np.array_equal(out[0][4], out[1][4])
    assert out[1][0] - out[0][0] <= (1500 / 8 + 2) * 32 + 100
