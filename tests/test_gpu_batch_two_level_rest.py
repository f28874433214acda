"""What the two-level solves of a batch do not bring to the tolerance follows in
the shared one-level iteration, beside instances that are done: their solutions
stay, bit for bit, and the rest ends within the tolerance.  And instances too
large for a cluster, over the whole GPU."""
import numpy as np
import pytest

from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W
from insilico_gb300.system import System

pytestmark = pytest.mark.gpu


def _tets(parts):
    """P2 Poisson problems (n, contrast of the half x > 0.5)"""
    problems = [W.config("c3", n=n) for n, _ in parts]
    kappa = [np.where(p.X[p.conn].mean(axis=1)[:, 0] > 0.5, c, 1.0) for p, (_, c) in zip(problems, parts)]
    S = System()
    S.upload_batch(A.TET, [(p.X, p.conn) for p in problems])
    S.create_field(2, 1)
    S.constrain_boundary(lambda x: (np.ones((len(x), 1), dtype=bool), 0.0))
    S.number_dofs()
    S.register_pattern()
    S.set_laplace(np.concatenate(kappa), 2)
    S.set_body_force_nodal(np.concatenate([p.body for p in problems]))
    S.assemble(A.PREC_MIXED)
    return S


def test_instances_that_the_two_level_solve_leaves():
    """8^3 with a contrast of 1e12: beyond the range of FP32 directions, the
    two-level iteration breaks down and the one-level one takes some 500"""
    parts = [(4, 1.0), (8, 1e-12), (6, 1.0)]
    S = _tets([parts[0], parts[2]])
    S.solve(A.SOLVE_CG_FP32_IR, tol=1e-8)
    off, _ = S.batch_info()
    alone = [S.solution()[off[k]:off[k + 1]] for k in range(2)]
    it_alone, _ = S.batch_stats()
    S.close()
    S = _tets(parts)
    l0 = S.launch_count()
    _, _, st = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-8)
    launches = S.launch_count() - l0
    x, (it, rel), (off, _) = S.solution(), S.batch_stats(), S.batch_info()
    S.set_option(A.OPT_TWO_LEVEL, 0)
    S.solve(A.SOLVE_CG_FP32_IR, tol=1e-8)
    y, (one, _) = S.solution(), S.batch_stats()
    S.close()
    assert st == A.ISL_OK and np.all(rel <= 1e-8)
    assert launches > 7 * 32  # at least one replay of the shared iteration
    assert it[1] == one[1] and np.array_equal(x[off[1]:off[2]], y[off[1]:off[2]])
    for k, j in ((0, 0), (2, 1)):
        assert it[k] == it_alone[j] and np.array_equal(x[off[k]:off[k + 1]], alone[j])


@pytest.mark.parametrize("deg,sides", [(2, (12, 150, 30)), (2, (145, 160)), (1, (9, 300))])
def test_instances_larger_than_a_cluster(deg, sides):
    """89,401 equations and more: about 251 KB of shared memory per CTA of a
    cluster of 16; solved in one launch each, which the hook can time out"""
    meshes = [W.unit_cube("quad", s, s) for s in sides]
    S = System()
    S.upload_batch(A.QUAD, meshes)
    S.create_field(deg, 1)
    S.constrain_boundary(lambda x: (np.ones((len(x), 1), dtype=bool), 0.0))
    S.number_dofs()
    S.register_pattern()
    S.set_laplace(np.concatenate([np.exp(np.random.default_rng(s).normal(0.0, 0.5, len(c))) for s, (_, c) in zip(sides, meshes)]), 2 * deg)
    S.set_body_force_nodal(np.ones((sum(len(x) for x, _ in meshes), 1)))
    S.assemble(A.PREC_MIXED)
    S.solve(A.SOLVE_CG_FP64, tol=1e-12)
    x64 = S.solution()
    S.solve(A.SOLVE_CG_FP32_IR, tol=1e-11)
    x, (it, rel), (off, _) = S.solution(), S.batch_stats(), S.batch_info()
    S.set_option(A.OPT_BARRIER_TEST, 1)
    assert S.solve(A.SOLVE_CG_FP32_IR, tol=1e-11, check=False)[2] == A.ISL_ERR_TIMEOUT  # a grid ran
    S.set_option(A.OPT_TWO_LEVEL, 0)
    S.solve(A.SOLVE_CG_FP32_IR, tol=1e-11)
    one, _ = S.batch_stats()
    S.close()
    assert np.all(rel <= 1e-11)
    for k, s in enumerate(sides):
        a, b = x[off[k]:off[k + 1]], x64[off[k]:off[k + 1]]
        assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(b)
        assert s * deg < 40 or it[k] <= 0.6 * one[k]
