"""Batched mixed solve with the two-level preconditioner: an instance in a
thread-block cluster of its own, or over the whole GPU where its share of a
CTA does not fit.  Every instance within 1e-8 of its FP64 solution (the bar of
the batched tests) in fewer iterations than one-level, bitwise the same in any
batch."""
import numpy as np
import pytest

from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W
from insilico_gb300.system import System

pytestmark = pytest.mark.gpu


def _instance(side, seed):
    X, conn = W.unit_cube("quad", side, side)
    g = np.random.default_rng(seed)
    return X, conn, np.exp(g.normal(0.0, 0.5, len(conn))), g.uniform(0.0, 1.0, (len(X), 1))


def _batch(sides, deg):
    data = [_instance(s, 10 + s) for s in sides]
    S = System()
    S.upload_batch(A.QUAD, [(d[0], d[1]) for d in data])
    S.create_field(deg, 1)
    S.constrain_boundary(lambda x: (np.ones((len(x), 1), dtype=bool), 0.0))
    S.number_dofs()
    S.register_pattern()
    S.set_laplace(np.concatenate([d[2] for d in data]), 2 * deg)
    S.set_body_force_nodal(np.concatenate([d[3] for d in data]))
    return S


# side 1 and Q1: no equation; 125 and Q2: 62,001 equations, more than a cluster's shared memory holds
@pytest.mark.parametrize("deg,sides", [(1, (1, 2, 64, 5, 33)), (2, (3, 40, 1, 17)), (2, (12, 125, 30))])
def test_every_instance_matches_fp64(deg, sides):
    S = _batch(sides, deg)
    S.assemble(A.PREC_MIXED)
    S.solve(A.SOLVE_CG_FP64, tol=1e-12)
    x64 = S.solution()
    S.solve(A.SOLVE_CG_FP32_IR, tol=1e-11)
    x, (it, rel) = S.solution(), S.batch_stats()
    S.solve(A.SOLVE_CG_FP32_IR, tol=1e-11)
    assert np.array_equal(S.solution(), x)
    S.set_option(A.OPT_TWO_LEVEL, 0)
    S.solve(A.SOLVE_CG_FP32_IR, tol=1e-11)
    one, _ = S.batch_stats()
    off, _ = S.batch_info()
    assert np.all(rel <= 1e-11)
    for k, s in enumerate(sides):
        a, b = x[off[k]:off[k + 1]], x64[off[k]:off[k + 1]]
        assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(b)
        assert it[k] <= one[k] + 2 and (s * deg < 40 or it[k] <= 0.6 * one[k])
    # FP32 tangent only
    S.set_option(A.OPT_TWO_LEVEL, 1)
    S.assemble(A.PREC_FP32)
    S.solve(A.SOLVE_CG_FP32_IR, tol=1e-6)
    assert np.all(S.batch_stats()[1] <= 1e-6)
    S.close()


@pytest.mark.parametrize("deg", [1, 2])
def test_an_instance_does_not_depend_on_its_batch(deg):
    got = {}
    for sides in ((9, 37, 60), (37, 4), (61, 37, 12, 5, 20)):
        S = _batch(sides, deg)
        S.assemble(A.PREC_MIXED)
        S.solve(A.SOLVE_CG_FP32_IR, tol=1e-11)
        off, _ = S.batch_info()
        k = sides.index(37)
        got[sides] = (S.solution()[off[k]:off[k + 1]], S.batch_stats()[0][k])
        S.close()
    ref = next(iter(got.values()))
    for x, it in got.values():
        assert np.array_equal(x, ref[0]) and it == ref[1]


def test_masked_instances_stay_out():
    sides = (20, 33, 9)
    S = _batch(sides, 1)
    S.assemble(A.PREC_MIXED)
    S.solve(A.SOLVE_CG_FP32_IR, tol=1e-11)
    x = S.solution()
    S.assemble(A.PREC_MIXED)
    S.batch_set_mask([True, False, True])
    S.solve(A.SOLVE_CG_FP32_IR, tol=1e-11)
    y, (it, _) = S.solution(), S.batch_stats()
    off, _ = S.batch_info()
    assert it[1] == 0 and not y[off[1]:off[2]].any()
    for k in (0, 2):
        assert np.array_equal(y[off[k]:off[k + 1]], x[off[k]:off[k + 1]])
    S.close()
