"""Meshes far from the origin: the aggregates and their modes belong to positions
within the mesh, so a shift of 2^23 (where FP32 coordinates are 1 apart; every
coordinate stays exact in FP64) takes the same number of iterations within 3, as
the geometry's rounding, 1e-9 of a unit, moves the matrix by 1e-7."""
import numpy as np
import pytest

from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W
from insilico_gb300.system import System

pytestmark = pytest.mark.gpu

SHIFT = 2.0 ** 23


def _problem(config, n, shift):
    p = W.config(config, n=n)
    fun = p.dirichlet
    p.dirichlet = lambda x: fun(x - shift)
    p.X = p.X + shift
    if p.neumann_plane is not None:
        axis, value, t = p.neumann_plane
        p.neumann_plane = (axis, value + shift, t)
    return p


@pytest.mark.parametrize("persist", [1, 0])
@pytest.mark.parametrize("config,n", [("c1", 64), ("c2", 16), ("c3", 8)], ids=["quad Q1", "hex", "tet P2"])
def test_iterations_do_not_depend_on_the_position(config, n, persist):
    its = []
    for shift in (0.0, SHIFT):
        S = W.setup_system(_problem(config, n, shift))
        S.set_option(A.OPT_PERSISTENT, persist)
        S.assemble(A.PREC_MIXED)
        it, rel, _ = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-9)
        assert rel <= 1e-9
        its.append(it)
        S.close()
    assert its[1] <= its[0] + 3


def test_instances_of_a_batch_far_apart():
    sides = (16, 64, 32)
    its = []
    for shift in (0.0, SHIFT):
        meshes = [W.unit_cube("quad", s, s) for s in sides]
        S = System()
        S.upload_batch(A.QUAD, [(X + k * shift, conn) for k, (X, conn) in enumerate(meshes)])
        S.create_field(2, 1)
        S.constrain_boundary(lambda x: (np.ones((len(x), 1), dtype=bool), 0.0))
        S.number_dofs()
        S.register_pattern()
        S.set_laplace(np.random.default_rng(1).uniform(0.5, 2.0, sum(len(c) for _, c in meshes)), 4)
        S.set_body_force_nodal(np.ones((sum(len(X) for X, _ in meshes), 1)))
        S.assemble(A.PREC_MIXED)
        S.solve(A.SOLVE_CG_FP32_IR, tol=1e-9)
        it, rel = S.batch_stats()
        assert np.all(rel <= 1e-9)
        its.append(it)
        S.close()
    assert np.all(its[1] <= its[0] + 3)
