"""Batches of many small instances, two-level: the clusters follow the instances'
sizes, so the batch takes no longer than in the shared one-level iteration (the
best of three tries), with the same solutions within 1e-8."""
import time

import numpy as np
import pytest

from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W
from insilico_gb300.system import System

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,degree,side,count", [("quad", 1, 4, 600), ("quad", 1, 32, 600), ("quad", 2, 8, 600),
                                                    ("quad", 2, 16, 300), ("tet", 2, 3, 600), ("tet", 2, 5, 300)])
def test_not_slower_than_one_level(kind, degree, side, count):
    size = (lambda k: (side + k % 3, side)) if kind == "quad" else (lambda k: (side + k % 2, side, side))
    meshes = [W.unit_cube(kind, *size(k)) for k in range(count)]
    S = System()
    S.upload_batch(A.QUAD if kind == "quad" else A.TET, meshes)
    S.create_field(degree, 1)
    S.constrain_boundary(lambda x: (np.ones((len(x), 1), dtype=bool), 0.0))
    S.number_dofs()
    S.register_pattern()
    g = np.random.default_rng(1)
    S.set_laplace(np.exp(g.normal(0.0, 0.5, sum(len(c) for _, c in meshes))), 2 * degree if kind == "quad" else 2)
    S.set_body_force_nodal(np.ones((sum(len(x) for x, _ in meshes), 1)))
    S.assemble(A.PREC_MIXED)

    def run(two_level):
        S.set_option(A.OPT_TWO_LEVEL, two_level)
        S.solve(A.SOLVE_CG_FP32_IR, tol=1e-11)
        t0 = time.perf_counter()
        S.solve(A.SOLVE_CG_FP32_IR, tol=1e-11)
        return time.perf_counter() - t0, S.solution(), S.batch_stats()[1]
    ratio = []
    for _ in range(3):
        (a, x, rel), (b, y, _) = run(1), run(0)
        assert np.all(rel <= 1e-11)
        off, _ = S.batch_info()
        for k in range(count):
            u, v = x[off[k]:off[k + 1]], y[off[k]:off[k + 1]]
            assert np.linalg.norm(u - v) <= 1e-8 * np.linalg.norm(v)
        ratio.append(a / b)
    S.close()
    assert min(ratio) <= 1.0
