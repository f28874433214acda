"""Shared memory of a batch's one-launch solves: every instance lays out its own,
so an instance just below the limit of a cluster does not fail beside one with
more aggregates to a CTA, and a grid instance is the same in any batch.
Solutions within 1e-8 of the FP64 solve, as the other batched tests."""
import numpy as np
import pytest

from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W
from insilico_gb300.system import System

pytestmark = pytest.mark.gpu


def _uneven():
    """four quarters of a strip, two dense and two sparse in a chequerboard: the boxes of the
    sparse ones hold few rows, so a CTA's share of the work spans many aggregates"""
    parts = []
    for x0, y0 in ((0.0, 0.0), (15.0, 0.5)):
        X, conn = W.unit_cube("quad", 110, 12)
        parts.append((X * [14.7, 0.45] + [x0 + 0.15, y0 + 0.025], conn))
    for x0, y0 in ((15.0, 0.0), (0.0, 0.5)):
        for i in range(120):
            for j in range(4):
                X, conn = W.unit_cube("quad", 1, 1)
                parts.append((X * 0.005 + [x0 + 15.0 * (i + 0.5) / 120, y0 + 0.5 * (j + 0.5) / 4], conn))
    off = np.cumsum([0] + [len(X) for X, _ in parts])
    return np.concatenate([X for X, _ in parts]), np.concatenate([c + o for (_, c), o in zip(parts, off)])


def _solve(meshes, tol=1e-11):
    S = System()
    S.upload_batch(A.QUAD, meshes)
    S.create_field(2, 1)
    S.constrain_boundary(lambda x: (np.ones((len(x), 1), dtype=bool), 0.0))
    S.number_dofs()
    S.register_pattern()
    S.set_laplace(np.concatenate([np.exp(np.random.default_rng(len(c)).normal(0.0, 0.5, len(c))) for _, c in meshes]), 4)
    S.set_body_force_nodal(np.ones((sum(len(x) for x, _ in meshes), 1)))
    S.assemble(A.PREC_MIXED)
    S.solve(A.SOLVE_CG_FP64, tol=1e-12)
    x64 = S.solution()
    S.solve(A.SOLVE_CG_FP32_IR, tol=tol)
    x, (it, rel) = S.solution(), S.batch_stats()
    off, _ = S.batch_info()
    S.close()
    assert np.all(rel <= tol)
    out = []
    for k in range(len(meshes)):
        a, b = x[off[k]:off[k + 1]], x64[off[k]:off[k + 1]]
        assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(b)
        out.append((a, int(it[k])))
    return out


@pytest.mark.parametrize("side", [141, 142, 143])
def test_instance_at_the_limit_beside_one_of_many_aggregates(side):
    """142: 227,596 bytes of 229,376 with at most 9 aggregates to a CTA; the other
    instance has 40, at 204 bytes each; 143 is the first that takes a grid"""
    uneven = _uneven()
    alone = _solve([uneven, W.unit_cube("quad", 9, 9)])[0]
    x, it = _solve([uneven, W.unit_cube("quad", side, side)])[0]
    assert it == alone[1] and np.array_equal(x, alone[0])


def test_grid_instance_does_not_depend_on_its_batch():
    """sides of 150 (89,401 equations) and more are solved over the whole GPU, with
    512 or 1,024 threads a CTA by the rows of a CTA"""
    got = [_solve([W.unit_cube("quad", s, s) for s in sides])[0] for sides in ((150, 5), (150, 260, 12))]
    assert got[0][1] == got[1][1] and np.array_equal(got[0][0], got[1][0])
