"""Device memory for the coarse space runs out: each allocation of the two-level
plan fails in turn (test hook), the solve is then the one-level one, bit for
bit, and a new pattern gets its coarse space again."""
import numpy as np
import pytest

from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W
from insilico_gb300.system import System

pytestmark = pytest.mark.gpu


def _batch():
    data = [W.unit_cube("quad", s, s) for s in (9, 21)]
    S = System()
    S.upload_batch(A.QUAD, data)
    S.create_field(2, 1)
    S.constrain_boundary(lambda x: (np.ones((len(x), 1), dtype=bool), 0.0))
    S.number_dofs()
    S.register_pattern()
    S.set_laplace(np.random.default_rng(1).uniform(0.5, 2.0, sum(len(c) for _, c in data)), 4)
    S.set_body_force_nodal(np.ones((sum(len(x) for x, _ in data), 1)))
    return S


CASES = {"cluster, quad Q1 60": (lambda: W.setup_system(W.config("c1", n=60)), 1),
         "grid, hex 13": (lambda: W.setup_system(W.config("c2", n=13)), 1),
         "graph, quad Q1 60": (lambda: W.setup_system(W.config("c1", n=60)), 0),
         "graph, hex 13": (lambda: W.setup_system(W.config("c2", n=13)), 0),
         "batch": (_batch, 1)}


@pytest.mark.parametrize("name", CASES)
def test_every_failing_allocation_leaves_the_one_level_solve(name):
    make, persist = CASES[name]
    S = make()
    S.set_option(A.OPT_PERSISTENT, persist)

    def solve():
        S.register_pattern()
        S.assemble(A.PREC_MIXED)
        it, rel, st = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-10, check=False)
        assert st == A.ISL_OK and rel <= 1e-10
        return it, S.solution()
    S.set_option(A.OPT_TWO_LEVEL, 0)
    one = solve()
    S.set_option(A.OPT_TWO_LEVEL, 1)
    two = solve()
    assert two[0] < one[0]
    failed = 0
    for n in range(1, 80):
        S.set_option(A.OPT_ALLOC_TEST, n)
        it, x = solve()
        if it == two[0]:  # more than there are
            break
        assert it == one[0] and np.array_equal(x, one[1])
        failed += 1
        # the pattern keeps its one-level solve
        it, _, _ = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-10)
        assert it == one[0]
    assert 25 <= failed < 79 and np.array_equal(x, two[1])
    S.set_option(A.OPT_ALLOC_TEST, 0)
    it, x = solve()
    assert it == two[0] and np.array_equal(x, two[1])
    S.close()
