"""The scalar product of the two-level solve (contiguous runs of slots per CTA
and per warp): the residual of the solution, recomputed on the host, for fewer
slices than CTAs, rows of very different lengths and more slices per CTA than
one pass takes; every number of slots in flight, 16-bit and 32-bit columns."""
import numpy as np
import pytest
import scipy.sparse as sp

from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-8


def _quad(n):
    p = W.config("c1", n=n)
    p.fedeg, p.qdeg = 1, 2
    return p


CASES = {"quad Q1 47 (67 slices)": lambda: _quad(47), "tet P2 15": lambda: W.config("c3", n=15),
         "quad Q1 800 (19,951 slices)": lambda: _quad(800)}


@pytest.mark.parametrize("case", list(CASES))
def test_residual_of_the_solution(case):
    S = W.setup_system(CASES[case]())
    S.assemble(A.PREC_MIXED)
    rp, ci, v = S.csr()
    K = sp.csr_matrix((v, ci, rp))
    b = S.rhs()
    S.set_option(A.OPT_PERSISTENT, 0)
    kinds = (102, 104, 108) if S.get_option(A.OPT_SCALAR_SLOTS) else (0,)  # (below 20,000 equations: always 12 slots)
    for short in (1, 0):
        S.set_option(A.OPT_SHORT_COLUMNS, short)
        for kind in kinds:
            S.set_option(A.OPT_SPMV32_KIND, kind)
            it, rel, _ = S.solve(A.SOLVE_CG_FP32_IR, tol=TOL)
            assert kind in (0, S.get_option(A.OPT_SPMV32_KIND))
            # far below what (block) Jacobi takes: the two-level solve ran
            assert it < 400
            # the solve stops on the FP64 residual; at these sizes the host's differs by rounding well below 5 %
            r = np.linalg.norm(b - K @ S.solution()) / np.linalg.norm(b)
            assert r <= 1.05 * TOL and rel <= TOL
    S.close()
