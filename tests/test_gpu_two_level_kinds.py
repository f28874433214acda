"""The two-level and the one-level mixed solve choose their products by
themselves: neither takes over a kind that the other one found for a kernel and
a copy of the matrix of its own.  Solutions within 1e-8 of the FP64 solve at a
residual tolerance of 1e-12, the bar of the other solver tests."""
import numpy as np
import pytest

from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _system(case):
    if case == "quad Q1 60, graph of kernels (3,481 equations)":
        S = W.setup_system(W.config("c1", n=60))
        S.set_option(A.OPT_PERSISTENT, 0)
    else:  # scalar matrix of a node-blocked system above the one-cluster sizes
        S = W.setup_system(W.config("c2", n=28))
        S.set_option(A.OPT_BLOCK_SOLVER, 0)
    S.assemble(A.PREC_MIXED)
    S.solve(A.SOLVE_CG_FP64, tol=1e-13)
    return S, S.solution()


CASES = ["quad Q1 60, graph of kernels (3,481 equations)", "hex 28, scalar matrix (70,644 equations)"]


@pytest.mark.parametrize("case", CASES)
def test_one_level_solve_after_a_two_level_solve(case):
    S, x64 = _system(case)
    it, _, _ = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-12)
    S.set_option(A.OPT_TWO_LEVEL, 0)
    assert S.time_spmv(A.PREC_FP32, 2) > 0.0
    one, rel, st = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-12, check=False)
    assert st == A.ISL_OK and rel <= 1e-12 and one > it
    assert np.linalg.norm(S.solution() - x64) <= 1e-8 * np.linalg.norm(x64)
    # and back
    S.set_option(A.OPT_TWO_LEVEL, 1)
    assert S.solve(A.SOLVE_CG_FP32_IR, tol=1e-12)[0] == it
    S.close()


@pytest.mark.parametrize("case", CASES)
def test_iteration_limit_ends_as_one_level(case):
    S, _ = _system(case)
    it, rel, st = S.solve(A.SOLVE_CG_FP32_IR, tol=1e-12, max_iter=5, check=False)
    assert st == A.ISL_ERR_NOT_CONVERGED and it == 5 and np.isfinite(rel) and rel > 1e-12
    assert np.isfinite(S.solution()).all()
    S.close()


def test_tuning_one_solve_leaves_the_other_choice_alone(tmp_path):
    """100,489 equations: both solves time their products; each choice has a line
    of its own in the tuning file and stays what it was when the other is made"""
    L = A.load()
    path = tmp_path / "tune.txt"
    assert L.isl_tune_cache(str(path).encode()) == A.ISL_OK

    def run(two_level):
        S = W.setup_system(W.config("c1", n=318))
        S.set_option(A.OPT_TWO_LEVEL, two_level)
        S.assemble(A.PREC_MIXED)
        S.solve(A.SOLVE_CG_FP32_IR, tol=1e-8)
        out = S.get_option(A.OPT_SPMV32_KIND), S.get_option(A.OPT_TUNE_RUNS)
        S.close()
        return out
    try:
        two, _ = run(1)
        one, runs = run(0)
        assert runs >= 1
        choice = {}
        for line in path.read_text().splitlines():
            if line.startswith("spmv32"):
                choice.setdefault(line.split()[0], []).append(int(line.split()[-1]))
        assert len(choice) == 2 and all(len(v) == 1 for v in choice.values())
        assert sorted(v[0] for v in choice.values()) == sorted([two, one])
        assert run(1) == (two, 0) and run(0) == (one, 0)
    finally:
        L.isl_tune_cache(None)
