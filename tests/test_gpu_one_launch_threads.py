"""FP64 CG of several host threads at once, each on a context of its own: the
same bits as alone, and no slower in all than as graphs of kernels, which
overlap (8 threads of 17,161 equations; the best of three tries)."""
import threading
import time

import numpy as np
import pytest

from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _system(n, deg):
    p = W.config("c1", n=n)
    p.fedeg, p.qdeg = deg, 2 * deg
    S = W.setup_system(p)
    S.assemble(A.PREC_FP64)
    return S


def _together(systems, count):
    out, barrier = [None] * len(systems), threading.Barrier(len(systems) + 1)

    def work(i):
        barrier.wait()
        for _ in range(count):
            it, _, st = systems[i].solve(A.SOLVE_CG_FP64, tol=1e-10)
            assert st == A.ISL_OK
        out[i] = it, systems[i].solution()
    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(systems))]
    for t in threads:
        t.start()
    barrier.wait()
    t0 = time.perf_counter()
    for t in threads:
        t.join()
    return time.perf_counter() - t0, out


@pytest.mark.parametrize("n,deg", [(6, 1), (100, 1), (66, 2), (124, 2)])
def test_same_bits_beside_other_solves(n, deg):
    """124 and Q2, 61,009 equations: near the largest that half the shared memory of a CTA holds"""
    systems = [_system(n, deg) for _ in range(4)]
    it, _, _ = systems[0].solve(A.SOLVE_CG_FP64, tol=1e-10)
    x = systems[0].solution()
    _, out = _together(systems, 4)
    assert all(o[0] == it and np.array_equal(o[1], x) for o in out)
    for S in systems:
        S.close()


def test_not_slower_than_overlapping_graphs():
    systems = [_system(66, 2) for _ in range(8)]
    ratio = []
    for _ in range(3):
        t = {}
        for persist in (1, 0):
            for S in systems:
                S.set_option(A.OPT_PERSISTENT, persist)
            _together(systems, 1)
            t[persist], _ = _together(systems, 6)
        ratio.append(t[1] / t[0])
    for S in systems:
        S.close()
    assert min(ratio) <= 1.0
