"""Admission of the native server (simulated work, no GPU): the memory of the
two-level mixed solve counts where the server's requests run it (one request
per batch, mixed or FP32)."""
import pytest

from insilico_gb300 import _abi as A
from insilico_gb300 import serve


def _overlap(budget, precision, max_batch):
    """whether two equal requests run at the same time within the budget"""
    srv = serve.Server(device=0, max_batch=max_batch, max_batches=2, reserve_bytes=0, precision=precision,
                       test_budget_bytes=budget, test_fake_us_per_elem=40.0, size_ratio=0.0)
    done, _ = srv.run([serve.Request(i, 9, 1.0, 0.0) for i in range(2)], realtime=False)
    srv.close()
    a, b = sorted(done, key=lambda r: r.start)
    return b.start < a.finish


def _footprint(precision, max_batch):
    lo, hi = 0, 1 << 34  # two do not fit, two fit
    assert _overlap(hi, precision, max_batch)
    while hi - lo > 1 << 16:
        mid = (lo + hi) // 2
        if _overlap(mid, precision, max_batch):
            hi = mid
        else:
            lo = mid
    return hi / 2


def test_coarse_space_counts_where_it_is_built():
    plain = _footprint(A.PREC_FP64, 1)
    # 1,000 nodes: 16 aggregates of six modes, 128 coarse unknowns with padding; one FP32 block copy of the matrix
    nnz = min(9 ** 3 * 24 ** 2, 3000 * 24 * 4)
    least = 16 * 128 ** 2 + 4 * nnz
    for precision in (A.PREC_MIXED, A.PREC_FP32):
        assert _footprint(precision, 1) >= plain + least - (1 << 16)
