"""Sums and quotients of the one-launch two-level solves: the warps' FP32 sums
are added in double-float and alpha and beta are the FP32 numbers next to the
quotients of such sums, as with FP64.  Bounds: five adds of two numbers of 48 bits,
each off by at most 2 * 2^-48 of its operands' magnitudes: 2^-44 of the summands'
magnitudes; a quotient half an ulp, and the correction's own rounding, 2^-20 of one."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from insilico_gb300 import build as B

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("device_sums") / "libsums.so"
    cmd = [B.nvcc(), *B.ARCH, "-O3", "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "-o", str(out),
           os.path.join(ROOT, "tests", "device_sums", "sums.cu"), "-lcudart"]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return C.CDLL(str(out))


def _df(x):
    hi = x.astype(np.float32)
    return np.stack([hi, (x - hi).astype(np.float32)], axis=1)


def _run(lib, x, y, num, den):
    n = len(x)
    sx, sy, q = np.zeros((n, 2), np.float32), np.zeros((n, 2), np.float32), np.zeros(n, np.float32)
    p = [np.ascontiguousarray(a, dtype=np.float32) for a in (x, y, num, den)]
    assert lib.run(n, *[a.ctypes.data_as(C.c_void_p) for a in (*p, sx, sy, q)]) == 0
    return sx.astype(np.float64).sum(axis=1), sy.astype(np.float64).sum(axis=1), q


def test_sums_and_quotients(lib):
    g = np.random.default_rng(2)
    n = 4000
    x = (10.0 ** g.uniform(-6, 6, (n, 32))).astype(np.float32)                         # r.r: one sign, twelve decades
    y = (g.normal(size=(n, 32)) * 10.0 ** g.uniform(-4, 4, (n, 32))).astype(np.float32)  # p.q: both signs
    num, den = 10.0 ** g.uniform(-25, 25, n), 10.0 ** g.uniform(-25, 25, n)
    sx, sy, q = _run(lib, x, y, _df(num), _df(den))
    for got, v in ((sx, x), (sy, y)):
        v = v.astype(np.float64)
        # (the exact sum of 32 FP32 numbers over twelve decades needs 24 + 40 + 5 bits: two FP64 words)
        exact = np.array([np.sum(np.sort(r).astype(np.longdouble)) for r in v], dtype=np.longdouble)
        assert np.max(np.abs(got - exact) / np.abs(v).sum(axis=1)) <= 2.0 ** -44
    exact = num / den
    ok = (exact > 1e-30) & (exact < 1e30)
    ulp = np.spacing(np.abs(exact[ok]).astype(np.float32)).astype(np.float64)
    assert ok.sum() > n / 2 and np.max(np.abs(q[ok] - exact[ok]) / ulp) <= 0.5 + 2.0 ** -20


def test_undefined_quotients(lib):
    num = np.array([[1, 0], [0, 0], [-1, 0], [np.nan, 0], [0, 0]], np.float32)
    den = np.array([[0, 0], [0, 0], [0, 0], [1, 0], [2, 0]], np.float32)
    z = np.zeros((5, 32))
    with np.errstate(divide="ignore", invalid="ignore"):
        want = num[:, 0] / den[:, 0]
    assert np.array_equal(_run(lib, z, z, num, den)[2], want, equal_nan=True)
