"""FP32 tangents of NeoHookeanCompressible hexahedra against the FP64 ones of the
same kernel: the relative Frobenius error of the closed-form contraction is no
larger than that of the earlier one, which formed the 81 moduli of a point in
FP64, rounded them once and contracted them in FP32 (its figure on the same
inputs stands beside each case)."""
import numpy as np
import pytest

from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W
from insilico_gb300.system import System

pytestmark = pytest.mark.gpu

# cells, distortion, lam / mu, strain, error through rounded moduli
CASES = [((6, 5, 4), 0.0, 9.33, 0.05, 8.816e-08), ((6, 5, 4), 0.1, 9.33, 0.05, 5.963e-08),
         ((12, 12, 12), 0.1, 9.33, 0.3, 6.022e-08), ((12, 12, 12), 0.0, 9.33, 0.3, 7.332e-08),
         ((12, 12, 12), 0.1, 3.0, 0.02, 5.725e-08), ((12, 12, 12), 0.1, 1000.0, 0.05, 6.447e-08),
         ((12, 12, 12), 0.1, 0.1, 0.3, 5.561e-08), ((20, 20, 20), 0.0, 9.33, 0.1, 6.806e-08),
         ((8, 8, 8), 0.1, 9.33, 1.0, 5.826e-08), ((22, 7, 7), 0.1, 50.0, 0.5, 6.445e-08)]


@pytest.mark.parametrize("cells,distortion,ratio,strain,before", CASES)
def test_error_is_no_larger_than_through_rounded_moduli(cells, distortion, ratio, strain, before):
    X, conn = W.unit_cube("hex", *cells)
    g = np.random.default_rng(3)
    X = X + distortion * g.uniform(-1, 1, X.shape) / max(cells)
    mu = np.exp(g.normal(0.0, 0.3, len(conn)))
    S = System()
    S.upload_mesh(A.HEX, X, conn)
    S.create_field(1, 3)
    S.constrain_boundary(lambda x: (np.repeat((x[:, 0] < 0.3 / cells[0])[:, None], 3, axis=1), 0.0))
    S.number_dofs()
    S.register_pattern()
    S.set_hyperelastic("neohooke", ratio * mu, mu, 3)
    wave = np.sin(2 * X[:, [1, 2, 0]] + g.uniform(0, 6, 3)) * X[:, :1]
    S.set_values((strain * 0.4 * wave + strain * X * np.array([1.0, -0.3, -0.3])).ravel())
    S.assemble(A.PREC_FP64, incremental=True, with_residual=True)
    v64 = S.csr()[2]
    S.assemble(A.PREC_FP32, incremental=True, with_residual=True)
    v32 = S.csr()[2]
    S.close()
    assert np.linalg.norm(v32 - v64) <= before * np.linalg.norm(v64)
