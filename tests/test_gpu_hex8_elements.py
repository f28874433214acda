"""solid::HyperElastic on trilinear hexahedra with the 2x2x2 rule (kernel
k_hyper_hex8): tangent and residual against the oracle at element counts that
take each number of elements per block, with a last block that is not full, for
both materials (NeoHookeanCompressible is contracted in closed form) and both
precisions of the tangent."""
import numpy as np
import pytest

import oracle as O
from insilico_gb300 import _abi as A
from insilico_gb300 import workloads as W
from insilico_gb300.system import System

from helpers import csr_entry_err

pytestmark = pytest.mark.gpu

# FP64: as the other tangents here.  FP32: an entry adds up to 8 elements' sums
# of 8 points and about 6 products each, of factors rounded once or twice, so
# some 50 roundings of 2^-24 of terms no larger than the entry's scale.
TOL = {A.PREC_FP64: 1e-12, A.PREC_FP32: 50 * 2.0 ** -24}


@pytest.mark.parametrize("sizes,per_block", [((1, 1, 1), 4), ((9, 7, 8), 4), ((11, 9, 10), 8), ((13, 13, 12), 16),
                                             ((17, 17, 16), 32)])
@pytest.mark.parametrize("material", ["stvenant", "neohooke"])
@pytest.mark.parametrize("precision", [A.PREC_FP64, A.PREC_FP32])
def test_hex8_tangent_matches_oracle(sizes, per_block, material, precision):
    X, conn = W.unit_cube("hex", *sizes)
    rng = np.random.default_rng(17)
    X = X + rng.uniform(-0.1, 0.1, X.shape) / max(sizes)
    lam, mu = rng.uniform(1.0, 2.0, len(conn)), rng.uniform(0.5, 1.0, len(conn))
    S = System(device=0)
    S.upload_mesh(A.HEX, X, conn)
    S.create_field(1, 3)
    S.constrain_boundary(lambda x: (np.repeat((np.abs(x[:, 2]) < 0.2 / max(sizes))[:, None], 3, axis=1), 0.0))
    S.number_dofs()
    S.register_pattern()
    S.set_hyperelastic(material, lam, mu, 2)
    P = O.Problem(O.HEX, X, conn, 1, 3)
    x, d = P.boundary_points()
    dd = np.repeat(d[np.abs(x[:, 2]) < 0.2 / max(sizes)], 3)
    P.constrain(dd, np.tile(np.arange(3), len(dd) // 3), np.zeros(len(dd)))
    P.number()
    P.set_hyperelastic(material, lam, mu, 2)
    u = rng.uniform(-0.05, 0.05, 3 * S.ndofobj) / max(sizes)
    S.set_values(u)
    P.set_values(u)
    S.assemble(precision, incremental=True, with_residual=True)
    if precision == A.PREC_FP64 and material == "neohooke":  # (StVenant's moduli leave room for 16 at most)
        assert S.get_option(A.OPT_ELEM_VARIANT) == per_block
    rp, ci, v, b = P.assemble(incremental=True, with_residual=True)
    srp, sci, sv = S.csr()
    np.testing.assert_array_equal(srp, rp)
    np.testing.assert_array_equal(sci, ci)
    assert csr_entry_err(rp, ci, sv, v) <= TOL[precision]
    # (the clamped nodes are displaced, so the right-hand side lifts K u with the tangent's entries)
    assert np.max(np.abs(S.rhs() - b)) <= TOL[precision] * np.max(np.abs(b))
    S.close()
