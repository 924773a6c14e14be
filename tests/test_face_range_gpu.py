"""AWENO residuals over the range of the state's units. The WENO weights share
one division (face.cuh: weno5), which multiplies three squared smoothness
indicators: of the order of the twelfth power of the characteristic values, whose
scale is the density's. A gas in units that make its density and pressure large
has the residual of the oracle, which divides weight by weight, to the bound that
the residual has at ordinary densities.

The state carries 1 % of noise, and the four cells next to the symmetry faces are
left out: there the mirrored stencils give smoothness indicators of rounding size,
and weights that are quotients of those once they are far above WENO's eps (inputs
changed in their last bit move the oracle's residual there by 1e-4, and by less than
1e-13 in the cells compared)."""
import numpy as np
import pytest

import ostc
from oracle_bind import OracleRun, rhs_errors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e11, 1e13, 1e22, 1e24, 1e30, 1e50])
def test_aweno_residual_at_large_densities(scale):
    case = ostc.case_vortex(33, 24, 12)
    bv = case.blocks[0].arrays["bv"]
    rng = np.random.default_rng(0)
    f = 1 + 0.01 * (2 * rng.random(bv.shape[1:]) - 1)
    bv[0] *= f * scale
    bv[4] *= f * scale
    bv[1:4] += 5 * (2 * rng.random(bv[1:4].shape) - 1)
    for face in case.faces:
        face.density *= scale
        face.pressure *= scale
    ref = OracleRun(case)
    ref.initialize()
    ref.compute_rhs()
    s, blocks = case.solver()
    s.initialize()
    s.compute_rhs()
    inner = (slice(None), slice(None), slice(4, -4))
    want = ref.blocks[0].arrays["dq"].copy()[inner]
    assert np.isfinite(want).all()
    assert max(rhs_errors(blocks[0].download("dq")[inner], want, ref.flux_scale())) <= 1e-11
    s.close()
