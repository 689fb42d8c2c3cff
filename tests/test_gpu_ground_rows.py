"""Order-2 scattering density: the ground's irradiance along a theta row as a
line, a line with one kink, or a lookup per direction."""
import pytest

from parity import TOL_SCATTERING, check_masked, robust_masks
from test_gpu_parity import gpu_precompute, torch  # noqa: F401

pytestmark = pytest.mark.gpu


# Irradiance rows of one interval (every ground row a line) to many, over a
# large planet (lines and kinks) and a small one under a thick atmosphere
# (grazing rows reach several intervals: lookups).
@pytest.mark.parametrize("iw", [2, 3, 16, 64, 256])
@pytest.mark.parametrize("rb,rt", [(6360.0, 6420.0), (3000.0, 3120.0)])
def test_ground_rows_vs_oracle(atmo, oracle, torch, iw, rb, rt):  # noqa: F811
    shape = (64, 16, 5, 16, 8, 4, iw, 4)
    atm = oracle.earth_atmosphere(ground_albedo=0.5)
    atm.bottom_radius, atm.top_radius = rb, rt
    ref, masks = robust_masks(oracle, atm, shape, 2, True)
    scattering = gpu_precompute(atmo, torch, atm, shape, 2)[1]
    check_masked("scattering", scattering, ref.scattering, TOL_SCATTERING, masks["scattering"],
                 channels=4)
