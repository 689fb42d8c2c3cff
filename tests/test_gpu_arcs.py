"""Scattering density above order 2 by arcs (LUTs large enough to take it),
texel by texel against the FP64 GPU oracle."""
import pytest

from parity import TOL_SCATTERING, check, check_masked, robust_masks
from test_gpu_parity import gpu_precompute, torch  # noqa: F401

pytestmark = pytest.mark.gpu


# (R, MU, MU_S, NU, IW).  4 nodes per warp: no kink (NU 2), one, a tile of 2
# rows and idle warps (MU 34, MU_S 33), a chunk of one node (NU 5); 8 per warp:
# a chunk of one (NU 9), of all (NU 8) and two full ones (NU 16), an odd MU_S;
# just below the smallest LUT, which takes lookups.
@pytest.mark.parametrize("r,mu,mus,nu,iw", [
    (8, 48, 64, 2, 2), (8, 64, 33, 3, 16), (12, 34, 33, 4, 16), (8, 64, 20, 5, 64),
    (16, 64, 16, 8, 16), (9, 98, 33, 9, 16), (16, 66, 32, 8, 64), (16, 64, 16, 16, 128),
    (13, 48, 19, 4, 16)])
def test_sizes_vs_gpu_oracle(atmo, oracle, torch, r, mu, mus, nu, iw):  # noqa: F811
    shape = (64, 16, r, mu, mus, nu, iw, 4)
    atm = oracle.earth_atmosphere()
    ref = oracle.gpu_precompute(atm, shape, 3, combined=True)
    scattering = gpu_precompute(atmo, torch, atm, shape, 3)[1]
    check("scattering", scattering, ref.scattering, TOL_SCATTERING, channels=4)


def test_many_ground_kinks_vs_gpu_oracle(atmo, oracle, torch):  # noqa: F811
    """A small planet under a thick atmosphere with a 512-texel irradiance
    row: grazing ground rows of the top slices have over 100 irradiance nodes
    in range, taken 32 candidates at a time."""
    shape = (64, 16, 8, 64, 32, 4, 512, 4)
    atm = oracle.earth_atmosphere()
    atm.bottom_radius, atm.top_radius = 3000.0, 3120.0
    ref, masks = robust_masks(oracle, atm, shape, 3, True, precompute=oracle.gpu_precompute)
    scattering = gpu_precompute(atmo, torch, atm, shape, 3)[1]
    check_masked("scattering", scattering, ref.scattering, TOL_SCATTERING, masks["scattering"],
                 channels=4)
