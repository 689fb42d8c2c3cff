"""Transmittance: the horizon column's texels in the first warps of the first
blocks, the others around them, at the smallest and at odd sizes."""
import pytest

from parity import TOL_TRANSMITTANCE, check
from test_gpu_parity import gpu_precompute, torch  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tw,th", [(2, 2), (2, 33), (3, 2), (17, 15), (33, 3), (15, 64), (257, 17)])
def test_every_texel_vs_oracle(atmo, oracle, torch, tw, th):  # noqa: F811
    shape = (tw, th, 4, 8, 4, 3, 8, 4)
    atm = oracle.earth_atmosphere()
    ref = oracle.gpu_precompute(atm, shape, 2, combined=True)
    check("transmittance", gpu_precompute(atmo, torch, atm, shape, 2)[0], ref.transmittance,
          TOL_TRANSMITTANCE)
