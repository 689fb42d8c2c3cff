"""A sun of angular radius 0 over irradiance LUTs with a column at the horizon
(mu_s = 0), where its average cosine is 0 / 0 as a quotient."""
import numpy as np
import pytest

from parity import TOL_IRRADIANCE, TOL_SCATTERING, check
from test_gpu_parity import gpu_precompute, torch  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iw,mus,nu", [(7, 40, 2), (9, 32, 4), (41, 16, 9), (117, 32, 17)])
def test_luts_are_finite_and_the_limit_of_small_suns(atmo, oracle, torch, iw, mus, nu):  # noqa: F811
    shape = (33, 9, 3, 12, mus, nu, iw, 5)

    def luts(radius):
        atm = oracle.earth_atmosphere()
        atm.sun_angular_radius = radius
        return gpu_precompute(atmo, torch, atm, shape, 4)

    T, S, _, I = luts(0.0)
    _, S1, _, I1 = luts(1e-7)
    assert np.all(np.isfinite(S)) and np.all(np.isfinite(I))
    check("scattering", S, S1, TOL_SCATTERING, channels=4)
    check("irradiance", I, I1, TOL_IRRADIANCE)


@pytest.mark.parametrize("radius", [0.0, 1e-42, 1e-39, 1e-37, 1e-6])
def test_sun_irradiance_at_the_horizon(atmo, oracle, torch, radius):  # noqa: F811
    """On the ground, the sun's centre at the horizon."""
    atm = oracle.earth_atmosphere()
    atm.sun_angular_radius = radius
    b = atmo.Batch([atm], [(33, 9, 3, 12, 8, 4, 8, 5)], 1)
    b.run()
    point = torch.tensor([[atm.bottom_radius, 0.0, 0.0]], device="cuda")
    sun = torch.tensor([[0.0, 1.0, 0.0]], device="cuda")
    direct, sky = b.lut_set(0).sun_and_sky_irradiance(point, sun, sun)
    assert bool(torch.isfinite(direct).all()) and bool(torch.isfinite(sky).all())
