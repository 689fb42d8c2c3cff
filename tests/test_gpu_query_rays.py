"""Render queries along rays at the ends of the lookups' ranges."""
import numpy as np
import pytest

from test_capi_host import earth_model
from test_gpu_render import (OracleRender, ROBUST_POSITION, ROBUST_STEP, compare,  # noqa: F401
                             gpu_outputs, make_queries, oracle_outputs, torch, unit)

pytestmark = pytest.mark.gpu

SHAPE = (16, 8, 4, 8, 5, 3, 8, 4)


def cuda(torch, x):  # noqa: F811
    return torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda()


@pytest.mark.parametrize("combined", [True, False])
def test_far_rays_that_miss_the_atmosphere(atmo, torch, combined):  # noqa: F811
    """Black and unattenuated from any distance."""
    m = earth_model(atmo, combined=combined, shape=SHAPE)
    m.Init(2)
    rng = np.random.default_rng(3)
    out = unit(rng, 256)
    distance = 10.0 ** rng.uniform(4.0, 18.0, (256, 1))
    sky, t = m.lut_set().sky_radiance(cuda(torch, out * distance), cuda(torch, out),
                                      cuda(torch, unit(rng, 256)))
    assert bool((sky == 0).all()) and bool((t == 1).all())


@pytest.mark.parametrize("combined", [True, False])
def test_rays_straight_away_from_the_sun(atmo, oracle, torch, combined):  # noqa: F811
    """view = -sun: rounding takes nu below -1, where the lookup's lower nu node
    is outside the LUT and the upper one has all the weight."""
    shape = oracle.MEDIUM_SHAPE
    m = earth_model(atmo, combined=combined, shape=shape)
    m.Init(3)
    a = m.atmosphere_at()
    rng = np.random.default_rng(19)
    cam, view, _, point, normal, shadow = make_queries(rng, 400, a.bottom_radius, a.top_radius)
    sun = -view
    assert ((view * view).astype(np.float32).sum(1) > 1).sum() > 20
    q = (cam, view, sun, point, normal, shadow)
    S = m.scattering()
    ref = OracleRender(oracle, a, shape, m.transmittance(), S,
                       S if combined else m.single_mie_scattering(), m.irradiance(), combined)
    ref_out = oracle_outputs(ref, q, rng, False)
    # The robustness mask turns view and sun together, so that nu stays -1.
    turned = oracle_outputs(ref, together(q, rng), rng, False)
    terms = np.array([ref.sky(cam[i], view[i], 0.0, sun[i])[0] for i in range(len(cam))])
    factor = 0.5 * (1.0 + np.sum(normal * point, axis=1) / np.linalg.norm(point, axis=1))
    compare(ref_out, turned, gpu_outputs(torch, m.lut_set(), q), "away", terms, factor)


def together(q, rng):
    """The queries moved by what FP32 resolves, view and sun by the same turn."""
    cam, view, sun, point, normal, shadow = q
    n = len(cam)
    turn = rng.normal(size=(n, 3)) * ROBUST_STEP
    v = view + turn
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    move = lambda x: x + rng.normal(size=(n, 3)) * ROBUST_POSITION * np.linalg.norm(  # noqa: E731
        x, axis=1, keepdims=True)
    return move(cam), v, -v, move(point), normal, shadow
