"""Render queries along rays at the ends of the lookups' ranges."""
import numpy as np
import pytest

from test_capi_host import earth_model
from test_gpu_render import torch, unit  # noqa: F401

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
