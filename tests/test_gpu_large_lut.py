"""A shading request on a scattering LUT of more than 4 GB, whose texels have
64-bit offsets, against the queries along the same rays."""
import math

import numpy as np
import pytest

from test_gpu_parity import torch  # noqa: F401
from test_gpu_render import TOL_RENDER

pytestmark = pytest.mark.gpu


def test_shade_view_past_4_gb(atmo, oracle, torch):  # noqa: F811
    shape = (64, 16, 160, 1664, 64, 16, 16, 4)
    assert shape[2] * shape[3] * shape[4] * shape[5] * 16 > 1 << 32
    b = atmo.Batch([oracle.earth_atmosphere()], [shape], 1)
    b.run()
    luts = b.lut_set(0)
    # 55 of 60 km high, looking down at 45 degrees: the rays start in slices past
    # 4 GB and end on the ground, where nothing is steep.
    v = atmo.PinholeView()
    s = math.sqrt(0.5)
    for name, x in (("camera", (0.0, 0.0, 6415.0)), ("right", (0.0, 1.0, 0.0)),
                    ("up", (s, 0.0, s)), ("forward", (s, 0.0, -s)),
                    ("sun_direction", (0.36, 0.48, 0.8)), ("albedo", (0.0, 0.0, 0.0))):
        setattr(v, name, (atmo.C.c_float * 3)(*x))
    v.fov_y, v.width, v.height = math.radians(30.0), 64, 48
    sky, shaded = luts.shade_view(v, torch.full((v.height, v.width), 30.0, device="cuda"))
    tan = math.tan(0.5 * v.fov_y)
    sx = ((2 * np.arange(v.width) + 1) / v.width - 1) * tan * v.width / v.height
    sy = (1 - (2 * np.arange(v.height) + 1) / v.height) * tan
    ray = np.array(list(v.forward)) + sx[None, :, None] * np.array(list(v.right)) + \
        sy[:, None, None] * np.array(list(v.up))
    ray = (ray / np.linalg.norm(ray, axis=-1, keepdims=True)).reshape(-1, 3)
    f = lambda x: torch.from_numpy(np.ascontiguousarray(x, np.float32)).cuda()   # noqa: E731
    cam = np.tile(np.array([0.0, 0.0, 6415.0]), (len(ray), 1))
    sun = f(list(v.sun_direction))
    want, _ = luts.sky_radiance(f(cam), f(ray), sun)
    point, _ = luts.sky_radiance_to_point(f(cam), f(cam + 30.0 * ray), sun)
    assert float(want.min()) > 0
    assert float((sky.reshape(-1, 4)[:, :3] / want - 1).abs().max()) <= TOL_RENDER
    # Albedo 0: the in-scattered radiance alone.
    assert float(((shaded.reshape(-1, 4)[:, :3] - point).abs() / want).max()) <= TOL_RENDER
