"""A LUT's device pointer suits consumers that need 512 bytes, as texture
objects on linear memory do, at sizes whose buffers end anywhere."""
import pytest

from test_capi_host import earth_model
from test_gpu_parity import torch  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(17, 5, 3, 6, 5, 3, 7, 3), (33, 9, 5, 14, 5, 3, 17, 5)])
def test_lut_pointers_are_aligned(atmo, oracle, torch, shape):  # noqa: F811
    kinds = (atmo.LUT_TRANSMITTANCE, atmo.LUT_SCATTERING, atmo.LUT_SINGLE_MIE,
             atmo.LUT_IRRADIANCE)
    b = atmo.Batch([oracle.earth_atmosphere()] * 2, [shape] * 2, 2, combined=False)
    views = [b.lut_view(i, k) for i in range(2) for k in kinds]
    m = earth_model(atmo, combined=False, half=True, shape=shape)
    m.Init(2)
    views += [m.lut_view(k) for k in kinds]
    assert [v.device_ptr % 512 for v in views] == [0] * len(views)
