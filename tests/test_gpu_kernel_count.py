"""The kernels of one run, counted for launch accounting: the descriptors'
launch, and a pass's one kernel per kind that its instances take."""
import pytest

from test_gpu_parity import torch  # noqa: F401

pytestmark = pytest.mark.gpu


# Tables, transmittance and direct irradiance; single scattering of up to 128 and
# of 257 to 512 columns; two orders of lookups, indirect irradiance and multiple
# scattering by nodes of one and of two columns per lane and by lines.
@pytest.mark.parametrize("sizes,orders,count", [
    (((8, 4),), 1, 1 + 3 + 1), (((8, 4),), 4, 1 + 3 + 1 + 3 * 3),
    (((32, 4), (40, 7), (65, 4)), 3, 1 + 3 + 2 + 2 * (1 + 1 + 3))])
def test_kernel_count(atmo, oracle, torch, sizes, orders, count):  # noqa: F811
    shapes = [(64, 16, 3, 12, mus, nu, 16, 4) for mus, nu in sizes]
    b = atmo.Batch([oracle.earth_atmosphere()] * len(shapes), shapes, orders)
    assert b.kernel_count() == count
