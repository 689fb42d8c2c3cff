"""Queries whose lookups two lanes make together: a query's result must not
depend on its partner, its place in the warp or the length of the array."""
import numpy as np
import pytest

from test_capi_host import earth_model
from test_gpu_render import gpu_outputs, make_queries, torch, unit  # noqa: F401

pytestmark = pytest.mark.gpu


def queries(n):
    """Inside and outside queries, and one in five that looks away from above
    the atmosphere, so that lookups and early results are partners."""
    rng = np.random.default_rng(7)
    cam, view, sun, point, normal, shadow = make_queries(rng, n, 6360.0, domain=False)
    away = np.arange(n) % 5 == 0
    out = unit(rng, n).astype(np.float32).astype(np.float64)
    cam[away], view[away], point[away] = 6500.0 * out[away], out[away], 6550.0 * out[away]
    return cam, view, sun, point, normal, shadow


@pytest.mark.parametrize("shape", [(16, 8, 4, 8, 5, 3, 8, 4), (64, 16, 16, 64, 4, 16, 64, 16)])
@pytest.mark.parametrize("combined", [True, False])
def test_result_does_not_depend_on_the_partner(atmo, torch, combined, shape):  # noqa: F811
    m = earth_model(atmo, combined=combined, shape=shape)
    m.Init(2)
    q = queries(300)
    luts = m.lut_set()
    whole = gpu_outputs(torch, luts, q)
    assert all(np.all(np.isfinite(v)) for v in whole.values())
    # The same operations on the same texels: equal to the bit.
    for first, n in ((0, 1), (1, 1), (0, 2), (1, 31), (3, 32), (2, 33), (1, 127), (1, 129),
                     (43, 257)):
        part = gpu_outputs(torch, luts, tuple(x[first:first + n] for x in q))
        for k, v in part.items():
            assert np.array_equal(v, whole[k][first:first + n]), (k, first, n)
