"""A program's first run launches its kernels, the later ones replay a graph;
its descriptors travel as kernel parameters or, many, through a pinned buffer."""
import numpy as np
import pytest

from test_gpu_parity import random_atmosphere, torch  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 3, 30])
def test_later_runs_repeat_the_first(atmo, oracle, torch, count):  # noqa: F811
    rng = np.random.default_rng(5)
    atms = [random_atmosphere(oracle, rng) for _ in range(count)]
    shape = (64, 16, 4, 16, 8, 4, 16, 4)
    b = atmo.Batch(atms, [shape] * count, [3] * count)

    def luts():
        b.run()
        atmo.synchronize_stream()
        return [b.read(i, k) for i in range(count)
                for k in (atmo.LUT_TRANSMITTANCE, atmo.LUT_SCATTERING, atmo.LUT_IRRADIANCE)]

    first = luts()
    for _ in range(2):
        for x, y in zip(luts(), first):
            np.testing.assert_array_equal(x, y)
    # Descriptors of another atmosphere reach the graph's kernels.
    b.set_atmosphere(0, atms[-1] if count > 1 else random_atmosphere(oracle, rng))
    assert any(not np.array_equal(x, y) for x, y in zip(luts()[:3], first[:3]))
