"""Multiple scattering by nu nodes: a lane holds one or two mu_s columns of a
node and a texel's taps are shuffles; the texels whose nu is clamped are the
sum of two nodes' parts."""
import numpy as np
import pytest

from parity import TOL_SCATTERING, check
from test_gpu_parity import gpu_precompute, torch  # noqa: F401

pytestmark = pytest.mark.gpu


# Nodes per warp 16, 10 (2 idle lanes), 4, 2 and 1, the last warp of a row
# partly filled, with 24 and 31 of 32 lanes; 22 and 19 lanes (lines in shared
# memory); two columns per lane: odd (unaligned pairs and a lane of one
# column), even, and full; the first sizes past either range.
@pytest.mark.parametrize("mus,nu", [(2, 2), (3, 13), (8, 6), (16, 3), (24, 5), (31, 2), (32, 4),
                                    (11, 4), (19, 3), (33, 8), (33, 7), (40, 7), (64, 5), (64, 4),
                                    (65, 4)])
def test_column_counts_vs_oracle(atmo, oracle, torch, mus, nu):  # noqa: F811
    shape = (64, 16, 3, 12, mus, nu, 16, 4)
    atm = oracle.earth_atmosphere()
    ref = oracle.precompute(atm, shape, 3, combined=True)
    scattering = gpu_precompute(atmo, torch, atm, shape, 3)[1]
    check("scattering", scattering, ref.scattering, TOL_SCATTERING, channels=4)


def test_kinds_together_equal_alone(atmo, oracle):
    """One batch whose members take all three multiple-scattering kernels."""
    shapes = [(64, 16, 3, 12, mus, nu, 16, 4) for mus, nu in ((16, 3), (40, 7), (19, 3), (32, 4))]
    atm = oracle.earth_atmosphere()

    def luts(some):
        b = atmo.Batch([atm] * len(some), some, 3)
        b.run()
        atmo.synchronize_stream()
        return [b.read(i, atmo.LUT_SCATTERING) for i in range(len(some))]

    for together, shape in zip(luts(shapes), shapes):
        np.testing.assert_array_equal(together, luts([shape])[0])
