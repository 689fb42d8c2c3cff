"""Single scattering: one, two or four texel columns per thread, transmittance
lines of three-float entries, blocks of two sizes."""
import numpy as np
import pytest

from parity import TOL_SCATTERING, check_masked, robust_masks
from test_gpu_parity import gpu_precompute, torch  # noqa: F401

pytestmark = pytest.mark.gpu


# Columns per row at the edges of the three kernels and of several rows per
# block; transmittance rows of the least width, around a line column per
# thread (128, 256) and beyond what a thread keeps in registers.
@pytest.mark.parametrize("tw,mus,nu", [
    (2, 4, 2), (3, 8, 4), (64, 21, 3), (255, 64, 2), (128, 43, 3), (257, 32, 4), (64, 51, 5),
    (256, 32, 8), (300, 29, 9), (513, 40, 8), (64, 64, 16)])
def test_single_scattering_vs_oracle(atmo, oracle, torch, tw, mus, nu):  # noqa: F811
    shape = (tw, 16, 3, 8, mus, nu, 16, 4)
    atm = oracle.earth_atmosphere()
    ref, masks = robust_masks(oracle, atm, shape, 2, True)
    scattering = gpu_precompute(atmo, torch, atm, shape, 2)[1]
    check_masked("scattering", scattering, ref.scattering, TOL_SCATTERING, masks["scattering"],
                 channels=4)


def test_block_size_does_not_change_the_luts(atmo, oracle, torch):  # noqa: F811
    atm = oracle.earth_atmosphere()
    shape = (64, 16, 4, 16, 8, 4, 16, 4)

    def scattering(count):
        b = atmo.Batch([atm] * count, [shape] * count, [2] * count)
        b.run()
        atmo.synchronize_stream()
        return [b.read(i, atmo.LUT_SCATTERING) for i in (0, count - 1)]

    alone = scattering(1)[0]
    for many in scattering(48):   # 768 blocks, of 128 threads
        np.testing.assert_array_equal(many, alone)


# Lines of two and more columns per thread beside several rows per block, rows
# of one and of three columns per thread.
@pytest.mark.parametrize("tw,mus,nu", [
    (127, 7, 7), (200, 10, 3), (97, 16, 8), (258, 32, 8), (129, 40, 8), (257, 51, 13),
    (400, 8, 3)])
def test_line_columns_vs_oracle(atmo, oracle, torch, tw, mus, nu):  # noqa: F811
    test_single_scattering_vs_oracle(atmo, oracle, torch, tw, mus, nu)
