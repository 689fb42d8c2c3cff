"""The autotuner's choice where tunings come to the same launch, and the LUTs
of the line kernel's tunings."""
import numpy as np
import pytest

from test_gpu_parity import torch  # noqa: F401

pytestmark = pytest.mark.gpu


def shape(mus, nu):
    return (64, 16, 4, 16, mus, nu, 16, 4)


# Nodes (no multiple-scattering tuning) and a block of one row of single
# scattering; nodes and up to three rows.
@pytest.mark.parametrize("mus,nu,single_rows", [(16, 8, (1,)), (10, 4, (1, 2, 4))])
def test_no_choice_where_the_launch_is_the_same(atmo, oracle, torch, mus, nu,  # noqa: F811
                                                single_rows):
    for _ in range(2):
        t = atmo.autotune(oracle.earth_atmosphere(), shape(mus, nu), instances=2)
        assert (t.multiple_rows, t.multiple_group) == (1, 1)
        assert t.single_rows in single_rows and t.single_group >= 1
        assert t.multiple_ms > 0 and t.single_ms > 0
    atmo.set_tuning(shape(mus, nu), None)


# Shapes whose multiple scattering keeps lines: several rows per block, and one
# row of more than 256 columns.
@pytest.mark.parametrize("mus,nu,tunings", [
    (19, 3, [(1, 1, 1, 1), (4, 3, 2, 4), (2, 6, 1, 2)]), (19, 4, [(2, 8, 2, 1), (1, 3, 1, 8)]),
    (65, 4, [(1, 1, 1, 1), (1, 5, 1, 2), (1, 3, 0, 0)])])
def test_lines_do_not_depend_on_the_tuning(atmo, oracle, torch, mus, nu, tunings):  # noqa: F811
    kinds = (atmo.LUT_TRANSMITTANCE, atmo.LUT_SCATTERING, atmo.LUT_IRRADIANCE)

    def luts():
        b = atmo.Batch([oracle.earth_atmosphere()], [shape(mus, nu)], 3)
        b.run()
        atmo.synchronize_stream()
        return [b.read(0, k) for k in kinds]

    ref = luts()
    for t in tunings:
        atmo.set_tuning(shape(mus, nu), atmo.Tuning(*t))
        for x, y in zip(luts(), ref):
            np.testing.assert_array_equal(x, y)
    t = atmo.autotune(oracle.earth_atmosphere(), shape(mus, nu), instances=2)
    assert t.multiple_rows >= 1 and t.multiple_group >= 1
    for x, y in zip(luts(), ref):
        np.testing.assert_array_equal(x, y)
    atmo.set_tuning(shape(mus, nu), None)
