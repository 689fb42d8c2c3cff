"""Tunings at the limits of what the lines in shared memory allow, for shapes
of every multiple-scattering kernel."""
import pytest


# Lines of W columns: rows x 51 samples of 64 bytes + 2 x group x rows x W x 16
# bytes, at most 48 KB.
@pytest.mark.parametrize("mus,nu,rows,most", [(32, 8, 1, 5), (16, 8, 2, 5), (8, 4, 4, 8),
                                              (40, 8, 1, 4), (65, 4, 1, 5), (64, 16, 1, 1)])
def test_multiple_scattering_limits(atmo, mus, nu, rows, most):
    shape = (64, 16, 4, 16, mus, nu, 16, 4)
    for group in range(1, 10):
        tuning = atmo.Tuning(rows, group, 0, 0)
        if group <= most:
            atmo.set_tuning(shape, tuning)
            assert atmo.get_tuning(shape).multiple_group == group
        else:
            with pytest.raises(atmo.AtmoError) as e:
                atmo.set_tuning(shape, tuning)
            assert e.value.status == atmo.INVALID_ARG
    atmo.set_tuning(shape, None)
