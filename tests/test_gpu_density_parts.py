"""Scattering density by lookups: the tasks of a block's last round split into
parts of the theta rows (order 2 at every size, order 3 of small LUTs)."""
import pytest

from parity import TOL_SCATTERING, check
from test_gpu_parity import gpu_precompute, torch  # noqa: F401

pytestmark = pytest.mark.gpu


# (R, MU, MU_S, NU): the last round's tasks (MU x ceil(NU / 4)) are 8 (8
# parts), 34 (4), 66 (2), 128 (2), 130 (unsplit), 300 - 256 (4), 516 - 512 (8),
# 256 (none), and 24 of 13 nodes (shared memory).
@pytest.mark.parametrize("r,mu,mus,nu", [
    (4, 8, 6, 3), (4, 34, 5, 4), (4, 66, 5, 2), (4, 128, 4, 3), (4, 130, 4, 3), (4, 150, 4, 8),
    (4, 258, 3, 5), (4, 64, 4, 16), (4, 6, 4, 13)])
def test_parts_vs_gpu_oracle(atmo, oracle, torch, r, mu, mus, nu):  # noqa: F811
    shape = (64, 16, r, mu, mus, nu, 16, 4)
    atm = oracle.earth_atmosphere()
    ref = oracle.gpu_precompute(atm, shape, 3, combined=True)
    scattering = gpu_precompute(atmo, torch, atm, shape, 3)[1]
    check("scattering", scattering, ref.scattering, TOL_SCATTERING, channels=4)
