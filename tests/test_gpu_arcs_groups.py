"""Scattering density by arcs: groups of 4 and of 8 nu nodes at the edges of
the ranges that take them."""
import pytest

from test_gpu_arcs import test_sizes_vs_gpu_oracle as check_size
from test_gpu_parity import torch  # noqa: F401

pytestmark = pytest.mark.gpu


# (R, MU, MU_S, NU, IW): the smallest LUT of the arcs and one below; groups of
# 4 with 1 to 4 nodes in the last; groups of 8 with 5 nodes, 8, and 13 to 16.
@pytest.mark.parametrize("r,mu,mus,nu,iw", [
    (12, 64, 16, 5, 16), (12, 62, 16, 5, 16), (12, 64, 16, 9, 16), (16, 64, 24, 10, 16),
    (16, 64, 24, 12, 64), (16, 64, 17, 5, 16), (16, 64, 17, 8, 16), (16, 64, 17, 13, 64),
    (16, 64, 17, 16, 16), (16, 64, 16, 13, 16)])
def test_groups_vs_gpu_oracle(atmo, oracle, torch, r, mu, mus, nu, iw):  # noqa: F811
    check_size(atmo, oracle, torch, r, mu, mus, nu, iw)
