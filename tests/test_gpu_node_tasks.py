"""Multiple scattering's packed tasks at the edges of its kernels' ranges: few
lanes used with wide rows, three nu nodes (every column clamped at both ends),
even and odd node counts of two columns per lane."""
import pytest

from test_gpu_nodes import test_column_counts_vs_oracle as check_columns
from test_gpu_parity import torch  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mus,nu", [(17, 8), (17, 7), (11, 5), (32, 3), (5, 3), (32, 9),
                                    (39, 4), (40, 4), (40, 2), (48, 6), (64, 3)])
def test_packed_tasks_vs_oracle(atmo, oracle, torch, mus, nu):  # noqa: F811
    check_columns(atmo, oracle, torch, mus, nu)
