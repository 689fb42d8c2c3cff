"""Multiple scattering by nodes where every column is clamped at both ends (two
nu nodes), and of two and three nodes of 16 columns."""
import pytest

from test_gpu_nodes import test_column_counts_vs_oracle as check_columns
from test_gpu_parity import torch  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mus,nu", [(16, 2), (32, 2), (64, 2), (16, 4), (16, 5), (16, 7),
                                    (11, 2), (2, 80)])
def test_clamped_columns_vs_oracle(atmo, oracle, torch, mus, nu):  # noqa: F811
    check_columns(atmo, oracle, torch, mus, nu)
