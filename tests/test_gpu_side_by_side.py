"""atmo_precompute runs passes side by side, atmo_precompute_noalloc the same
passes in a chain: every repetition gives the same LUTs bit for bit."""
import pytest

from test_zz_no_alloc import identical, run, torch  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,combined", [((150, 37, 13, 46, 19, 5, 40, 12), False),
                                            ((33, 9, 5, 14, 5, 3, 17, 5), True)])
def test_repetitions_equal_the_chain(atmo, oracle, torch, shape, combined):  # noqa: F811
    earth = oracle.earth_atmosphere()
    chain = run(atmo, torch, "atmo_precompute_noalloc", earth, shape, 5, combined)
    for _ in range(20):
        identical(chain, run(atmo, torch, "atmo_precompute", earth, shape, 5, combined), combined)
