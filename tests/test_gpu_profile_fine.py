"""Pressure profiles on either side of the number of own bins (six) from which the
slots of a warp add their windows one by one instead of merged."""
import pytest

from tests.test_gpu_profile_bins import test_profiles_against_the_oracle as against_the_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nb,walled", [(3001, 60, False), (3001, 90, False), (3001, 130, False),
                                         (3017, 2000, False), (2000, 400, True)])
def test_fine_bins(built, n, nb, walled):
    against_the_oracle(built, n, nb, walled)
