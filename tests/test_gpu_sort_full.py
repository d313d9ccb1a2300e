"""The radix sort of completely filled capacities at the top of each range that
chooses a tile size, and of one pair more than a tile: the stable sort's
permutation, bit for bit."""
import pytest

from .test_gpu_sort_tiles import test_sort_is_the_stable_sort as check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capacity, live", [(4096, 4096), (4097, 1025), (200000, 200000), (200001, 2049),
                                            (500000, 500000)])
@pytest.mark.parametrize("lattice", [False, True])
def test_sort_of_full_capacities(gbh_lib, capacity, live, lattice):
    check(gbh_lib, capacity, live, lattice)
