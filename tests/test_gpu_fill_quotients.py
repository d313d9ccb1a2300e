"""Centres of mass whose quotients leave the normal range, bit for bit against
the oracle's divisions: ties between subnormal numbers, and quotients beside
the largest number."""
import numpy as np
import pytest

from gravity_gb300 import abi

from .test_gpu_fill_ranges import _fill_both

pytestmark = pytest.mark.gpu


def _two_bodies(masses, coordinates):
    b = np.zeros(2, abi.BODY_DTYPE)
    b["pos_mass"][:, :3] = np.array(coordinates, np.float32)[:, None]
    b["pos_mass"][:, 3] = np.array(masses, np.float32)
    b["vel_density"][:, 3] = 1.0
    return b


@pytest.mark.parametrize("k", [684, 686, 1000, 1368])
def test_fill_subnormal_ties(gbh_lib, oracle_mod, k):
    # masses 2^57 and 5 2^57: the weighted mean of the coordinates (units of
    # 2^-149) is k + 1/2, a tie that rounds to the even k
    u = [6 * k + 3 - 5 * k, k]
    _fill_both(oracle_mod, _two_bodies([2.0**57, 5 * 2.0**57], [x * 2.0**-149 for x in u]))


# masses in units of 2^-75: the rounded sum of the weighted coordinates times
# the rounded reciprocal passes the largest number, the quotient does not (the
# first five) or does (the last two)
@pytest.mark.parametrize("left, right", [(12046372, 15956846), (14199468, 15383124), (16397254, 15675830),
                                         (16322553, 13809597), (16609301, 13688467), (9487999, 8609530),
                                         (12320029, 11605540)])
def test_fill_quotients_beside_the_largest_number(gbh_lib, oracle_mod, left, right):
    largest = float(np.finfo(np.float32).max)
    _fill_both(oracle_mod, _two_bodies([left * 2.0**-75, right * 2.0**-75], [largest, largest]))
