"""The plain walk at thetas from the exact sum upwards, on a tree that is both
wide and as tall as trees get, against the oracle's per-body walk: the same
interactions, and a stack that holds them (batches of opened nodes, then the
depth-first descent)."""
import numpy as np
import pytest

from gravity_gb300 import BarnesHut, abi

from .helpers import bounds_of, make_pair, rel_err
from .test_gpu_group_saturation import _corner_state
from .test_gpu_walk_plain import _walk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("theta", [-0.5, 0.0, 1e-30, 1e-18, 1e-9, 1e-4, 2e-3, 0.05])
@pytest.mark.parametrize("mode", [abi.MODE_NEITHER, abi.MODE_MERGE])
def test_small_thetas_match_oracle(gbh_lib, oracle_mod, theta, mode):
    # 19 key levels of 64 bodies per split towards a corner, 4,000 bodies in it
    b = _corner_state(19, 64)
    corner = np.repeat(b[-1:], 4000)
    b = np.concatenate([b, corner])
    b["pos_mass"][:, 3] = 1.0 / len(b)
    b["vel_density"][:, 3] = 1e30  # radii too small for tasks outside the corner
    g, o = make_pair(oracle_mod, BarnesHut, b, bounds_of(b))
    ag, ao = _walk(g, o, abi.step_params(theta=theta, softening=1e-4, mode=mode, flags=abi.FLAG_STORE_ACCEL))
    sg, so = g.read_stats(), o.read_stats()
    assert sg.tree_height == so.tree_height and sg.tree_height > 60
    assert sg.max_stack <= 289
    # nodes exactly at the threshold may fall either way (rsqrtf against 1/sqrtf)
    assert abs(int(sg.interactions) - int(so.interactions)) <= (1e-4 * so.interactions if theta > 0.0 else 0)
    if theta <= 0.0:
        assert sg.interactions == len(b) * (len(b) - 1)
    assert np.median(rel_err(ag, ao)) < 1e-5
