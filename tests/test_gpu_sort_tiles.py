"""The radix sort at the edges of its tiles and of the ranges of capacities that
choose a tile size: the permutation of a stable sort, bit for bit.  And the
compaction of one tile's capacity by one block, bit for bit the oracle's.
"""
import numpy as np
import pytest

from gravity_gb300 import BarnesHut, abi, ic

from .helpers import bounds_of, make_pair, plummer_case

pytestmark = pytest.mark.gpu


# capacity, live bodies: partial and full tiles of 1,024, 2,048 and 4,096 pairs,
# one pair, none beyond the first tile
@pytest.mark.parametrize("capacity, live", [(2, 1), (33, 33), (1024, 1024), (1025, 1025), (4096, 4095),
                                            (4097, 4097), (8192, 8192), (8192, 0), (8193, 8193), (200000, 199681), (200001, 200001),
                                            (500000, 2048), (500001, 500001), (500001, 4097), (1867776, 1867776),
                                            (1867777, 1867777), (2490368, 2490368), (2490368, 8193), (2490369, 2490369)])
@pytest.mark.parametrize("lattice", [False, True])
def test_sort_is_the_stable_sort(gbh_lib, capacity, live, lattice):
    b = plummer_case(capacity, seed=5)
    if lattice:  # few different digits, many equal keys
        k = np.arange(capacity)
        b["pos_mass"][:, 0] = k * 7919 % 13
        b["pos_mass"][:, 1] = k * 104729 % 4
        b["pos_mass"][:, 2] = k % 2
    dead = np.random.default_rng(2).permutation(capacity)[live:]
    b["pos_mass"][dead, 3] = 0.0
    sim = BarnesHut(capacity, ic.exact_bounds(b) if live > 1 else np.array([-1, -1, -1, 1, 1, 1], np.float32),
                    abi.units(G=1.0))
    sim.upload_bodies(b)
    sim.init()
    p = abi.step_params(bounds=abi.BOUNDS_DYNAMIC)
    sim.reset_values(p)
    sim.partition_dead_bodies(p)
    keys, idx = sim.read_morton()[:live].copy(), sim.read_index()[:live].copy()
    sim.radix_sort()
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(sim.read_morton()[:live], keys[order])
    assert np.array_equal(sim.read_index()[:live], idx[order])
    sim.close()


@pytest.mark.parametrize("dynamic", [True, False])
@pytest.mark.parametrize("n, dead, nans, outliers", [(3, 0.0, 0, 0), (64, 0.97, 0, 0), (257, 0.5, 1, 2), (2047, 0.1, 3, 5),
                                                     (2048, 0.5, 3, 5), (2049, 0.5, 3, 5)])
def test_prepare_of_one_tile(gbh_lib, oracle_mod, n, dead, nans, outliers, dynamic):
    b = plummer_case(n, seed=n, dead_frac=dead, nan_count=nans, outliers=outliers)
    g, o = make_pair(oracle_mod, BarnesHut, b, bounds_of(b))
    p = abi.step_params(bounds=abi.BOUNDS_DYNAMIC if dynamic else abi.BOUNDS_STATIC)
    for x in (g, o):
        x.stage_reset(p)
        x.stage_prepare(p)
    sg, so = g.read_sim_values(), o.read_sim_values()
    assert sg.num_bodies == so.num_bodies
    for k in range(3):
        assert np.float32(sg.bounds_min[k]).tobytes() == np.float32(so.bounds_min[k]).tobytes()
        assert np.float32(sg.bounds_max[k]).tobytes() == np.float32(so.bounds_max[k]).tobytes()
    assert np.array_equal(g.read_index(), o.read_index())
    live = sg.num_bodies
    assert np.array_equal(g.read_morton()[:live], o.read_morton()[:live])
    assert np.array_equal(g.read_bodies().view(np.uint32), o.read_bodies().view(np.uint32))
