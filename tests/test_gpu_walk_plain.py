"""The plain walk's box classification against the oracle's per-body walk: the
same interactions for every warp shape, for parameters outside the range its
margins cover, for positions that are not finite, and for a walk that opens
everything (the stack's depth-first mode)."""
import numpy as np
import pytest

from gravity_gb300 import BarnesHut, abi

from .helpers import bounds_of, make_pair, plummer_case, rel_err

pytestmark = pytest.mark.gpu


def _walk(g, o, p):
    for x in (g, o):
        x.stage_reset(p)
        x.stage_prepare(p)
        x.stage_sort()
        x.stage_build()
        x.stage_fill()
        x.stage_walk(p)
    assert g.read_stats().error_word == 0
    return g.read_accel()[:, :3], o.read_accel()[:, :3]


@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 127, 129, 4097])
@pytest.mark.parametrize("theta,soft", [(0.5, 1e-4), (0.5, 0.0), (0.0, 1e-4), (5e-4, 1e-6), (3.0, 1e-2), (2e3, 1e-4)])
def test_walk_forms_match_oracle(gbh_lib, oracle_mod, n, theta, soft):
    b = plummer_case(n, seed=n)
    g, o = make_pair(oracle_mod, BarnesHut, b, bounds_of(b))
    ag, ao = _walk(g, o, abi.step_params(theta=theta, softening=soft, flags=abi.FLAG_STORE_ACCEL))
    # a node exactly at the threshold may fall either way (rsqrtf against
    # 1/sqrtf): 1e-4 of the interactions, as in the parity tests
    ig, io = g.read_stats().interactions, o.read_stats().interactions
    assert abs(int(ig) - int(io)) <= 1e-4 * io
    if theta == 0.0:
        assert ig == n * (n - 1)  # every leaf of every other body
    assert np.median(rel_err(ag, ao)) < 1e-5


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_walk_with_positions_not_finite(gbh_lib, oracle_mod, bad):
    b = plummer_case(2000, seed=3)
    b["pos_mass"][[7, 900], 0] = bad
    g, o = make_pair(oracle_mod, BarnesHut, b, bounds_of(b))
    ag, ao = _walk(g, o, abi.step_params(theta=0.5, softening=1e-4, flags=abi.FLAG_STORE_ACCEL))
    ig, io = g.read_stats().interactions, o.read_stats().interactions
    assert abs(int(ig) - int(io)) <= 1e-4 * io
    assert np.array_equal(np.isnan(ag), np.isnan(ao))


def test_walk_of_a_tall_tree(gbh_lib, oracle_mod):
    # bodies halving their distance to a corner (one tree level each) and
    # coinciding bodies (levels of the index tie-break)
    k = np.arange(1, 21)
    line = np.repeat((0.5 ** k)[:, None], 3, axis=1)
    pos = np.concatenate([line, np.zeros((300, 3)), np.ones((4, 3))]).astype(np.float32)
    b = plummer_case(len(pos), seed=1)
    b["pos_mass"][:, :3] = pos
    g, o = make_pair(oracle_mod, BarnesHut, b, bounds_of(b))
    for theta in (0.0, 0.5):
        ag, ao = _walk(g, o, abi.step_params(theta=theta, softening=1e-3, flags=abi.FLAG_STORE_ACCEL))
        assert abs(int(g.read_stats().interactions) - int(o.read_stats().interactions)) <= 2
        far = np.linalg.norm(ao, axis=1) > 0
        assert np.median(rel_err(ag[far], ao[far])) < 1e-5


# capacities at the edges of the ranges with 4, 8 and 32 bodies per warp, live
# bodies at the edges of a warp and of a block
@pytest.mark.parametrize("capacity, live", [(4096, 4096), (4096, 5), (4097, 4096), (8192, 8191), (8192, 33), (8193, 31),
                                            (8193, 32), (8193, 33), (8193, 129), (8193, 8193)])
@pytest.mark.parametrize("theta", [0.0, 0.5])
def test_walk_bodies_per_warp(gbh_lib, oracle_mod, capacity, live, theta):
    b = plummer_case(capacity, seed=capacity)
    alive = np.sort(np.random.default_rng(3).permutation(capacity)[:live])
    dead = np.setdiff1d(np.arange(capacity), alive)
    b["pos_mass"][dead, 3] = 0.0
    g, o = make_pair(oracle_mod, BarnesHut, b, bounds_of(b))
    ag, ao = _walk(g, o, abi.step_params(theta=theta, softening=1e-4, flags=abi.FLAG_STORE_ACCEL))
    ig, io = g.read_stats().interactions, o.read_stats().interactions
    assert abs(int(ig) - int(io)) <= 1e-4 * io
    if theta == 0.0:
        assert ig == live * (live - 1)
    assert np.median(rel_err(ag[alive], ao[alive])) < 1e-5


# the collision walk's result does not depend on the bodies per warp (4, 8, 16
# or 32 by capacity): the same live bodies in capacities of all four ranges
@pytest.mark.parametrize("live", [1, 5, 33, 129, 8191])
def test_collision_walk_bodies_per_warp(gbh_lib, live):
    rng = np.random.default_rng(live)
    pos = rng.uniform(-1, 1, (live, 3)).astype(np.float32)
    results = []
    for capacity in (8192, 8193, 16385, 32769):
        b = np.zeros(capacity, abi.BODY_DTYPE)
        b["pos_mass"][:live, :3] = pos
        b["pos_mass"][:live, 3] = 1.0 / live
        b["vel_density"][:live, :3] = 1.0 - 2.0 * pos[:, ::-1]
        b["vel_density"][:live, 3] = 2.0  # radii of some percent of the box: contacts
        sim = BarnesHut(capacity, np.array([-1, -1, -1, 1, 1, 1], np.float32), abi.units(G=1.0))
        sim.upload_bodies(b)
        sim.init()
        p = abi.step_params(dt=1e-3, theta=0.7, softening=1e-4, mode=abi.MODE_COLLISION)
        for _ in range(2):
            sim.step(p)
        results.append(sim.read_bodies()[:live].view(np.uint32).copy())
        assert sim.read_stats().error_word == 0
        sim.close()
    for r in results[1:]:
        assert np.array_equal(r, results[0])
