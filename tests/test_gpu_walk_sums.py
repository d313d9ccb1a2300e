"""The plain walk's sums, body by body, at the edges of its warps and blocks:
every body's acceleration against float64 sums where (almost) every leaf is
met, the merge form's tasks against the pairs that overlap, and at theta 0.5
the last warp's bodies and the 99th percentile against the oracle's walk.

Bounds, u = 2^-24, S the float64 sum of the terms' magnitudes.  A term: offset
1 u, its square and the sum with the softening 5 u, the reciprocal square root
2.5 u + 4 u (2 ulp), its cube 3 of these + 2 u, mass and offset 3 u: 25 u (40 u
in the precision form, whose offset has two more roundings).  A sum of k terms
in FP32: 8 sqrt(k) u (the probabilistic bound, 8 standard deviations).  At
theta 1e-3 a node is accepted where its half side is below theta d; its bodies
lie within 2 sqrt(3) half sides of the centre of mass, so the quadrupole and
all beyond it are below 3 (2 sqrt(3) theta)^2 = 36 theta^2 of the term."""
import numpy as np
import pytest

from gravity_gb300 import BarnesHut, abi

from .helpers import bounds_of, make_pair, plummer_case
from .test_gpu_walk_plain import _walk

pytestmark = pytest.mark.gpu

U = 2.0**-24
SOFT = 1e-4
# capacities at the edges of the ranges with 4, 8 and 32 bodies per warp, live
# bodies at the edges of a warp and of a block (four warps)
EDGES = [(4096, 5), (4096, 17), (4096, 4096), (8192, 7), (8192, 33), (8192, 8191), (8193, 2), (8193, 31), (8193, 33),
         (8193, 129), (8193, 8193)]


def _state(capacity, live):
    b = plummer_case(capacity, seed=capacity)
    alive = np.sort(np.random.default_rng(3).permutation(capacity)[:live])
    b["pos_mass"][np.setdiff1d(np.arange(capacity), alive), 3] = 0.0
    return b, alive


def _direct(x, m, soft):
    """float64 accelerations and sums of the terms' magnitudes."""
    a, s = np.zeros((len(x), 3)), np.zeros(len(x))
    for i in range(0, len(x), 256):
        r = x[None, :, :] - x[i:i + 256, None, :]
        d2 = np.sum(r * r, axis=2)
        w = m[None, :] * (d2 + soft) ** -1.5
        a[i:i + 256] = np.sum(w[:, :, None] * r, axis=1)
        s[i:i + 256] = np.sum(w * np.sqrt(d2), axis=1)
    return a, s


def _evaluate(sim, p):
    a = sim.evaluate_walk(p).astype(np.float64)
    assert sim.read_stats().error_word == 0
    return a


@pytest.mark.parametrize("capacity, live", EDGES)
@pytest.mark.parametrize("theta", [0.0, 1e-3])
@pytest.mark.parametrize("form", ["fp32", "precision", "merge"])
def test_every_body_sums_every_leaf(gbh_lib, capacity, live, theta, form):
    b, alive = _state(capacity, live)
    soft = float(np.float32(SOFT))
    m = b["pos_mass"][alive, 3].astype(np.float64)
    x = b["pos_mass"][:, :3].astype(np.float64)
    radius = 0.6 * live ** (-1 / 3)
    sim = BarnesHut(capacity, bounds_of(b), abi.units(G=1.0))
    if form == "merge":  # some overlaps: every body the same radius
        b["vel_density"][:, 3] = 1.0
        sim.upload_bodies(b)
        sim.init()
        blc = float(sim.read_sim_values().body_length_constant)
        b["vel_density"][alive, 3] = m * (blc / radius) ** 3
    sim.upload_bodies(b)
    sim.init()
    if form == "precision":  # positions between the FP32 numbers
        x = x * (1.0 + np.random.default_rng(4).uniform(-0.4, 0.4, x.shape) * 2 * U)
        sim.write_positions_fp64(x)
    a = _evaluate(sim, abi.step_params(
        theta=theta, softening=SOFT, mode=abi.MODE_MERGE if form == "merge" else abi.MODE_NEITHER,
        precision=abi.PRECISION_COMPENSATED if form == "precision" else abi.PRECISION_FP32))[alive]
    ref, s = _direct(x[alive], m, soft)
    bound = ((40 if form == "precision" else 25) + 8 * np.sqrt(live)) * U + 36 * theta * theta
    worst = np.max(np.abs(a - ref) / s[:, None])
    assert worst <= bound, (worst, bound)
    if form == "merge" and theta == 0.0:
        # radii by powf (a few ulp), distances in FP32: pairs whose overlap is
        # within 1e-5 of the distance may go either way
        sure, maybe = set(), set()
        for i in range(live):
            d = np.sqrt(np.sum((x[alive[i + 1:]] - x[alive[i]]) ** 2, axis=1))
            for j in np.nonzero(d < 2 * radius * (1 + 1e-5))[0]:
                pair = (int(alive[i]), int(alive[i + 1 + j]))
                maybe.add(pair)
                if d[j] < 2 * radius * (1 - 1e-5):
                    sure.add(pair)
        tasks = [tuple(sorted(map(int, t))) for t in sim.read_merge_tasks()]
        assert len(tasks) == len(set(tasks))
        assert sure <= set(tasks) <= maybe
    sim.close()


@pytest.mark.parametrize("capacity, live", EDGES)
@pytest.mark.parametrize("mode", [abi.MODE_NEITHER, abi.MODE_MERGE])
def test_last_warp_and_tail_match_oracle(gbh_lib, oracle_mod, capacity, live, mode):
    b, alive = _state(capacity, live)
    g, o = make_pair(oracle_mod, BarnesHut, b, bounds_of(b))
    p = abi.step_params(theta=0.5, softening=SOFT, mode=mode, flags=abi.FLAG_STORE_ACCEL)
    ag, ao = _walk(g, o, p)
    terms = o.read_stats().interactions / live
    _, s = _direct(b["pos_mass"][alive, :3].astype(np.float64), b["pos_mass"][alive, 3].astype(np.float64), SOFT)
    e = np.zeros(capacity)
    e[alive] = np.max(np.abs(ag[alive].astype(np.float64) - ao[alive]), axis=1) / s
    # two FP32 sums of the same terms
    bound = 2 * (25 + 8 * np.sqrt(terms)) * U
    assert np.percentile(e[alive], 99) <= bound
    per_warp = 4 if capacity <= 4096 else 8 if capacity <= 8192 else 32
    last = g.read_index()[(live - 1) // per_warp * per_warp:live]
    assert np.max(e[last]) <= bound


@pytest.mark.parametrize("capacity", [4096, 8193])
def test_infinite_positions_leave_the_other_components(gbh_lib, oracle_mod, capacity):
    # a body at x = inf pulls along x only, by a sum that is not a number
    b = plummer_case(capacity, seed=3)
    far = [7, 900]
    b["pos_mass"][far, 0] = np.inf
    g, o = make_pair(oracle_mod, BarnesHut, b, bounds_of(b))
    ag, ao = _walk(g, o, abi.step_params(theta=0.5, softening=SOFT, flags=abi.FLAG_STORE_ACCEL))
    near = np.setdiff1d(np.arange(capacity), far)
    assert np.isfinite(ao[near][:, 1:]).all() and np.isfinite(ag[near][:, 1:]).all()
    _, s = _direct(b["pos_mass"][near, :3].astype(np.float64), b["pos_mass"][near, 3].astype(np.float64), SOFT)
    terms = o.read_stats().interactions / capacity
    e = np.max(np.abs(ag[near][:, 1:].astype(np.float64) - ao[near][:, 1:]), axis=1) / s
    assert np.percentile(e, 99) <= 2 * (25 + 8 * np.sqrt(terms)) * U
