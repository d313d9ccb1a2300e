"""gbh_stats.frontier_saturated: the group walks whose candidate stack filled
up, against a restatement of the walk's rounds on the GPU's own tree.

The walks here open every internal node (theta 0, or a band below every node),
so the restatement needs no arithmetic: rounds of up to 32 candidates from the
top of the stack, starting from the group's start list; a round whose opened
nodes do not fit lists them instead."""
import os

import numpy as np
import pytest

from gravity_gb300 import BarnesHut, abi, ic

from .test_gpu_group_walk import _groups

pytestmark = pytest.mark.gpu

STACK = {abi.MAC_GROUP: 768, abi.MAC_LEARNED: 640}  # entries per walk
WEIGHTS = os.path.join(os.path.dirname(ic.__file__), "mac_weights", "diverse.npy")


def _corner_state(levels, per):
    """At every split of the way to a corner `per` bodies on the far side: a walk
    from outside opens a full subtree per level before it goes down."""
    rng = np.random.default_rng(11)
    pos = []
    for level in range(1, levels + 1):
        side = 0.5**level
        for axis in range(3):
            lo, hi = np.full(3, 1 - 2 * side), np.ones(3)
            lo[:axis] = 1 - side
            hi[axis] = 1 - side
            pos.append(rng.uniform(lo, hi, (per, 3)))
    pos = np.concatenate(pos + [[[0.0] * 3, [1.0] * 3]]).astype(np.float32)
    b = np.zeros(len(pos), abi.BODY_DTYPE)
    b["pos_mass"][:, :3] = pos
    b["pos_mass"][:, 3] = 1.0 / len(pos)
    b["vel_density"][:, 3] = 1.0
    return b


def _walk_all(internal, n, stack_entries):
    """(walks that saturate, interactions) when every node is opened."""
    kids = {i + n: (int(internal[i]["child_a"]), int(internal[i]["child_b"])) for i in range(n - 1)}
    parent = {c: i for i, pair in kids.items() for c in pair}
    # node of the group that begins at a slot: the highest of at most 96 bodies
    count = lambda k: 1 if k < n else int(internal[k - n]["bodies_contained"])
    saturated = interactions = 0
    for first, bodies in _groups(internal, n, n):
        node = first
        while count(node) < bodies:
            node = parent[node]
        path = []
        while node != n:
            a, c = kids[parent[node]]
            path.append(c if a == node else a)
            node = parent[node]
        # 63 nodes at most in a start list; deeper groups start from the root
        stack = path + list(range(first, first + bodies)) if len(path) <= 62 else [n]
        full, listed = False, 0
        while stack:
            pop = stack[-32:]
            del stack[-32:]
            opened = [k for k in pop if k >= n]
            if len(stack) + 2 * len(opened) > stack_entries:
                full = True
                listed += len(pop)
                continue
            listed += len(pop) - len(opened)
            for k in opened:
                stack.extend(kids[k])
        saturated += full
        interactions += listed * bodies
    return saturated, interactions


@pytest.mark.parametrize("levels, per, mac", [(12, 64, abi.MAC_GROUP), (12, 64, abi.MAC_LEARNED),
                                              (14, 32, abi.MAC_LEARNED), (14, 32, abi.MAC_GROUP)])
def test_saturated_walks_are_counted(gbh_lib, levels, per, mac):
    b = _corner_state(levels, per)
    n = len(b)
    sim = BarnesHut(n, ic.exact_bounds(b), abi.units(G=1.0))
    sim.upload_bodies(b)
    sim.init()
    if mac == abi.MAC_LEARNED:
        sim.mac_set_weights(np.load(WEIGHTS))
        sim.mac_set_band(1e-9, 1e-8)
    p = abi.step_params(theta=0.0, softening=1e-4, mac=mac)
    sim.evaluate_walk(p)
    want, interactions = _walk_all(sim.read_internal_nodes(), n, STACK[mac])
    st = sim.read_stats()
    assert st.error_word == 0
    assert (want > 0) == (per == 64 or mac == abi.MAC_LEARNED)
    assert st.frontier_saturated == want
    assert st.interactions == interactions
    # the count is of the last step alone
    sim.evaluate_walk(abi.step_params(theta=2.0, softening=1e-4, mac=abi.MAC_GROUP))
    assert sim.read_stats().frontier_saturated == 0


@pytest.mark.parametrize("mac", [abi.MAC_GROUP, abi.MAC_LEARNED])
def test_no_walk_of_a_large_state_saturates(gbh_lib, mac):
    b = ic.plummer_uniform(2097152, seed=3)
    sim = BarnesHut(len(b), ic.exact_bounds(b), abi.units(G=1.0))
    sim.upload_bodies(b)
    sim.init()
    sim.mac_set_weights(np.load(WEIGHTS))
    sim.step(abi.step_params(dt=1e-3, theta=0.5, softening=2.5e-5, mac=mac, mac_tolerance=-2.35), count=2)
    st = sim.read_stats()
    assert st.error_word == 0 and st.interactions > 0
    assert st.frontier_saturated == 0
