"""The fill's shared-reciprocal division and its body groups, bit for bit
against the oracle: masses and coordinates over the whole FP32 range (zeros,
subnormals and overflowing sums among them), coinciding bodies (the tallest
trees) and sizes at the edges of a group's words."""
import numpy as np
import pytest

from gravity_gb300 import BarnesHut, abi

from .helpers import bounds_of, make_pair, plummer_case

pytestmark = pytest.mark.gpu


def _fill_both(oracle_mod, b):
    bounds = bounds_of(b) if len(b) > 1 else np.array([-1, -1, -1, 1, 1, 1], np.float32)
    g, o = make_pair(oracle_mod, BarnesHut, b, bounds)
    p = abi.step_params()
    for x in (g, o):
        x.stage_reset(p)
        x.stage_prepare(p)
        x.stage_sort()
        x.stage_build()
        x.stage_fill()
    n = len(b)
    for a, c in ((g.read_leaf_nodes()[:n], o.read_leaf_nodes()[:n]),
                 (g.read_internal_nodes()[: max(n - 1, 1)], o.read_internal_nodes()[: max(n - 1, 1)])):
        for f in ("com_mass", "aabb"):
            u, v = a[f], c[f]
            same = (u.view(np.uint32) == v.view(np.uint32)) | (np.isnan(u) & np.isnan(v))
            assert same.all(), f
        for f in ("child_a", "child_b", "node_depth", "bodies_contained", "ready_children", "parent_id"):
            assert np.array_equal(a[f], c[f]), f


@pytest.mark.parametrize("mass_exp,pos_exp", [((-3, 3), (-3, 3)), ((-37, 37), (-30, 30)), ((-44, -36), (-44, -30)),
                                              ((-18, 18), (-24, 24)), ((30, 38), (0, 5))])
def test_fill_divisions_bit_exact(gbh_lib, oracle_mod, mass_exp, pos_exp):
    n = 5000
    rng = np.random.default_rng(7)
    b = plummer_case(n, seed=5)
    b["pos_mass"][:, 3] = np.maximum(10.0 ** rng.uniform(*mass_exp, n), 1e-45)
    b["pos_mass"][:, :3] = rng.choice([-1.0, 1.0], (n, 3)) * 10.0 ** rng.uniform(*pos_exp, (n, 3))
    b["pos_mass"][::17, 2] = 0.0
    b["pos_mass"][::31, 1] = -0.0
    _fill_both(oracle_mod, b)


@pytest.mark.parametrize("n", [1, 2, 32, 33, 64, 65, 95, 96, 97, 129, 2049, 65537, 140001])
def test_fill_group_edges_bit_exact(gbh_lib, oracle_mod, n):
    _fill_both(oracle_mod, plummer_case(n, seed=n))


@pytest.mark.parametrize("n", [130, 4100, 70001])
def test_fill_of_coinciding_bodies(gbh_lib, oracle_mod, n):
    b = plummer_case(n, seed=2)
    k = np.arange(n)
    # half in one point, the rest on a line of halving distances
    line = (0.5 ** (1 + k % 20)).astype(np.float32)
    b["pos_mass"][:, :3] = np.where((k % 2 == 0)[:, None], 0.0, line[:, None])
    _fill_both(oracle_mod, b)


@pytest.mark.parametrize("clusters", [3, 30, 400, 1300])
def test_fill_of_long_chains(gbh_lib, oracle_mod, clusters):
    # points of 97 coinciding bodies, each with bodies at halving distances:
    # some 15 nodes above the groups per 112 bodies, more than a block has
    # threads; the largest has a capacity whose fill climbs
    rng = np.random.default_rng(1)
    cells = rng.choice(16**3, clusters, replace=False)
    corner = np.stack([cells % 16, cells // 16 % 16, cells // 256], 1) / 16.0
    k = np.arange(6, 21)
    per = np.concatenate([np.zeros(97), 0.5**k])
    pos = (corner[:, None, :] + per[None, :, None]).reshape(-1, 3)
    pos = np.concatenate([pos, [[0.0] * 3, [1.0] * 3]]).astype(np.float32)
    b = plummer_case(len(pos), seed=1)
    b["pos_mass"][:, :3] = pos
    _fill_both(oracle_mod, b)
