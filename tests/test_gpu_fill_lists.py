"""The fill above the body groups where a subtree has more nodes than a block
has threads, bit for bit against the oracle: clumps of coinciding bodies, each
the end of chains of bodies at halving distances, one tree level each."""
import numpy as np
import pytest

from .helpers import plummer_case
from .test_gpu_fill_ranges import _fill_both

pytestmark = pytest.mark.gpu


def _chains(clumps, bodies, axes):
    rng = np.random.default_rng(1)
    cells = rng.choice(16**3, clumps, replace=False)
    corner = np.stack([cells % 16, cells // 16 % 16, cells // 256], 1) / 16.0
    reach = 0.5 ** np.arange(6, 21)
    chain = reach[:, None] * np.ones(3) if axes == 1 else (reach[:, None, None] * np.eye(3)).reshape(-1, 3)
    per = np.concatenate([np.zeros((bodies, 3)), chain])
    pos = (corner[:, None, :] + per[None]).reshape(-1, 3)
    pos = np.concatenate([pos, [[-1.0] * 3, [2.0] * 3]]).astype(np.float32)
    b = plummer_case(len(pos), seed=1)
    b["pos_mass"][:, :3] = pos
    return b


# nodes of a subtree (of at most 4,096 bodies) above its groups: 49, then from
# 292 to 565, where a list of more than 128 is climbed from its lowest nodes; the
# last has 673 nodes above the subtrees
@pytest.mark.parametrize("clumps, bodies, axes", [(8, 97, 1), (36, 97, 1), (28, 97, 3), (60, 97, 1), (200, 97, 1),
                                                  (1100, 97, 1), (100, 97, 3), (800, 97, 3), (300, 400, 1),
                                                  (31, 4097, 3)])
def test_fill_lists_bit_exact(gbh_lib, oracle_mod, clumps, bodies, axes):
    _fill_both(oracle_mod, _chains(clumps, bodies, axes))
