"""The precision form's Morton keys against the quantisation formula in numpy
FP64 (integers: exact): random positions, positions on and next to cell edges
(where the fixed-point form hands over to the divisions) and at the box's
faces."""
import numpy as np
import pytest

from gravity_gb300 import BarnesHut, abi

from .helpers import plummer_case

pytestmark = pytest.mark.gpu


def _expand(v):
    x = v.astype(np.uint64) & np.uint64(0x1FFFFF)
    for s, m in ((32, 0x1F00000000FFFF), (16, 0x1F0000FF0000FF), (8, 0x100F00F00F00F00F), (4, 0x10C30C30C30C30C3),
                 (2, 0x1249249249249249)):
        x = (x | (x << np.uint64(s))) & np.uint64(m)
    return x


@pytest.mark.parametrize("lo,hi", [((-1, -1, -1), (1, 1, 1)), ((-3.7, 0.1, 100.0), (5.3, 0.30000001, 100.5)),
                                   ((0, 0, 0), (2097151, 2097151, 1e-3))])
def test_precision_keys_match_formula(gbh_lib, lo, hi):
    n = 30000
    rng = np.random.default_rng(3)
    lo32, hi32 = np.array(lo, np.float32), np.array(hi, np.float32)
    lo64, hi64 = lo32.astype(np.float64), hi32.astype(np.float64)
    ext = np.maximum(hi64 - lo64, 1e-9)
    x = lo64 + rng.uniform(0.0, 1.0, (n, 3)) * ext
    # cell edges and their neighbours in FP64
    edge = lo64 + rng.integers(0, 2097152, (n // 2, 3)) / 2097151.0 * ext
    x[: n // 2] = edge
    x[: n // 6] = np.nextafter(edge[: n // 6], np.inf)
    x[n // 6 : n // 3] = np.nextafter(edge[n // 6 : n // 3], -np.inf)
    x[-20:-10], x[-10:] = lo64, hi64
    b = plummer_case(n, seed=1)
    b["pos_mass"][:, :3] = x
    g = BarnesHut(n, np.concatenate([lo32, hi32]), abi.units(G=1.0))
    g.upload_bodies(b)
    g.init()
    g.write_positions_fp64(x)
    p = abi.step_params(bounds=abi.BOUNDS_STATIC, precision=abi.PRECISION_COMPENSATED)
    g.stage_reset(p)
    g.stage_prepare(p)
    pos = np.minimum(np.maximum(x, lo64), hi64)
    q = np.clip(np.floor((pos - lo64) / ext * 2097151.0), 0, 2097151).astype(np.uint64)
    want = (_expand(q[:, 0]) << np.uint64(2)) | (_expand(q[:, 1]) << np.uint64(1)) | _expand(q[:, 2])
    assert np.array_equal(g.read_index()[:n], np.arange(n))
    assert np.array_equal(g.read_morton()[:n], want)
