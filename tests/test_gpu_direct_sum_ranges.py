"""The FP64 direct sum's inverse cube over its whole range (the estimate with
its series, and the plain formula outside), with empty bodies, coinciding
bodies and no softening, against numpy in extended precision."""
import numpy as np
import pytest

from gravity_gb300 import BarnesHut, abi

from .helpers import bounds_of, plummer_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-18, 1e-39, 1e18])
@pytest.mark.parametrize("soft", [0.0, 1e-4])
@pytest.mark.parametrize("n", [2, 129, 3000])
def test_direct_sum_ranges(gbh_lib, n, scale, soft):
    b = plummer_case(n, seed=n)
    b["pos_mass"][:, :3] *= np.float32(scale)
    if n > 2:
        b["pos_mass"][5, :3] = b["pos_mass"][4, :3]  # coincide
        b["pos_mass"][7, 3] = 0.0  # empty
    g = BarnesHut(n, bounds_of(b), abi.units(G=1.0))
    g.upload_bodies(b)
    g.init()
    pick = np.unique(np.linspace(0, n - 1, 40).astype(np.uint32))
    eps2 = float(np.float32(soft))
    got = g.direct_sum(abi.step_params(softening=eps2), pick)
    p = b["pos_mass"].astype(np.longdouble)
    for k, i in enumerate(pick):
        r = p[:, :3] - p[i, :3]
        rr = (r * r).sum(1)
        use = (rr > 0) & (p[:, 3] != 0)
        term = p[use, 3:4] * r[use] * ((rr[use] + eps2) ** np.longdouble(-1.5))[:, None]
        want, size = term.sum(0), np.abs(term).sum(0)
        # seven roundings per term (2^-53 each) and one per addition, most of
        # which act on partial sums: 16 + n of them bound the error
        assert np.all(np.abs(got[k] - want) <= (16 + n) * 2.0**-53 * size + 1e-300)
