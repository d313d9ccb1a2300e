"""The step's graph with the group walk, whose start lists are a branch beside
the fill: bit for bit the stages run one after the other, also where the graph
is captured while streamed copies are under way."""
import numpy as np
import pytest

from gravity_gb300 import BarnesHut, abi, ic

pytestmark = pytest.mark.gpu

STAGES = ("stage_prepare", "stage_sort", "stage_build", "stage_fill")


@pytest.mark.parametrize("n", [40, 3000, 140001])
def test_group_step_graph_equals_stages_and_streamed(gbh_lib, n):
    torch = pytest.importorskip("torch")
    calls = 5
    states = [ic.plummer(n, seed=50 + k) for k in range(calls + 1)]
    bounds = ic.exact_bounds(states[0])
    p = abi.step_params(theta=0.8, softening=1e-4, bounds=abi.BOUNDS_DYNAMIC, mac=abi.MAC_GROUP)
    sims = [BarnesHut(n, bounds, abi.units(G=1.0)) for _ in range(3)]
    for x in sims:
        x.upload_bodies(states[0])
        x.init()
    graph, eager, streamed = sims

    def pinned():
        t = torch.empty(n * abi.BODY_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True)
        return t.numpy().view(abi.BODY_DTYPE)

    nxt, out = pinned(), pinned()
    want = []
    for k in range(calls):
        for x in (graph, eager):
            x.upload_bodies(states[k])
        graph.step(p)
        eager.stage_reset(p)
        for s in STAGES:
            getattr(eager, s)(*((p,) if s == "stage_prepare" else ()))
        eager.stage_walk(p)
        eager.stage_merge(p)
        eager.stage_swap()
        want.append(graph.read_bodies())
        assert np.array_equal(eager.read_bodies().view(np.uint32), want[k].view(np.uint32)), k
    for k in range(calls):
        nxt[:] = states[k + 1]
        streamed.step_streamed(p, nxt, out)
        if k:
            assert np.array_equal(out.view(np.uint32), want[k - 1].view(np.uint32)), k
    streamed.step_streamed_finish(out)
    assert np.array_equal(out.view(np.uint32), want[-1].view(np.uint32))
