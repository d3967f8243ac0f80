"""Per-kernel timing of steps that are two launches (e_iso's tile
configurations, whose sources and receivers have a launch of their own): events
around each update launch, inside replayed graphs too.  Every update is timed
once, the durations sum to less than the steps they sit in take, and timing
changes no result."""
import numpy as np
import pytest
import torch

from seismod_b200 import api
from seismod_b200 import workloads as W

pytestmark = pytest.mark.gpu

TILE = 6


@pytest.mark.parametrize("graph", [0, 16])
def test_tile_steps(graph):
    p = W.cfg2(nx=600, nz=300, nsteps=300, nshots=16, nrec=16)
    n = 3 * 16 + 5   # whole graphs and single steps
    devs = [api.eiso_device(p, "fp32")[0] for _ in range(2)]
    for d in devs:
        d.set_config(TILE)
        d.set_graph(graph)
        d.kernel_stats(reset=True)
    plain, timed = devs
    plain.run(n)
    timed.set_timing(True)
    timed.run(n)
    ms, updates, launches = timed.kernel_stats(reset=True)
    assert updates == n and launches == 2 * n
    timed.set_timing(False)
    st = torch.cuda.ExternalStream(timed.stream())
    e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    timed.sync()
    e0.record(st)
    timed.run(n)
    e1.record(st)
    e1.synchronize()
    # the same steps untimed; events around a launch add a few microseconds to
    # it, here a few percent of its 100 or so
    assert 0 < ms < 1.2 * e0.elapsed_time(e1)
    plain.run(n)
    for s in (0, 15):
        np.testing.assert_array_equal(plain.traces_array(s), timed.traces_array(s))
        np.testing.assert_array_equal(plain.get_field("txx", s), timed.get_field("txx", s))
    for d in devs:
        d.close()
