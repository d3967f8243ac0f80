"""e_iso block storage: sources and receivers that have a launch of their own
(batches and groups that fill the device many times over) against those that
the step's warps serve, bit for bit.  Receivers in every column of the
sources' row: more than a block's 128 threads per shot, in the source patches
and across their edges."""
import numpy as np
import pytest

from seismod_b200 import api
from seismod_b200 import workloads as W

pytestmark = pytest.mark.gpu

STEPS = 45


def _problem(nshots):
    # 84 slabs of 8 rows by 60 cells per shot
    return W.cfg2(nx=200, nz=130, npml=9, nsteps=STEPS, nshots=nshots, nrec=200, seed=4)


def _launches_per_step(dev, run):
    dev.kernel_stats(reset=True)
    run()
    return dev.kernel_stats(reset=True)[2] / STEPS


@pytest.mark.parametrize("graph", [0, 16])
def test_large_batch_equals_single_shots(graph):
    p = _problem(176)                    # 14784 slabs: above 96 per SM
    dev, n = api.eiso_device(p, "bfp16")
    dev.set_graph(graph)
    assert _launches_per_step(dev, lambda: dev.run(STEPS)) == 2
    for s in (0, 1, 87, 174, 175):
        one, _ = api.eiso_device(p, "bfp16", [s])
        assert _launches_per_step(one, lambda: one.run(STEPS)) == 1
        np.testing.assert_array_equal(dev.traces_array(s), one.traces_array(0))
        assert np.abs(one.traces_array(0)).max() > 0
        one.close()
    dev.close()


def test_large_group_equals_single_runs():
    p = _problem(180)
    parts = [list(range(k, 180, 4)) for k in range(4)]     # 45 shots each: alone, below the limit
    devs = [api.eiso_device(p, "bfp16", part)[0] for part in parts]
    per_step = _launches_per_step(devs[0], lambda: api.group_run(devs, STEPS))
    assert per_step == 2
    for d, part in zip(devs, parts):
        one, _ = api.eiso_device(p, "bfp16", part)
        assert _launches_per_step(one, lambda: one.run(STEPS)) == 1
        for s in range(len(part)):
            np.testing.assert_array_equal(d.traces_array(s), one.traces_array(s))
        one.close()
        d.close()
