"""Which a_iso_3d grids take the block step by default (on the fake runtime)."""
import numpy as np
import pytest

from fake_device import fake  # noqa: F401
from seismod_b200 import api

BLOCK = 9


def _config(fake, n, precision):
    npml = 2
    m = tuple(x - 2 * npml for x in n)
    vp = np.full(m, 2000.0)
    coef = api.a3d_cpml(npml, n, (5.0, 5.0, 5.0), 1e-4, 2.0, 5000.0, 1e-3, 1.0, 1, 25.0)
    with fake.device():
        d = api.A3DDevice(vp, vp, npml, (5.0, 5.0, 5.0), 1e-4, coef, precision=precision, padded=False)
        c = d.get_config()[0]
        d.close()
    return c


@pytest.mark.parametrize("precision,n,block", [
    # rows of 31 and 32 cells: two warps of the block step, half of its lanes idle
    ("fp64", (400, 400, 32), False), ("fp64", (400, 400, 31), False), ("fp64", (350, 350, 32), True),
    ("fp64", (400, 400, 30), True), ("fp64", (400, 400, 33), True), ("fp64", (300, 260, 64), True),
    # FP32 keeps one limit
    ("fp32", (100, 100, 64), True), ("fp32", (130, 130, 32), True), ("fp16", (100, 100, 64), True),
    # beyond the sizes where the ring step overtakes it on full rows
    ("fp32", (100, 100, 90), False)])
def test_rows_that_waste_lanes_take_the_ring_earlier(fake, precision, n, block):
    assert (_config(fake, n, precision) == BLOCK) == block
