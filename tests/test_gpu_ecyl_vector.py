"""The e_cyl_iso launches' vector cells (16 bytes of consecutive z rows away
from the layers, the axis and the edges) beside their single cells, at grid
sizes where the split between the two falls on every remainder.

From a random state, four steps, every field: FP64 bit for bit with the
oracle, with values over the whole exponent range (zeros, and magnitudes too
small for the reciprocal quotients, which then take the division) in the
state; FP32 within 1e-5 of it (four steps of at most ten roundings of 6e-8
each, summed with cancellation: about 2e-6).
"""
import numpy as np
import pytest

import harness as H
from oracle import oracle as O
from seismod_b200 import api
from seismod_b200 import workloads as W

pytestmark = pytest.mark.gpu

FIELDS = ("vr", "vt", "vz", "trr", "ttt", "tzz", "trz", "trt", "ttz")
# nx, nz, npml, absorb: no vector column, one, a single vector row, every
# remainder of nz + npml by 2 and 4, more than one CTA of vectors per column,
# no layer (row 0 reads across columns)
GRIDS = [(2, 20, 5, 1), (3, 17, 5, 1), (6, 9, 4, 1), (9, 30, 1, 1), (9, 31, 3, 1), (12, 32, 6, 1),
         (12, 33, 7, 1), (5, 1030, 8, 1), (17, 50, 6, 0), (6, 8, 6, 0)]


def _state(shape, wide, seed):
    rng = np.random.default_rng(seed)
    out = {}
    for f in FIELDS:
        v = rng.standard_normal(shape)
        if wide:
            v *= 10.0 ** rng.choice([-300.0, -285.0, -150.0, -3.0, 0.0, 8.0], size=shape)
            v[rng.random(shape) < 0.1] = 0.0
        out[f] = v
    return out


def _four_steps(precision, grid, n, wide):
    nx, nz, npml, absorb = grid
    p = W.ecyl_case(nx=nx, nz=nz, npml=npml, nsteps=8, nrec=2, n=n, seed=7 + nx + nz, dx=1.3, dz=0.9,
                    absorb=absorb)
    s = H.ecyl_setup(p)
    o = O.ECyl(p.nx, p.nz, p.np_used, p.n, p.dx, p.dz, s["dt"], s["mats"], s["coef"])
    dev, _ = api.ecyl_device(p, precision)
    dev.set_sources([], [], np.zeros((1, 1)), [])
    for f, v in _state(dev.shape, wide, nz).items():
        dev.set_field(f, v)
        o.set(f, v if precision == "fp64" else v.astype(np.float32).astype(np.float64))
    dev.run(4)
    for _ in range(4):
        o.velocity()
        o.stress()
    got = {f: dev.get_field(f) for f in FIELDS}
    ref = {f: o.get(f) for f in FIELDS}
    dev.close()
    return got, ref


@pytest.mark.parametrize("n", [0, 1, 2])
@pytest.mark.parametrize("grid", GRIDS)
def test_fp64_vector_cells_bit_for_bit(grid, n):
    got, ref = _four_steps("fp64", grid, n, wide=True)
    for f in FIELDS:
        np.testing.assert_array_equal(got[f], ref[f], err_msg=f)


@pytest.mark.parametrize("n", [0, 1])
@pytest.mark.parametrize("grid", GRIDS)
def test_fp32_vector_cells(grid, n):
    got, ref = _four_steps("fp32", grid, n, wide=False)
    for f in FIELDS:
        assert O.rel_l2(got[f], ref[f]) < 1e-5, (f, O.rel_l2(got[f], ref[f]))
