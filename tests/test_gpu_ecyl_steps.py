"""e_cyl_iso steps beside the oracle where the launches' own bookkeeping and the
vector cells' quotients have to give what the plain form gives."""
import numpy as np
import pytest

import harness as H
from oracle import oracle as O
from seismod_b200 import api
from seismod_b200 import workloads as W

pytestmark = pytest.mark.gpu

FIELDS = ("vr", "vt", "vz", "trr", "ttt", "tzz", "trz", "trt", "ttz")


def _pair(nx, nz, npml, n, precision="fp64", nrec=2):
    p = W.ecyl_case(nx=nx, nz=nz, npml=npml, nsteps=40, nrec=nrec, n=n, seed=11 + nx + nz, dx=1.3, dz=0.9)
    s = H.ecyl_setup(p)
    o = O.ECyl(p.nx, p.nz, p.np_used, p.n, p.dx, p.dz, s["dt"], s["mats"], s["coef"])
    dev, _ = api.ecyl_device(p, precision)
    return p, s, o, dev


@pytest.mark.parametrize("n", [0, 1, 2])
def test_fp64_signs_of_zero(n):
    """A state of zeros of both signs and a few values: the same bits as the
    oracle, a quotient of -0 being -0."""
    p, s, o, dev = _pair(24, 45, 6, n)
    dev.set_sources([], [], np.zeros((1, 1)), [])
    rng = np.random.default_rng(n)
    for f in FIELDS:
        v = np.where(rng.random(dev.shape) < 0.7, -0.0, 0.0)
        some = rng.random(dev.shape) < 0.1
        v[some] = rng.standard_normal(int(some.sum()))
        dev.set_field(f, v)
        o.set(f, v)
    dev.run(1)
    o.velocity()
    o.stress()
    for f in FIELDS:
        got, ref = np.ascontiguousarray(dev.get_field(f)), np.ascontiguousarray(o.get(f))
        assert np.signbit(ref[ref == 0]).any()
        np.testing.assert_array_equal(got.view(np.uint64), ref.view(np.uint64), err_msg=f)
    dev.close()
