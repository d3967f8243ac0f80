"""The device-memory estimates, by which the request loop admits work, against
what handles hold after the calls that build every table (on the fake
runtime), with lists long enough that the estimates' slack does not cover them."""
import ctypes as C

import numpy as np
import pytest

from fake_device import fake  # noqa: F401
from seismod_b200 import _lib as L
from seismod_b200 import api
from seismod_b200 import serving
from seismod_b200 import workloads as W


def _estimate(fake, fn, *args):
    b = C.c_size_t()
    f = getattr(fake.lib, fn)
    f.restype, f.argtypes = serving._SIGS[fn]
    assert f(*args, C.byref(b)) == 0
    return b.value


@pytest.mark.parametrize("precision", ["fp32", "fp64", "bfp16"])
def test_eiso_many_shots(fake, precision):
    shots, nrec, steps = 3000, 80, 2
    p = W.cfg2(nx=24, nz=20, npml=4, nsteps=steps, nshots=1, nrec=nrec)
    with fake.device():
        live = fake.lib.fake_live_bytes()
        q = api.eiso_inputs(p)
        dev = api.EIsoDevice(q["nx"], q["nz"], q["npml"], q["h"], q["dt"], q["la"], q["mu"], q["l2m"],
                             q["b"], q["bm"], q["d"], q["dh"], q["dH"], precision, shots)
        idx, typ, fct, ln = q["src"][0]
        dev.set_sources(None, idx, typ, fct[:, :steps], [steps], q["src_scale"])
        dev.set_receivers(None, *q["rec"], steps)
        dev.autotune(1)
        dev.run(1)
        api.group_run([dev], 1)
        held = fake.lib.fake_live_bytes() - live
        dev.close()
    assert held <= _estimate(fake, "sm_eiso_device_bytes", p.nx, p.nz, p.npml, L.PRECISIONS[precision], shots,
                             nrec, steps)


@pytest.mark.parametrize("precision", ["fp32", "bfp16"])
def test_a3d_many_receivers(fake, precision):
    nrec, steps, npml = 1000000, 2, 4
    n = (60, 60, 60)
    vp = np.full(tuple(x - 2 * npml for x in n), 2000.0)
    coef = api.a3d_cpml(npml, n, (5.0, 5.0, 5.0), 1e-4, 2.0, 5000.0, 1e-3, 1.0, 1, 25.0)
    with fake.device():
        live = fake.lib.fake_live_bytes()
        dev = api.A3DDevice(vp, vp, npml, (5.0, 5.0, 5.0), 1e-4, coef, precision=precision, padded=False)
        at = np.arange(nrec) % int(np.prod(n))
        dev.set_receivers(at, np.full(nrec, 2), np.zeros(nrec), np.full(nrec, 1e-4), steps)
        dev.run(1)
        api.a3d_group_run([dev], 1)
        held = fake.lib.fake_live_bytes() - live
        dev.close()
    assert held <= _estimate(fake, "sm_a3d_device_bytes", *n, npml, L.PRECISIONS[precision], nrec, steps)
