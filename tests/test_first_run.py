"""What the first run of a fresh handle allocates (on the fake runtime).  A
cudaMalloc on a device with gigabytes in use has taken tens of milliseconds, so
a handle like one that was closed before makes few of its own: the source and
receiver tables come from the device cache, and lists that only grouped steps
read are uploaded by them."""
import ctypes as C

from fake_device import fake  # noqa: F401
from seismod_b200 import api
from seismod_b200 import workloads as W


def _mallocs(fake, make, first):
    fake.lib.sm_pool_set_limit(0, C.c_size_t(1 << 30))   # keep closed handles' blocks
    try:
        for _ in range(2):
            dev = make()
            fake.clear()
            first(dev)
            n = fake.lib.fake_mallocs()
            dev.close()
        return n
    finally:
        fake.lib.sm_pool_set_limit(0, C.c_size_t(0))


def test_a3d_first_run(fake):
    p = W.cfg1(n=24, npml=6, nsteps=40, seed=3, rec_stride=6, nrec_side=4)
    with fake.device():
        make = lambda: api.a3d_device(p, "fp32")[0]  # noqa: E731
        assert _mallocs(fake, make, lambda d: d.run(2)) == 2                      # samples, slots
        assert _mallocs(fake, make, lambda d: api.a3d_group_run([d], 2)) == 4     # ... and two lists


def test_eiso_first_run(fake):
    p = W.cfg2(nx=40, nz=36, nsteps=20, nshots=2, nrec=8)
    with fake.device():
        make = lambda: api.eiso_device(p, "fp32")[0]  # noqa: E731
        # sources, receivers, their firsts, samples, slots
        assert _mallocs(fake, make, lambda d: d.run(2)) == 6
