"""What a failed allocation or a refused call leaves behind: a step must never
be given source or receiver tables that were not completed for it.  On the
fake runtime, where launches do nothing and allocations fail on request."""
import numpy as np
import pytest

from fake_device import fake  # noqa: F401
from seismod_b200 import _lib as L
from seismod_b200 import api
from seismod_b200 import workloads as W


def _a3d():
    p = W.cfg1(n=24, npml=6, nsteps=40, seed=3, rec_stride=6, nrec_side=4)
    return api.a3d_device(p, "fp32")[0]


def test_a3d_tables_are_built_again_after_a_failed_build(fake):
    """Configuration A, a run that fails in B for want of memory, A again: what
    the failed run left is not A's tables, so they are built anew, whichever
    of the allocations it was that failed."""
    with fake.device():
        for k in range(8):
            dev = _a3d()
            dev.set_config(9)
            dev.run(2)
            fake.clear()
            dev.run(2)
            assert fake.lib.fake_uploads() == 0          # the tables stand
            dev.set_config(8)
            fake.fail_malloc(k, 2)                       # (cached allocations are tried twice)
            try:
                dev.run(2)
                failed = False
            except L.SeismodError:
                failed = True
            fake.fail_malloc(0, 0)
            dev.set_config(9)
            fake.clear()
            dev.run(2)
            dev.close()
            assert fake.lib.fake_uploads() > 0, k
            if not failed:                               # every allocation has had its turn
                break
        assert 0 < k < 7


def test_a3d_refused_sources_and_receivers_leave_the_old_ones(fake):
    with fake.device():
        sizes = []
        for refuse in (False, True):
            dev = _a3d()
            dev.run(2)
            if refuse:
                n = int(np.prod(dev.shape))
                w = np.ones((3, 9))
                with pytest.raises(L.SeismodError):
                    dev.set_sources([1, 2, n], w, [9, 9, 9], 1.0)
                with pytest.raises(L.SeismodError):
                    dev.set_receivers([1, 2, n], [2, 2, 2], [0.0] * 3, [1e-3] * 3, 80)
            dev.set_config(8)                            # tables for other owners
            fake.clear()
            dev.run(2)
            sizes.append(fake.lib.fake_upload_bytes())
            dev.close()
        assert sizes[0] == sizes[1]


def _ecyl():
    p = W.ecyl_case(nx=12, nz=33, npml=7, nsteps=40, nrec=5, n=1, seed=5)
    return api.ecyl_device(p, "fp32")[0]


def _served(fake, dev):
    """Sources and records that the velocity and the stress launch of a step
    are given: mask and first table, number of records, tables, step count."""
    out = []
    for name in ("velocity", "stress"):
        fake.watch(name, 2)
        dev.run(2)
        v = fake.watched()
        out.append(dict(mask=v[0], first=v[1], nrec=v[5] >> 32, rec=v[6], table=v[7], nsteps=v[8], traces=v[9]))
    return out


def test_ecyl_failed_sources_and_records_leave_none(fake):
    with fake.device():
        for k in range(12):
            dev = _ecyl()
            n = int(np.prod(dev.shape))
            w = np.ones((3, 9))
            fake.fail_malloc(k, 1)
            failed = 0
            try:
                dev.set_sources([1, 40, n - 1], [9, 11, 12], w, [9, 9, 9])
            except L.SeismodError:
                failed = 1
                assert all(v["mask"] == 0 for v in _served(fake, dev))
            try:
                dev.set_receivers([1, 2], [L.SM_VZ, L.SM_TZZ], [0.0] * 2, [1e-3] * 2, 80)
            except L.SeismodError:
                failed = 1
                assert all(v["nrec"] == 0 for v in _served(fake, dev))
            fake.fail_malloc(0, 0)
            for v in _served(fake, dev):
                assert not v["mask"] or v["first"]
                assert not v["nrec"] or (v["rec"] and v["table"] and v["traces"])
            dev.close()
            if not failed:
                break
        assert 3 < k < 11


def test_ecyl_refused_sources_and_records_leave_the_old_ones(fake):
    with fake.device():
        dev = _ecyl()
        before = _served(fake, dev)
        assert before[0]["mask"] and before[1]["nrec"]
        n = int(np.prod(dev.shape))
        with pytest.raises(L.SeismodError):
            dev.set_sources([1, 2, n], [9, 11, 11], np.ones((3, 9)), [9, 9, 9])
        with pytest.raises(L.SeismodError):
            dev.set_receivers([1, 2, n], [L.SM_VZ] * 3, [0.0] * 3, [1e-3] * 3, 17)
        assert _served(fake, dev) == before
        dev.close()


@pytest.mark.parametrize("precision", ["fp32", "bfp16"])
def test_eiso_uploads_again_after_a_failure(fake, precision):
    """The first run fails for want of memory at each of its allocations in
    turn; the next one uploads everything a run without a failure uploads
    after that allocation, the traces' read-back included."""
    p = W.cfg2(nx=40, nz=36, nsteps=20, nshots=2, nrec=8)
    with fake.device():
        dev = api.eiso_device(p, precision)[0]
        fake.clear()
        dev.run(2)
        whole = fake.lib.fake_upload_bytes()
        dev.close()
        for k in range(24):
            dev = api.eiso_device(p, precision)[0]
            fake.clear()
            fake.fail_malloc(k, 2)
            try:
                dev.run(2)
                failed = False
            except L.SeismodError:
                failed = True
            fake.fail_malloc(0, 0)
            at_failure = fake.lib.fake_upload_bytes()
            dev.run(2)
            got = fake.lib.fake_upload_bytes()
            assert got >= whole, (k, at_failure, got, whole)
            dev.traces_array(0)
            dev.close()
            if not failed:
                break
        assert 6 < k < 23
