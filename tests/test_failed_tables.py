"""What a failed allocation or a refused call leaves behind: a step must never
be given source or receiver tables that were not completed for it.  On the
fake runtime, where launches do nothing and allocations fail on request."""
import numpy as np
import pytest

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
