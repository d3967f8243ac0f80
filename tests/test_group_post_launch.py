"""How many launches a step of an e_iso group in block storage makes (on the
fake runtime): one that serves its own sources and receivers, or a second one
for them where the group fills the device many times over."""
import pytest

from fake_device import fake  # noqa: F401
from seismod_b200 import api
from seismod_b200 import workloads as W


@pytest.mark.parametrize("precision,shots,per_step", [("bfp16", 40, 1), ("bfp16", 48, 2), ("fp32", 48, 1)])
def test_launches_per_step(fake, precision, shots, per_step):
    # 84 slabs per shot; four handles; the limit is 96 slabs per SM
    p = W.cfg2(nx=200, nz=130, npml=9, nsteps=8, nshots=shots, nrec=20, seed=4)
    assert (4 * shots * 84 > 96 * 148) == (shots == 48)
    with fake.device():
        devs = [api.eiso_device(p, precision)[0] for _ in range(4)]
        api.group_run(devs, 1)
        fake.clear()
        api.group_run(devs, 3)
        names = [l[0] for l in fake.launches()]
        for d in devs:
            d.close()
    assert len(names) == 3 * per_step
    assert sum("post" in n for n in names) == 3 * (per_step - 1)
