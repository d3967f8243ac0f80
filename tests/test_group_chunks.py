"""How long the chunks of a grouped a_iso_3d launch are (on the fake runtime):
short ones only while the whole group leaves the device unfilled, and the
caller's own where one is set.  CTAs of a launch: the sum over the problems of
tiles times chunks."""
import pytest

from fake_device import fake  # noqa: F401
from seismod_b200 import api
from seismod_b200 import workloads as W

SMS = 148


def _ctas(fake, sides, precision, chunks=None):
    with fake.device():
        devs, models = [], {}
        for k, n in enumerate(sides):
            p = models[n] = models.get(n) or W.cfg1(n=n, npml=8, nsteps=8, seed=3, rec_stride=8, nrec_side=2)
            devs.append(api.a3d_device(p, precision)[0])
            if chunks and chunks[k]:
                devs[-1].set_chunk(chunks[k])
        fake.clear()
        api.a3d_group_run(devs, 2)
        got = [l[1] for l in fake.launches() if "group_step" in l[0]]
        for d in devs:
            d.close()
    assert len(got) == 2 and got[0] == got[1]
    return got[0]


def _tiles(n, precision):
    ty = 32 if precision == "bfp16" else 16
    return -(-(n + 16) // 32) * -(-(n + 16) // ty)


@pytest.mark.parametrize("precision", ["fp32", "bfp16", "fp64"])
def test_a_group_that_fills_the_device_takes_long_chunks(fake, precision):
    """At least 16 planes once chunks of 16 give every place on the device its
    three CTAs; alone these grids take 4 to 8 planes."""
    got = _ctas(fake, [96] * 16, precision)
    assert got <= 16 * _tiles(96, precision) * -(-(96 + 16) // 16)


@pytest.mark.parametrize("precision", ["fp32", "bfp16", "fp64"])
def test_a_small_group_spreads_over_the_device(fake, precision):
    for n, count in ((48, 2),) if precision == "fp64" else ((48, 2), (64, 2), (96, 1)):
        got = _ctas(fake, [n] * count, precision)
        assert got > 1.5 * count * _tiles(n, precision) * -(-(n + 16) // 16)
        assert got <= count * _tiles(n, precision) * -(-(n + 16) // (8 if precision == "fp64" else 4))


def test_the_callers_chunk_stands(fake):
    t = _tiles(96, "fp32")
    assert _ctas(fake, [96, 96], "fp32", chunks=[7, 28]) == t * 16 + t * 4
    # ... for the handle it is set on only
    free = _ctas(fake, [96, 96], "fp32") // 2
    assert _ctas(fake, [96, 96], "fp32", chunks=[0, 28]) == free + t * 4
