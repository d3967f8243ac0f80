"""The e_iso warp step (lean bands and frame tasks, sources and receivers served
by their cells' warps) at grid sizes where its tasks end: no lean rectangle, one
cell of it, whole and partial bands and 30-lane columns, frames wider than a
task's 30 cells.

From a random state with sources and receivers in the corners, at the
rectangle's rim and inside, three steps: every field, split part and trace bit
for bit what the tile kernel with its separate source and receiver launches
gives (the arithmetic is the same), FP64 within 1e-12 of the oracle (the
relative rounding of three steps, about 30 operations of 1.1e-16 each, with
room for cancellation), grouped runs bit for bit as single ones.
"""
import math

import numpy as np
import pytest

import harness as H  # noqa: F401  (path set-up)
from oracle import oracle as O
from seismod_b200 import api
from seismod_b200 import _lib as L

pytestmark = pytest.mark.gpu

FIELDS = ("vx", "vz", "txx", "tzz", "txz")
TILE, WARP = 6, (17, 18)
# nx, nz, npml, shots
GRIDS = [(2, 2, 1, 1), (3, 3, 1, 1), (3, 40, 2, 2), (4, 62, 1, 1), (5, 63, 3, 5), (9, 124, 2, 1),
         (66, 5, 4, 3), (7, 70, 35, 1), (131, 33, 8, 2)]


def _device(grid, precision, seed=3):
    nx, nz, P, shots = grid
    rng = np.random.default_rng([seed, nx, nz])
    vp = 3000 + 1000 * rng.random((nx, nz))
    la, mu, l2m, b, bm, vpmax = O.eiso_materials(vp, vp / 1.7, 2000 + 400 * rng.random((nx, nz)))
    dt = 0.5 / (math.sqrt(2) * vpmax)
    prof = O.eiso_profiles(P, 1.0, vp)
    dev = api.EIsoDevice(nx, nz, P, 1.0, dt, la, mu, l2m, b, bm, *prof, precision, shots)
    orc = [O.EIso(nx, nz, P, 1.0, dt, la, mu, l2m, b, bm, *prof) for _ in range(shots)]
    inter = np.zeros((nx + 2 * P, nz + 2 * P), bool)
    inter[P:P + nx, P:P + nz] = True
    cells = [0, nz - 1, (nx - 1) * nz, nx * nz - 1, (nx // 2) * nz + nz // 2, (nx - 2) * nz + 1,
             min(1, nx - 1) * nz + min(1, nz - 1)]
    types = [L.SM_SRC[t] for t in ("bulk", "sx", "sz", "sxz", "bulk", "sxz", "bulk")]
    # two sources in one cell: their order is part of the result
    idx, typ = cells + [cells[4]], types + [L.SM_SRC["sx"]]
    for s in range(shots):
        for f in FIELDS:
            scale = 1e-3 if f.startswith("v") else 1e4
            tot, xp, zp = (scale * rng.standard_normal(inter.shape) for _ in range(3))
            for part, v in (("x", np.where(inter, 0, xp)), ("z", np.where(inter, 0, zp)),
                            ("total", np.where(inter, tot, 0))):
                dev.set_field(f, v, shot=s, part=part)
                orc[s].set(f, part, v)
        fct = 1e4 * rng.standard_normal((len(idx), 8))
        dev.set_sources(s, idx, typ, fct, [8, 2, 8, 1, 8, 8, 3, 8], dt)
        orc[s].src = (idx, typ, fct * dt, [8, 2, 8, 1, 8, 8, 3, 8])
    rec = [(c, f) for c in cells for f in FIELDS]
    comps = [L.SM_COMP[f] for _, f in rec]
    dev.set_receivers(None, [c for c, _ in rec], comps, [0.0] * len(rec), [dt] * len(rec), 8)
    return dev, orc, rec


def _state(dev):
    return [dev.get_field(f, shot=s, part=p) for s in range(dev.nshots) for f in FIELDS
            for p in ("total", "x", "z")] + [dev.traces_array(s) for s in range(dev.nshots)]


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("grid", GRIDS)
def test_warp_step_equals_the_tile_step(grid, precision):
    states = []
    for config in (TILE,) + WARP:
        dev, _, _ = _device(grid, precision)
        dev.set_config(config)
        dev.run(3)
        states.append(_state(dev))
        dev.close()
    for other in states[1:]:
        for a, b in zip(states[0], other):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("grid", GRIDS)
def test_warp_step_against_the_oracle(grid):
    dev, orc, rec = _device(grid, "fp64")
    dev.run(3)
    for s, o in enumerate(orc):
        idx, typ, val, length = o.src
        traces = dev.traces_array(s)
        for it in range(3):
            o.velocity()
            o.stress()
            for k, (i, t) in enumerate(zip(idx, typ)):
                if it < length[k]:
                    o.add_source(i, t, val[k, it])
            ref = np.array([o.probe(f, c) for c, f in rec])
            assert O.rel_l2(traces[:, it], ref) < 1e-12
        for f in FIELDS:
            for part in ("total", "x", "z"):
                a, b = dev.get_field(f, shot=s, part=part), o.get(f, part)
                assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b), (f, part)
    dev.close()


def test_grouped_warp_steps_equal_single_ones():
    single, grouped = [], []
    for grid in GRIDS:
        dev, _, _ = _device(grid, "fp32")
        dev.run(3)
        single.append(_state(dev))
        dev.close()
    devs = [_device(grid, "fp32")[0] for grid in GRIDS]
    api.group_run(devs, 3)
    for dev, ref in zip(devs, single):
        for a, b in zip(_state(dev), ref):
            np.testing.assert_array_equal(a, b)
        dev.close()
