"""The a_iso_3d block step, and sources and receivers served inside the steps,
at grid sizes where the blocks' lanes, rows and frames end: one lane column and
two, odd extents, a frame that covers the grid, no frame at all.

From a random state with sources and receivers on corners, edges and inside,
three steps: every field and trace bit for bit what the ring step gives for
several chunk lengths (the arithmetic is the same), FP64 within 1e-12 of the
oracle (three steps of about 30 roundings of 1.1e-16, with room for
cancellation).
"""
import numpy as np
import pytest

import harness as H  # noqa: F401  (path set-up)
from oracle import oracle as O
from seismod_b200 import api
from seismod_b200 import _lib as L

pytestmark = pytest.mark.gpu

FIELDS = ("p", "vx", "vy", "vz")
RING, BLOCK = 8, 9
# padded extents and frame width
GRIDS = [((3, 3, 3), 0), ((5, 4, 7), 1), ((6, 7, 29), 2), ((9, 8, 31), 3), ((7, 9, 61), 2), ((8, 10, 62), 3),
         ((12, 11, 64), 4), ((13, 37, 121), 5), ((40, 34, 66), 0)]


def _handles(grid, precision):
    shape, np_ = grid
    rng = np.random.default_rng(list(shape) + [np_])
    vp = 2000 + 1000 * rng.random(shape)
    rho = 1500 + 500 * rng.random(shape)
    d = (5.0, 4.0, 6.0)
    dt = 0.4 * 4.0 / (np.sqrt(3.0) * 3000.0)
    if np_:
        coef = api.a3d_cpml(np_, shape, d, dt, Rc=1e-3, f0=20.0)
    else:   # no frame: the coefficients' defaults everywhere
        coef = [np.full(shape[k // 3 % 3] - k // 9, 0.0 if k % 3 == 0 else 1.0) for k in range(18)]
    n = int(np.prod(shape))
    src = [0, n - 1, n // 2, n // 2, shape[2] - 1, n // 3]
    fct = 1e3 * rng.standard_normal((len(src), 6))
    length = [6, 2, 6, 6, 1, 6]
    rec = sorted({0, n - 1, n // 2, n // 3, shape[2] - 1, n - shape[2], shape[1] * shape[2]})
    recs = [(c, f) for c in rec for f in FIELDS]
    state = {f: (1e2 if f == "p" else 1e-4) * rng.standard_normal(shape) for f in FIELDS}

    def device():
        dev = api.A3DDevice(vp, rho, np_, d, dt, coef, precision)
        dev.set_sources(src, fct, length, 1.0)
        dev.set_receivers([c for c, _ in recs], [L.SM_COMP[f] for _, f in recs], [0.0] * len(recs),
                          [dt] * len(recs), 6)
        for f, v in state.items():
            dev.set_field(f, v)
        return dev

    def oracle():
        o = O.A3D(vp, rho, *d, dt, coef)
        for f, v in state.items():
            o.set(f, v)
        return o

    return device, oracle, (src, fct, length), recs


def _run(dev):
    dev.run(2)
    dev.run(1)
    out = [dev.get_field(f) for f in FIELDS] + [dev.traces_array()]
    dev.close()
    return out


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("grid", GRIDS)
def test_block_step_equals_the_ring_step(grid, precision):
    device, _, _, _ = _handles(grid, precision)
    out = []
    for config, chunk in ((RING, 0), (RING, 1), (RING, 3), (BLOCK, 0)):
        dev = device()
        dev.set_config(config)
        dev.set_chunk(chunk)
        out.append(_run(dev))
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("grid", GRIDS)
def test_block_step_against_the_oracle(grid):
    device, oracle, (src, fct, length), recs = _handles(grid, "fp64")
    dev, o = device(), oracle()
    dev.set_config(BLOCK)
    got = _run(dev)
    for it in range(3):
        o.velocity()
        o.pressure()
        for s, q in enumerate(src):
            if it < length[s]:
                o.add_source(q, fct[s, it])
        ref = np.array([o.probe(f, c) for c, f in recs])
        assert O.rel_l2(got[-1][:, it], ref) < 1e-12
    for f, a in zip(FIELDS, got):
        assert O.rel_l2(a, o.get(f)) < 1e-12, f
