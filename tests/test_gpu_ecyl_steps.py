"""What the e_cyl_iso launches keep track of besides the fields: stress records
that the next step's launch samples, or one of their own at the end of a run;
sources that the cell's own CTA adds.  Steps taken in several runs, beside
the oracle, with sources that share a cell and sources on the axis, in the
layers and on both sides of the vector cells' edges.

FP64: fields and the records of single fields bit for bit; div and curl 1e-12
(the same operations in another order)."""
import numpy as np
import pytest

import harness as H
from oracle import oracle as O
from seismod_b200 import _lib as L
from seismod_b200 import api
from seismod_b200 import workloads as W

pytestmark = pytest.mark.gpu

FIELDS = ("vr", "vt", "vz", "trr", "ttt", "tzz", "trz", "trt", "ttz")
RUNS = (1, 1, 7, 2, 14)


def _sources(nx, nz, npml, rng):
    """(i, j, type, samples)"""
    v = 2                                       # cells per vector in FP64
    ja, jb = -(-npml // v) * v, (nz + npml - 1) // v * v
    fr, ft, fz, bulk = 9, 10, 11, 6
    cells = [(8, 20, fz), (8, 20, fr), (8, 20, fz), (8, 21, ft),        # one cell, one vector
             (0, 25, fz), (0, 25, fr), (nx + 2, 30, fz), (8, npml - 2, bulk),
             (8, ja, fz), (8, ja - 1, fr), (8, jb - 1, fz), (8, jb, bulk),
             (1, 22, fz), (nx - 2, 20, bulk), (nx - 1, 20, ft), (nx - 1, nz + 2 * npml - 2, fz)]
    return [(i, j, t, rng.standard_normal(5 if k == 1 else 30)) for k, (i, j, t) in enumerate(cells)]


@pytest.mark.parametrize("n", [0, 1, 2])
def test_runs_in_pieces_follow_the_oracle(n):
    nx, nz, npml = 24, 45, 6
    p = W.ecyl_case(nx=nx, nz=nz, npml=npml, nsteps=40, nrec=2, n=n, seed=17, dx=1.3, dz=0.9)
    s = H.ecyl_setup(p)
    o = O.ECyl(p.nx, p.nz, p.np_used, p.n, p.dx, p.dz, s["dt"], s["mats"], s["coef"])
    dev, _ = api.ecyl_device(p, "fp64")
    nz2, dt = dev.shape[1], s["dt"]
    rng = np.random.default_rng(n)
    src = _sources(nx, nz, npml, rng)
    kurk = (5 * nz2 + 20, rng.standard_normal(20))
    fct = np.zeros((len(src) + 1, 30))
    for k, q in enumerate(src):
        fct[k, :len(q[3])] = q[3]
    fct[-1, :20] = kurk[1]
    dev.set_sources([i * nz2 + j for i, j, _, _ in src] + [kurk[0]],
                    [t for _, _, t, _ in src] + [api.ECYL_SRC["kurkjian"]], fct, [len(q[3]) for q in src] + [20])
    comps = FIELDS + ("div", "curl")
    rec = [(i * nz2 + j, c, k % 3 * 2 * dt, (1, 3)[k % 2] * dt)
           for k, (i, j, c) in enumerate((i, j, c) for i, j in ((8, 20), (0, 25), (nx - 2, 21)) for c in comps)]
    steps = sum(RUNS)
    code = dict(api.ECYL_FIELD, div=L.SM_DIV, curl=L.SM_CURL)
    dev.set_receivers([r[0] for r in rec], [code[r[1]] for r in rec], [r[2] for r in rec], [r[3] for r in rec], steps)
    ref = [[] for _ in rec]
    for it in range(steps):
        o.velocity()
        for i, j, t, w in src:
            if it < len(w):
                o.force(i * nz2 + j, t, w[it])
        o.stress()
        if it < 20:
            o.kurkjian(kurk[0], kurk[1][it])
        for k, (q, c, t0, rdt) in enumerate(rec):
            if O.sample(it, dt, t0, rdt):
                ref[k].append(o.probe(c, q))

    def check():
        for got, want, r in zip(dev.traces(), ref, rec):
            if r[1] in ("div", "curl"):
                np.testing.assert_allclose(got, want, rtol=1e-12, atol=1e-12 * np.abs(want).max(), err_msg=r[1])
            else:
                np.testing.assert_array_equal(got, want, err_msg=r[1])

    for k in RUNS:
        dev.run(k)
    check()
    for f in FIELDS:
        np.testing.assert_array_equal(dev.get_field(f), o.get(f), err_msg=f)
    dev.reset()
    dev.run(steps)
    check()
    dev.close()
