"""The work that programs built on this framework have it do, as timed cases.

One pass is one shot (or one batch or group of shots) on handles that the
program keeps: reset the state, advance the time loop, read the traces back to
the host, as the drop-in programs and the request loop do it; with `snap` the
last vz field too, as their snapshot records do.  The kinds:

  eiso   e_iso, `shots` shots over one model in one handle
  group  several e_iso handles of different grids stepped together
  a3d    a_iso_3d
  ecyl   e_cyl_iso, azimuthal mode `n`

Grid sizes are the interior's; every grid gets an absorbing frame of `npml`
cells.  Sizes, frames, receiver layouts and step counts are those of
seismod_b200.workloads (the two-layer 400 x 400 shot, the 64-shot 1000 x 500
batch, the 256^3 and 512^3 cubes, the cylindrical 2000 x 4000 run, the request
stream) and of the tests; the largest runs take fewer steps than a whole shot,
every step being like the next.  Models are random layers with a smooth lateral
variation, sources Ricker wavelets strong from the first steps on.

exact() restates the three schemes in 64 bits with torch alone.
"""
import math

import numpy as np
import torch

from seismod_b200 import api
from seismod_b200 import workloads as W


def listed():
    return [
        # a test-sized shot: latency and launches are everything
        dict(name="eiso_96x80", kind="eiso", nx=96, nz=80, npml=8, shots=1, nrec=16, steps=300,
             precision="fp32", graph=0, snap=1),
        # the two-layer 400 x 400 shot, whole, launched as the drop-in program launches it
        dict(name="eiso_400sq", kind="eiso", nx=400, nz=400, npml=20, shots=1, nrec=64, steps=1500,
             precision="fp32", graph=0, snap=1),
        # one shot of the batch model, replayed as graphs: the plain form of a survey
        dict(name="eiso_1000x500", kind="eiso", nx=1000, nz=500, npml=20, shots=1, nrec=256,
             steps=1000, precision="fp32", graph=16),
        # the 64-shot survey batch in FP32 and in 16-bit block storage
        dict(name="eiso_1000x500_64", kind="eiso", nx=1000, nz=500, npml=20, shots=64, nrec=256,
             steps=200, precision="fp32", graph=16),
        dict(name="eiso_1000x500_64_b", kind="eiso", nx=1000, nz=500, npml=20, shots=64, nrec=256,
             steps=200, precision="bfp16", graph=16),
        # uneven requests advanced together, as the request loop groups them
        dict(name="eiso_group", kind="group", sides="203x203,377x377,612x612,865x865,431x298",
             npml=20, nrec=32, steps=400, precision="fp32"),
        # the smallest cube of the request stream
        dict(name="a3d_128", kind="a3d", nx=128, ny=128, nz=128, npml=16, nside=16, steps=300,
             precision="fp32", graph=16),
        # the 256^3 shot in FP32 and in block storage, and the 512^3 shot
        dict(name="a3d_256", kind="a3d", nx=256, ny=256, nz=256, npml=16, nside=128, steps=200,
             precision="fp32", graph=16),
        dict(name="a3d_256_b", kind="a3d", nx=256, ny=256, nz=256, npml=16, nside=128, steps=200,
             precision="bfp16", graph=16),
        dict(name="a3d_512", kind="a3d", nx=512, ny=512, nz=512, npml=16, nside=128, steps=40,
             precision="fp32", graph=16),
        # the cylindrical run (mode 1), and a ragged mode-0 one in the reference's FP64
        dict(name="ecyl_2000x4000", kind="ecyl", nx=2000, nz=4000, npml=20, n=1, nrec=64, steps=100,
             precision="fp32"),
        dict(name="ecyl_381x707_d", kind="ecyl", nx=381, nz=707, npml=12, n=0, nrec=24, steps=300,
             precision="fp64", snap=1),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another shot of the same kinds: any sizes between a test's and the
    largest run's, odd ones too, at most the largest listed case's work."""
    kind = rng.choice(["eiso", "eiso", "a3d", "a3d", "ecyl", "group"])
    if kind == "eiso":
        nx, nz, npml = _logint(rng, 64, 1100), _logint(rng, 64, 1100), rng.randint(8, 20)
        cells = (nx + 2 * npml) * (nz + 2 * npml)
        shots = min(_logint(rng, 1, 64), max(1, int(3.6e7 / cells)))
        steps = max(20, min(_logint(rng, 100, 1500), int(3.5e9 / (cells * shots))))
        return dict(kind=kind, nx=nx, nz=nz, npml=npml, shots=shots, nrec=_logint(rng, 8, 256),
                    steps=steps, precision=rng.choice(["fp32", "fp32", "fp64", "bfp16"]),
                    graph=rng.choice([0, 16]), snap=int(cells < 2e5))
    if kind == "group":
        sides = [(_logint(rng, 100, 900), _logint(rng, 100, 900)) for _ in range(rng.randint(2, 8))]
        return dict(kind=kind, sides=",".join("%dx%d" % s for s in sides), npml=20,
                    nrec=_logint(rng, 8, 64), steps=_logint(rng, 100, 500), precision="fp32")
    if kind == "a3d":
        npml = rng.randint(6, 16)
        while True:
            nx, ny, nz = (_logint(rng, 24, 512) for _ in range(3))
            cells = (nx + 2 * npml) * (ny + 2 * npml) * (nz + 2 * npml)
            if cells <= 1.0e8:
                break
        steps = max(20, min(_logint(rng, 50, 400), int(2.5e9 / cells)))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, npml=npml, nside=_logint(rng, 4, 64),
                    steps=steps, precision=rng.choice(["fp32", "fp32", "fp64", "bfp16"]),
                    graph=rng.choice([0, 16]))
    nx, nz, npml = _logint(rng, 60, 2000), _logint(rng, 80, 4000), rng.randint(8, 20)
    cells = (nx + npml) * (nz + 2 * npml)
    steps = max(20, min(_logint(rng, 100, 400), int(8.0e8 / cells)))
    return dict(kind=kind, nx=nx, nz=nz, npml=npml, n=rng.randint(0, 2), nrec=_logint(rng, 8, 64),
                steps=steps, precision=rng.choice(["fp32", "fp32", "fp64"]), snap=int(cells < 3e5))


# ----------------------------------------------------------------------------
# problems, from the seed alone
# ----------------------------------------------------------------------------

def _layers(rng, nz, vmin, vmax):
    nlay = int(rng.integers(4, 9))
    cuts = np.sort(rng.integers(1, max(nz - 1, 2), size=nlay - 1))
    return rng.uniform(vmin, vmax, size=nlay)[np.searchsorted(cuts, np.arange(nz), side="right")]


def _wave(rng, n):
    """A smooth factor near 1 along one axis."""
    return 1.0 + 0.02 * np.sin(np.arange(n) * (2 * np.pi / n) * rng.uniform(0.7, 3.0) + rng.uniform(0, 6))


def _eiso_problem(nx, nz, npml, shots, nrec, steps, rng):
    h = 1.0
    vp = _wave(rng, nx)[:, None] * _layers(rng, nz, 2000.0, 5000.0)[None, :]
    vs = vp / rng.uniform(1.7, 1.9)
    rho = W.gardner(vp)
    dt_ms = 0.5 * h / (math.sqrt(2.0) * float(vp.max())) * 1e3
    f = 0.05 / (dt_ms * 1e-3)                      # 20 steps a period: strong at once
    zs = float(rng.integers(3, 9))
    sx = [float(round((k + rng.uniform(0.3, 0.7)) * (nx - 1) / shots)) * h for k in range(shots)]
    src = [[("Bulk", 1.0, f, x, zs)] for x in sx]
    rec = [("Vz" if k % 4 else "Vx", round(k * (nx - 1) / max(nrec - 1, 1)) * h, zs, 0.0, dt_ms)
           for k in range(nrec)]
    return W.EIsoProblem(vp, vs, rho, h, npml, dt_ms, W.steps_duration(steps, dt_ms), src, rec)


def _a3d_problem(case, rng):
    nx, ny, nz, npml = case["nx"], case["ny"], case["nz"], case["npml"]
    dx = 5.0
    base = _layers(rng, nz, 1500.0, 4500.0)
    lat = _wave(rng, nx)[:, None] * _wave(rng, ny)[None, :]
    vp = lat[:, :, None] * base[None, None, :]
    rho = np.broadcast_to(W.gardner(base)[None, None, :], vp.shape).copy()
    rho *= _wave(rng, nx)[:, None, None]
    dt_ms = 0.5 * dx / (math.sqrt(3.0) * float(base.max() * lat.max())) * 1e3
    f = 0.05 / (dt_ms * 1e-3)
    src = [("Bulk", 1.0, f, int(rng.integers(nx // 3, 2 * nx // 3 + 1)) * dx,
            int(rng.integers(ny // 3, 2 * ny // 3 + 1)) * dx, min(10, nz // 3) * dx)]
    n = case["nside"]
    xs = [round(i * (nx - 1) / max(n - 1, 1)) * dx for i in range(n)]
    ys = [round(i * (ny - 1) / max(n - 1, 1)) * dx for i in range(n)]
    rec = [("Vz", x, y, 0.0, 0.0, dt_ms) for x in xs for y in ys]
    return W.A3DProblem(vp, rho, (dx, dx, dx), npml, dt_ms, W.steps_duration(case["steps"], dt_ms),
                        src, rec, Rc=1e-3)


def _ecyl_problem(case, rng):
    nx, nz = case["nx"], case["nz"]
    vp = _wave(rng, nx)[:, None] * _layers(rng, nz, 1800.0, 4200.0)[None, :]
    vs = vp / 1.73
    rho = W.gardner(vp)
    dt_ms = 0.5 * 1.0 / (math.sqrt(2.0) * float(vp.max())) * 1e3
    f = 0.05 / (dt_ms * 1e-3)
    ir, iz = int(rng.integers(nx // 4, nx // 2)), int(rng.integers(nz // 3, 2 * nz // 3))
    comps = ("Vr", "Vz", "Trr", "Tzz")
    # records around the source, where the field is strong in the steps taken
    rec = [(comps[k % 4], float(min(max(ir - 24 + 2 * k, 2), nx - 2)), float(iz + 3), 0.0, dt_ms)
           for k in range(case["nrec"])]
    return W.ECylProblem(vp, vs, rho, 1.0, 1.0, case["npml"], dt_ms,
                         W.steps_duration(case["steps"], dt_ms), [("Fz", 1.0, f, float(ir), float(iz))],
                         rec, n=case["n"])


def _problems(case, seed):
    rng = np.random.default_rng([seed, 11])
    if case["kind"] == "eiso":
        return [_eiso_problem(case["nx"], case["nz"], case["npml"], case["shots"], case["nrec"],
                              case["steps"], rng)]
    if case["kind"] == "group":
        sides = [tuple(int(v) for v in s.split("x")) for s in case["sides"].split(",")]
        return [_eiso_problem(nx, nz, case["npml"], 1, case["nrec"], case["steps"], rng)
                for nx, nz in sides]
    if case["kind"] == "a3d":
        return [_a3d_problem(case, rng)]
    return [_ecyl_problem(case, rng)]


# ----------------------------------------------------------------------------
# the timed work
# ----------------------------------------------------------------------------

def prepare(case, seed):
    make = {"eiso": api.eiso_device, "group": api.eiso_device, "a3d": api.a3d_device,
            "ecyl": api.ecyl_device}[case["kind"]]
    devs = [make(p, case["precision"])[0] for p in _problems(case, seed)]
    if case.get("graph"):
        devs[0].set_graph(case["graph"])
    return dict(kind=case["kind"], steps=case["steps"], snap=case.get("snap", 0), devs=devs)


def run(state):
    devs, steps = state["devs"], state["steps"]
    for d in devs:
        d.reset()
    if state["kind"] == "group":
        api.group_run(devs, steps)
        return [d.traces_array(0) for d in devs]
    dev = devs[0]
    dev.run(steps)
    if state["kind"] == "eiso":
        out = [dev.traces_array(s) for s in range(dev.nshots)]
    elif state["kind"] == "a3d":
        out = dev.traces_array()
    else:
        out = np.stack(dev.traces())
    return [out, dev.get_field("vz")] if state["snap"] else out


def work(case):
    """Bytes: per step the wavefields read and written once and the materials
    read once (split parts and memory variables of the frame likewise), and
    the traces written; operations: the updates' own."""
    v = {"fp32": 4, "fp64": 8, "bfp16": 2.25}[case["precision"]]
    m = 8 if case["precision"] == "fp64" else 4
    steps = case["steps"]
    if case["kind"] in ("eiso", "group"):
        np_ = case["npml"]
        sides = [(case["nx"], case["nz"])] if case["kind"] == "eiso" else \
            [tuple(int(x) for x in s.split("x")) for s in case["sides"].split(",")]
        shots = case.get("shots", 1)
        by = fl = 0.0
        for nx, nz in sides:
            alln = (nx + 2 * np_) * (nz + 2 * np_)
            by += shots * (10 * v * alln + 20 * m * (alln - nx * nz) + 8 * case["nrec"]) + 5 * m * alln
            fl += shots * 32 * alln
        return dict(bytes=by * steps, flops=fl * steps)
    if case["kind"] == "a3d":
        n2 = [case[k] + 2 * case["npml"] for k in ("nx", "ny", "nz")]
        alln = n2[0] * n2[1] * n2[2]
        slabs = sum(2 * case["npml"] * alln // n for n in n2)
        by = alln * (8 * v + 2 * m) + 4 * m * slabs + 8 * case["nside"] ** 2
        return dict(bytes=by * steps, flops=33.0 * alln * steps)
    alln = (case["nx"] + case["npml"]) * (case["nz"] + 2 * case["npml"])
    return dict(bytes=(alln * (18 * v + 8 * m) + 8 * case["nrec"]) * steps, flops=70.0 * alln * steps)


# ----------------------------------------------------------------------------
# the same in 64 bits, with torch alone
# ----------------------------------------------------------------------------

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=_dev())


def _half_up(v):
    return int(math.copysign(math.floor(abs(v) + 0.5), v))


def _ricker(A, f, dt):
    """A Ricker wavelet of 2/f seconds, its peak scaled to A."""
    tc = 1.0 / f
    t = np.arange(int(math.ceil(tc * 2.0 / dt))) * dt - tc
    k = (math.pi * f) ** 2 * t * t
    w = (1.0 - 2.0 * k) * np.exp(-k)
    return A * w / np.abs(w).max()


def _sampled(it, dt, t0, rdt):
    """Whether a record of period rdt takes the state after step it."""
    t = dt * (it + 1)
    d = t - t0 + 1e-15
    return abs(d) < 0.99 * dt or (t > t0 and rdt > 0 and abs(math.fmod(1e6 * d, 1e6 * rdt)) < 1e-8)


def _steps(p):
    n = int(p.duration / p.dt)
    return n + 1 if n * p.dt < p.duration else n


def _record(p, taken):
    """The steps of `taken` ([nstep] values per record) that a record keeps:
    every record of a case has the same start and period."""
    r = p.receivers[0]
    keep = [k for k in range(len(taken)) if _sampled(k, p.dt, r[-2], r[-1] * 1e-3)]
    return torch.stack([taken[k] for k in keep], -1)


def _exact_eiso(p):
    """Split parts everywhere (A = B = 1 inside the frame's inner edge): the
    sum of the two parts is the plain update there."""
    nx, nz, n, dt, h = p.nx, p.nz, p.npml, p.dt, p.h
    vp, vs, rho = _t(p.vp), _t(p.vs), _t(p.rho)
    la, mu, b = rho * (vp * vp - 2 * vs * vs), rho * vs * vs, 1.0 / rho
    l2 = la + 2 * mu

    def mean(a, dim):   # with the next node; the last one alone
        nxt = torch.cat([a.narrow(dim, 1, a.shape[dim] - 1), a.narrow(dim, a.shape[dim] - 1, 1)], dim)
        return (a + nxt) / 2

    def pad(a, corner=False):
        i = torch.arange(-n, nx + n, device=a.device)
        j = torch.arange(-n, nz + n, device=a.device)
        q = a[i.clamp(0, nx - 1)][:, j.clamp(0, nz - 1)]
        if corner:      # lambda and lambda + 2 mu beyond the last node in x and z
            c = nx * nx - 1 if nx <= nz else nx * nz - 1
            q[n + nx:, n + nz:] = a.reshape(-1)[c]
        return (dt / h) * q

    m_b, m_bm = pad(b), pad(mean(mean(b, 0), 1))
    m_la, m_l2, m_mu = pad(mean(la, 0), True), pad(mean(l2, 0), True), pad(mean(mu, 1))
    d0 = math.log(1e3) * 1.5 * float(vp.mean()) / (n * h)

    def prof(N, half):
        a, bb = torch.ones(N + 2 * n, dtype=torch.float64), torch.ones(N + 2 * n, dtype=torch.float64)
        for k in range(n):
            lo = d0 * ((n - k - (0.5 if half else 0.0)) / n) ** 2
            hi = d0 * ((n - k + (0.5 if half else 0.0)) / n) ** 2
            for at, d in ((k, lo), (N + 2 * n - 1 - k, hi)):
                a[at], bb[at] = (2 - dt * d) / (2 + dt * d), 2 / (2 + dt * d)
        return a.to(_dev()), bb.to(_dev())

    X, XH = [tuple(v[:, None] for v in prof(nx, s)) for s in (False, True)]
    Z, ZH = [tuple(v[None, :] for v in prof(nz, s)) for s in (False, True)]
    S = len(p.shots)
    shape = (S, nx + 2 * n, nz + 2 * n)
    new = lambda: torch.zeros(shape, dtype=torch.float64, device=_dev())  # noqa: E731
    f = {k: [new(), new(), new()] for k in ("vx", "vz", "txx", "tzz", "txz")}   # x part, z part, total
    d = new()

    def back(a, dim):
        torch.sub(a.narrow(dim, 1, a.shape[dim] - 1), a.narrow(dim, 0, a.shape[dim] - 1),
                  out=d.narrow(dim, 1, a.shape[dim] - 1))
        d.narrow(dim, 0, 1).copy_(a.narrow(dim, 0, 1))
        return d

    def fwd(a, dim):
        torch.sub(a.narrow(dim, 1, a.shape[dim] - 1), a.narrow(dim, 0, a.shape[dim] - 1),
                  out=d.narrow(dim, 0, a.shape[dim] - 1))
        d.narrow(dim, a.shape[dim] - 1, 1).copy_(-a.narrow(dim, a.shape[dim] - 1, 1))
        return d

    def upd(q, AB, m, delta):
        q.mul_(AB[0]).add_(delta * (AB[1] * m))

    def total(k):
        torch.add(f[k][0], f[k][1], out=f[k][2])

    si = torch.tensor([[s, _half_up(q[3] / h) + n, _half_up(q[4] / h) + n]
                       for s, qs in enumerate(p.shots) for q in qs], device=_dev()).T
    wav = [[_ricker(q[1], q[2], dt) for q in qs][0] for qs in p.shots]
    comp = [r[0].lower() for r in p.receivers]
    ri = torch.tensor([[_half_up(r[1] / h) + n, _half_up(r[2] / h) + n] for r in p.receivers],
                      device=_dev()).T
    isx = torch.tensor([c == "vx" for c in comp], device=_dev())
    got = []
    for it in range(_steps(p)):
        txx, tzz, txz = f["txx"][2], f["tzz"][2], f["txz"][2]
        upd(f["vx"][0], X, m_b, back(txx, 1)); upd(f["vx"][1], Z, m_b, back(txz, 2))
        upd(f["vz"][0], XH, m_bm, fwd(txz, 1)); upd(f["vz"][1], ZH, m_bm, fwd(tzz, 2))
        total("vx"); total("vz")
        vx, vz = f["vx"][2], f["vz"][2]
        ax = fwd(vx, 1)
        upd(f["txx"][0], XH, m_l2, ax); upd(f["tzz"][0], XH, m_la, ax)
        az = back(vz, 2)
        upd(f["txx"][1], Z, m_la, az); upd(f["tzz"][1], Z, m_l2, az)
        upd(f["txz"][0], X, m_mu, back(vz, 1)); upd(f["txz"][1], ZH, m_mu, fwd(vx, 2))
        add = _t([dt * w[it] if it < len(w) else 0.0 for w in wav])
        for k in ("txx", "tzz"):
            f[k][0][si[0], si[1], si[2]] += add
        for k in ("txx", "tzz", "txz"):
            total(k)
        got.append(torch.where(isx, vx[:, ri[0], ri[1]], vz[:, ri[0], ri[1]]))
    return list(_record(p, got)), f["vz"][2][0]


def _cpml(n, h, dt, Rc, alpha, x, a):
    """CPML b, c of a node x cells into the frame's profile, alpha a; kappa 1."""
    d = -3.0 * 5000.0 * math.log(Rc) / (2 * n * h) * (x / n) ** 2
    b = math.exp(-(d + a) * dt)
    return b, d * (b - 1.0) / (d + a)


def _exact_a3d(p):
    n, dt, (dx, dy, dz) = p.npml, p.dt, p.d
    N = [s + 2 * n for s in p.shape]
    rho = np.pad(p.rho, n, mode="edge")
    K = _t(rho) * _t(np.pad(p.vp, n, mode="edge")) ** 2 * dt
    rho = _t(rho)
    alpha = math.pi * p.sources[0][2] if p.alpha_max else 0.0

    def coef(ax, half):
        m = N[ax] - 1 if half else N[ax]
        s = 0.5 if half else 0.0
        b, c = torch.ones(m, dtype=torch.float64), torch.zeros(m, dtype=torch.float64)
        for k in range(n):
            v = _cpml(n, p.d[ax], dt, p.Rc, alpha, n - k - s, (k + s) * alpha / n)
            b[k], c[k] = v
            b[m - 1 - k], c[m - 1 - k] = v
        sh = [1, 1, 1]
        sh[ax] = m
        return b.reshape(sh).to(_dev()), c.reshape(sh).to(_dev())

    P = torch.zeros(N, dtype=torch.float64, device=_dev())
    v, ir, psi, phi, ch, cn = [], [], [], [], [], []
    for ax in range(3):
        lo, hi = rho.narrow(ax, 0, N[ax] - 1), rho.narrow(ax, 1, N[ax] - 1)
        ir.append(2 * dt / (lo + hi))
        v.append(torch.zeros(N, dtype=torch.float64, device=_dev()))
        psi.append(torch.zeros_like(ir[ax]))
        phi.append(torch.zeros_like(P))
        ch.append(coef(ax, True))
        cn.append(coef(ax, False))
    del rho
    at = [_half_up(q / h) + n for q, h in zip(p.sources[0][3:6], p.d)]
    w = _ricker(p.sources[0][1], p.sources[0][2], dt)
    ri = (torch.as_tensor(np.array([r[1:4] for r in p.receivers])) / torch.tensor(p.d)).add(0.5).floor().long().T + n
    ri = ri.to(_dev())
    inner = (slice(1, None),) * 3
    got = []
    for it in range(_steps(p)):
        for ax in range(3):
            m = N[ax] - 1
            g = (P.narrow(ax, 1, m) - P.narrow(ax, 0, m)).div_(p.d[ax])
            psi[ax].mul_(ch[ax][0]).add_(ch[ax][1] * g)
            v[ax].narrow(ax, 0, m).sub_(g.add_(psi[ax]).mul_(ir[ax]))
            del g
        s = torch.zeros_like(P[inner])
        for ax in range(3):
            cut = list(inner)
            cut[ax] = slice(0, -1)
            g = (v[ax][inner] - v[ax][tuple(cut)]).div_(p.d[ax])
            b, c = (q.narrow(ax, 1, N[ax] - 1) for q in cn[ax])
            phi[ax][inner].mul_(b).add_(c * g)
            s.add_(g).add_(phi[ax][inner])
        P[inner].sub_(s.mul_(K[inner]))
        if it < len(w):
            P[at[0], at[1], at[2]] += dt * 1e6 * w[it]
        got.append(v[2][ri[0], ri[1], ri[2]])
    return _record(p, got), v[2]


def _exact_ecyl(p):
    n, dt, dx, dz, mode = p.npml, p.dt, p.dx, p.dz, p.n
    nx, nz = p.nx, p.nz
    I, J = nx + n, nz + 2 * n
    pad = [(0, n), (n, n)]
    vp, vs, rho = (_t(np.pad(a, pad, mode="edge")) for a in (p.vp, p.vs, p.rho))
    mu0, lam = rho * vs * vs, rho * (vp * vp - 2 * vs * vs)
    l2m = lam + 2 * mu0

    def prev(a, dim):
        return torch.cat([a.narrow(dim, 0, 1), a.narrow(dim, 0, a.shape[dim] - 1)], dim)

    harm = lambda a, b: 2 * a * b / (a + b)  # noqa: E731
    muj, mui = harm(mu0, prev(mu0, 1)), harm(mu0, prev(mu0, 0))
    mu = 4 / (1 / mu0 + 1 / prev(mu0, 0) + 1 / prev(mu0, 1) + 1 / prev(prev(mu0, 0), 1))
    bij, bj, bi = 1 / rho, 2 / (rho + prev(rho, 1)), 2 / (rho + prev(rho, 0))
    alpha = math.pi * p.sources[0][2] if p.alpha_max else 0.0
    node = lambda h, k: _cpml(n, h, dt, p.Rc, alpha, n - k, k * alpha / n)  # noqa: E731
    half = lambda h, k: _cpml(n, h, dt, p.Rc, alpha, n - k - 0.5, (k + 0.5) * alpha / n)  # noqa: E731
    end = lambda h, k: _cpml(n, h, dt, p.Rc, alpha, k + 0.5, (n - k - 0.5) * alpha / (n + 1))  # noqa: E731

    def table(N, put, col):
        b, c = torch.zeros(N, dtype=torch.float64), torch.zeros(N, dtype=torch.float64)
        for k, v in put:
            if 0 <= k < N:
                b[k], c[k] = v
        return tuple((v[:, None] if col else v[None, :]).to(_dev()) for v in (b, c))

    zh = table(J, [(k, half(dz, k)) for k in range(n)] + [(nz + n - 1 + k, end(dz, k)) for k in range(n + 1)], False)
    zt = table(J, [(k, half(dz, k)) for k in range(n)] + [(nz + n + k, end(dz, k)) for k in range(n)], False)
    zn = table(J, [(k, node(dz, k)) for k in range(n)] + [(nz + n + k, node(dz, n - 1 - k)) for k in range(n)], False)
    rn = table(I, [(nx + k, node(dx, n - 1 - k)) for k in range(n)], True)
    rh = table(I, [(nx - 1 + k, end(dx, k)) for k in range(n + 1)], True)
    rt = table(I, [(nx + k, end(dx, k)) for k in range(n)], True)
    psi = {}

    def filt(key, bc, d, rows=slice(None), cols=slice(None)):
        """d plus its memory variable (zero wherever b = c = 0)."""
        b, c = (v[rows if v.shape[0] > 1 else slice(None), cols if v.shape[1] > 1 else slice(None)] for v in bc)
        if key not in psi:
            psi[key] = torch.zeros_like(d)
        psi[key].mul_(b).add_(c * d)
        return d + psi[key]

    z = lambda: torch.zeros(I, J, dtype=torch.float64, device=_dev())  # noqa: E731
    vr, vt, vz, trr, ttt, tzz, trz, trt, ttz = (z() for _ in range(9))
    r = torch.arange(I, dtype=torch.float64, device=_dev())[:, None] * dx
    r5 = r[:-1] + 0.5 * dx
    lo, up = slice(None, -1), slice(1, None)
    ps = p.sources[0]
    at = (_half_up(ps[3] / dx), _half_up(ps[4] / dz) + n)
    w = _ricker(ps[1], ps[2], dt)
    fields = dict(vr=vr, vt=vt, vz=vz, trr=trr, tzz=tzz)
    rec = [(q[0].lower(), _half_up(q[1] / dx), _half_up(q[2] / dz) + n) for q in p.receivers]
    by = {k: ([s for s, q in enumerate(rec) if q[0] == k],
              torch.tensor([q[1] for q in rec if q[0] == k], dtype=torch.long, device=_dev()),
              torch.tensor([q[2] for q in rec if q[0] == k], dtype=torch.long, device=_dev())) for k in fields}
    got = []
    for it in range(_steps(p)):
        # velocities
        ddz = filt("trz_z", zh, (trz[:, 1:] - trz[:, :-1]) / dz, cols=lo)
        a = filt("trr_r", rn, (trr[1:] - trr[:-1])[:, lo] / dx, rows=up)
        b = filt("trr_1", rn, ((trr[1:] + trr[:-1]) / (2 * r[1:]))[:, lo], rows=up)
        c = filt("ttt_1", rn, ((ttt[1:] + ttt[:-1]) / (2 * r[1:]))[:, lo], rows=up)
        s = a + b - c + ddz[1:]
        if mode:
            s += mode * filt("trt_1", rn, (trt[1:] / r[1:])[:, lo], rows=up)
        if mode % 2:
            vr[0, lo] += dt * bj[0, lo] * (2 * trr[0, lo] / dx + ddz[0])
        vr[1:, lo] += dt * bj[1:, lo] * s
        ddz = filt("ttz_z", zh, (ttz[:-1, 1:] - ttz[:-1, :-1]) / dz, cols=lo)
        s = filt("trt_2", rh, ((trt[1:] + trt[:-1]) / r5)[:, lo], rows=lo) + \
            filt("trt_r", rh, (trt[1:] - trt[:-1])[:, lo] / dx, rows=lo) + ddz
        if mode:
            s -= mode * filt("ttt_2", rh, (ttt[:-1] / r5)[:, lo], rows=lo)
        vt[:-1, lo] += dt * bij[:-1, lo] * s
        s = filt("tzz_z", zn, (tzz[:-1, 1:] - tzz[:-1, :-1]) / dz, cols=up) + \
            filt("trz_r", rh, (trz[1:] - trz[:-1])[:, up] / dx, rows=lo) + \
            filt("trz_2", rh, ((trz[1:] + trz[:-1]) / (2 * r5))[:, up], rows=lo)
        if mode:
            s += mode * filt("ttz_2", rh, (ttz[:-1] / r5)[:, up], rows=lo)
        vz[:-1, up] += dt * bi[:-1, up] * s
        if it < len(w):
            vz[at] += dt * bi[at] * w[it]
        # stresses
        e = filt("vr_r", rh, (vr[1:] - vr[:-1])[:, lo] / dx, rows=lo)
        g = filt("vr_2", rh, ((vr[1:] + vr[:-1]) / (2 * r5))[:, lo], rows=lo)
        if mode:
            g = g + mode * filt("vt_2", rh, (vt[:-1] / r5)[:, lo], rows=lo)
        q = filt("vz_z", zh, (vz[:-1, 1:] - vz[:-1, :-1]) / dz, cols=lo)
        L, M = dt * lam[:-1, lo], dt * l2m[:-1, lo]
        trr[:-1, lo] += M * e + L * (g + q)
        ttt[:-1, lo] += M * g + L * (e + q)
        tzz[:-1, lo] += M * q + L * (e + g)
        trz[1:, up] += dt * mu[1:, up] * (filt("vr_z", zt, (vr[1:, 1:] - vr[1:, :-1]) / dz, cols=up) +
                                          filt("vz_r", rt, (vz[1:] - vz[:-1])[:, up] / dx, rows=up))
        s = filt("vt_r", rn, (vt[1:] - vt[:-1]) / dx, rows=up) - \
            filt("vt_1", rn, (vt[1:] + vt[:-1]) / (2 * r[1:]), rows=up)
        if mode:
            s -= mode * filt("vr_1", rn, vr[1:] / r[1:], rows=up)
        if mode % 2:
            trt[0] += dt * muj[0] * 2 * vt[0] / dx
        trt[1:] += dt * muj[1:] * s
        s = filt("vt_z", zn, (vt[:-1, 1:] - vt[:-1, :-1]) / dz, cols=up)
        if mode:
            s = s - mode * filt("vz_2", rh, (vz[:-1] / r5)[:, up], rows=lo)
        ttz[:-1, up] += dt * mui[:-1, up] * s
        row = torch.empty(len(rec), dtype=torch.float64, device=_dev())
        for k, (who, ii, jj) in by.items():
            if who:
                row[who] = fields[k][ii, jj]
        got.append(row)
    return _record(p, got), vz


def exact(case, seed):
    f = {"eiso": _exact_eiso, "group": _exact_eiso, "a3d": _exact_a3d, "ecyl": _exact_ecyl}[case["kind"]]
    out = [f(p) for p in _problems(case, seed)]
    if case["kind"] == "group":
        return [traces[0] for traces, _ in out]
    traces, vz = out[0]
    return [traces, vz] if case.get("snap") else traces
