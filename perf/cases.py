"""Cases by which this engine's speed is followed, through its public API.

A pass is what a program does between two looks at a simulation: `Sim.step(n)`
(or `Batch.run(n)`), then the stored energy that decides whether to go on, and
the spectra of every port and probe; or, for a run that is saved and taken up
again, `Sim.restore`, `Sim.step`, `Sim.checkpoint`. What `prepare` gives is a
finalized simulation on the device, its pulse on the way (`lead` steps done).

Geometry comes from the package's own generators (scenes.py, boards.py). The
seed moves substrate permittivities and the exciting pulse, so two seeds of a
case have grids of one size and different coefficients and fields.

`exact` steps the same scene in float64 with plain torch: it hands the
generators a recorder in place of the library and works from the recorded
geometry. Scenes with surface impedance or mode ports have no such value (their
coefficients come out of a fit and of an eigenmode solver).
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from courant_b200 import boards, scenes
from courant_b200.api import C0, EPS0, MU0, Courant, DebyeModel

ETA0 = 376.730313668

# ------------------------------------------------------------------- the cases


def listed() -> list[dict]:
    return [
        # the every-feature known-answer scene, looked at every 10 steps: an interactive monitor; all latency
        dict(name="monitor_6k", kind="scene", scene="parity", lead=500, steps=10),
        # a saved run taken up again and saved: Debye poles, copper surface impedance, whole state in and out
        dict(name="resume_6k", kind="resume", scene="lossy", lead=400, steps=200),
        # the same of a lossless dielectric scene
        dict(name="resume_plain_6k", kind="resume", scene="parity", lead=400, steps=200),
        # PEC cavity without CPML, odd sizes, whole fields out (the reference's resonator test, larger)
        dict(name="cavity_100k", kind="cavity", nx=61, ny=47, nz=35, lead=300, steps=500),
        # the small GCPW line of the benchmark, one run-control interval, 401 frequencies
        dict(name="line_300k", kind="line", hmin=25e-6, hmax=200e-6, dx=105e-6, length=10e-3, npml=8, zair=4.2e-3,
             yair=0.9e-3, poles=0, copper=False, lead=800, steps=200),
        # the lossy line (6 poles, 35 um copper with rough surface impedance, solder mask) at its benchmark mesh
        dict(name="lossy_3p6m", kind="line", hmin=10e-6, hmax=30e-6, dx=45e-6, length=10e-3, npml=8, zair=1.8e-3,
             yair=1.2e-3, poles=6, copper=True, lead=300, steps=100),
        # the lossless line at the same mesh and a longer run of line: no auxiliaries but CPML
        dict(name="line_6m", kind="line", hmin=10e-6, hmax=30e-6, dx=45e-6, length=18e-3, npml=8, zair=1.8e-3,
             yair=1.2e-3, poles=0, copper=False, lead=300, steps=100),
        # a served request of the smaller sort: 4 mode ports, 4-pole cores
        dict(name="board_250k_mode", kind="board", layout=32, cells=2.5e5, ports="mode", nports=4, nf=16, lead=600,
             steps=200),
        # a served request of the middle of the range, lumped ports
        dict(name="board_1m", kind="board", layout=7, cells=1e6, ports="lumped", nports=2, nf=32, lead=500, steps=200),
        # the large board's proportions (500 x 330 x 64 cells)
        dict(name="board_10m", kind="board", layout=2026, cells=1.06e7, ports="lumped", nports=2, nf=201, lead=150,
             steps=100, tx=500, ty=330, tz=64),
        # the upper end of the served range
        dict(name="board_16m", kind="board", layout=11, cells=1.6e7, ports="lumped", nports=1, nf=32, lead=100,
             steps=80),
        # uneven boards advanced together (batching, serving)
        dict(name="batch_8", kind="batch", layout=40, members=8, cells=5e4, top=8e5, nports=2, nf=16, lead=200,
             steps=128),
    ]


def _log(rng: random.Random, lo: float, hi: float) -> float:
    return lo * (hi / lo) ** rng.random()


def draw(rng: random.Random) -> dict:
    """One more case of the same ranges: the generators' sizes between the listed ones, odd ones among them."""
    kind = rng.choice(["board", "board", "line", "lossy", "cavity", "batch", "resume", "scene"])
    layout = rng.randrange(1, 10000)
    if kind == "board":
        cells = _log(rng, 5e4, 1.4e7)
        return dict(kind="board", layout=layout, cells=cells, ports="lumped", nports=rng.randint(1, 4),
                    nf=rng.choice([16, 32, 101, 201]), lead=rng.randint(80, 200),
                    steps=max(20, min(rng.randint(40, 300), int(1.1e9 / cells))))
    if kind in ("line", "lossy"):
        hmin = _log(rng, 10e-6, 60e-6)
        small = hmin > 20e-6
        return dict(kind="line", hmin=hmin, hmax=hmin * rng.uniform(2.5, 8.0), dx=_log(rng, 45e-6, 120e-6),
                    length=rng.uniform(4e-3, 10e-3), npml=rng.randint(5, 10), zair=rng.uniform(1.0e-3, 2.5e-3),
                    yair=rng.uniform(0.6e-3, 1.2e-3), poles=rng.randint(1, 8) if kind == "lossy" else 0,
                    copper=kind == "lossy" and rng.random() < 0.7, lead=rng.randint(200, 500),
                    steps=rng.randint(100, 300) if small else rng.randint(40, 100))
    if kind == "cavity":
        return dict(kind="cavity", nx=int(_log(rng, 12, 160)), ny=int(_log(rng, 12, 120)), nz=int(_log(rng, 8, 100)),
                    lead=rng.randint(100, 300), steps=rng.randint(50, 500))
    if kind == "batch":
        return dict(kind="batch", layout=layout, members=rng.randint(2, 8), cells=_log(rng, 4e4, 1e5),
                    top=_log(rng, 2e5, 8e5), nports=rng.randint(1, 2), nf=rng.choice([16, 32]), lead=rng.randint(50, 300),
                    steps=rng.randint(20, 200))
    scene = rng.choice(["parity", "lossy"])
    if kind == "resume":
        return dict(kind="resume", scene=scene, lead=rng.randint(100, 600), steps=rng.randint(20, 300))
    return dict(kind="scene", scene=scene, lead=rng.randint(100, 600), steps=rng.randint(1, 60))


# ------------------------------------------------- scenes, on any "library"


def _pulse(rng: random.Random, fmax: float) -> tuple[float, float, float]:
    """Amplitude, delay and width of the exciting Gaussian."""
    tau = math.sqrt(6.9) / (math.pi * 1.25 * fmax) * rng.uniform(0.9, 1.1)
    return rng.uniform(0.5, 2.0), rng.uniform(2.4, 2.8) * tau, tau


def _small_scene(c, case, rng):
    """scenes.parity_scene or lossy_scene with a substrate and a pulse of the seed's."""
    fn = {"parity": scenes.parity_scene, "lossy": scenes.lossy_scene}[case["scene"]]
    scale = rng.uniform(0.9, 1.3)

    class Scaled:   # the library with every dielectric's permittivity scaled
        def __getattr__(self, name):
            return getattr(c, name)

        def createSim(self, x, y, z):
            s = c.createSim(x, y, z)
            box, deb = s.materialBox, s.materialBoxDebye
            s.materialBox = lambda *a: box(*a[:6], a[6] * scale, *a[7:])
            s.materialBoxDebye = lambda *a: deb(*a[:6], DebyeModel(a[6].eps_inf * scale, a[6].fp, a[6].deps, 0.0), *a[7:])
            return s

    s, meta = fn(Scaled())
    amp, t0, tau = _pulse(rng, 20e9)
    s.setGaussian(meta["ports"][0], amp, t0, tau)
    return s


def _line(c, case, rng):
    kw = dict(er=rng.uniform(3.6, 4.4), length=case["length"], hmin=case["hmin"], hmax=case["hmax"], dx=case["dx"],
              yair=case["yair"], zair=case["zair"], npml=case["npml"], probes=True)
    if case["poles"]:
        kw.update(debye_poles=case["poles"], nf=64)
    if case["copper"]:
        kw.update(tcu=35e-6, mask=20e-6, sigma_cu=5.8e7, huray=(0.5e-6, 2.0e11))
    s, meta = scenes.gcpw_line(c, **kw)
    amp, t0, tau = _pulse(rng, 40e9)
    s.setGaussian(meta["ports"][0], amp, t0, tau)
    return s


def _plan(case, cells=None, layout=None):
    target = (case["tx"], case["ty"], case["tz"]) if case.get("tx") else None
    return boards.plan_board(layout or case["layout"], cells or case["cells"], ports=case.get("ports", "lumped"),
                             nf=case["nf"], nports=case["nports"], target=target)


def _board(c, plan, rng):
    plan.eps = plan.eps * np.array([rng.uniform(0.97, 1.03) for _ in plan.eps])
    s, meta = boards.board_sim(c, plan)
    amp, t0, tau = _pulse(rng, plan.fmax)
    if plan.ports == "mode":
        s.setModeExcitation(meta["modeports"][0], t0, tau)
    else:
        s.setGaussian(meta["ports"][0], amp, t0, tau)
    return s


def _cavity(c, case, rng):
    """PEC box, graded a little in x, half filled with a lossy dielectric; a port and probes along z."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    x = np.cumsum(np.concatenate([[0.0], 1e-4 * (1 + 0.2 * np.sin(np.arange(nx) * 0.3))]))
    s = c.createSim(x, 1e-4 * np.arange(ny + 1), 0.9e-4 * np.arange(nz + 1))
    s.materialBox(-1, 1, -1, 1, 0, 0.9e-4 * (nz // 2), rng.uniform(2.0, 4.0), rng.uniform(0.0, 0.1))
    p = s.addLumpedPort(2, nx // 3, ny // 3, 0, nz // 4, 1, 50.0)
    amp, t0, tau = _pulse(rng, 60e9)
    s.setGaussian(p, amp, t0, tau)
    s.setFrequencies(np.linspace(2e9, 60e9, 30))
    s.addVProbe(2, 2 * nx // 3, ny // 2, 0, nz // 4, 1)
    s.addIProbe(0, nx // 2, ny // 4, ny // 2, nz // 4, nz // 2)
    s.finalize(0.99)
    return s


def _members(case):
    """(cells, layout) of a batch's boards: sizes spread over [cells, top] by their logarithm."""
    m = case["members"]
    return [(case["cells"] * (case["top"] / case["cells"]) ** (q / max(1, m - 1)), case["layout"] + q) for q in range(m)]


def _sims(c, case, seed):
    rng = random.Random(seed)
    if case["kind"] == "batch":
        return [_board(c, _plan(case, n, lay), rng) for n, lay in _members(case)]
    if case["kind"] == "board":
        return [_board(c, _plan(case), rng)]
    make = {"scene": _small_scene, "resume": _small_scene, "line": _line, "cavity": _cavity}[case["kind"]]
    return [make(c, case, rng)]


# ---------------------------------------------------------------- one pass


def prepare(case: dict, seed: int) -> dict:
    c = Courant()
    sims = _sims(c, case, seed)
    for s in sims:
        s.prepareDevice()
        s.step(case["lead"])
    ex = c.ex
    state = dict(kind=case["kind"], steps=case["steps"], sims=sims,
                 count=[(ex.cem_plan_nport(s.h), ex.cem_plan_nvprobe(s.h), ex.cem_plan_niprobe(s.h)) for s in sims])
    if case["kind"] == "batch":
        state["batch"] = c.createBatch()
        for s in sims:
            state["batch"].add(s, 10 ** 9)
    if case["kind"] == "resume":
        state["saved"] = sims[0].checkpoint()
    return state


def _spectra(s, count) -> dict:
    nport, nv, ni = count
    return {"V": np.array([s.portV(p) for p in range(nport)]), "I": np.array([s.portI(p) for p in range(nport)]),
            "vprobe": np.array([s.vprobe(p) for p in range(nv)]), "iprobe": np.array([s.iprobe(p) for p in range(ni)]),
            "source": s.sourceSpectrum()}


def _parts(s, buf) -> dict:
    """A checkpoint's fields and the rest of it."""
    n = 6 * s.N
    return {"fields": buf[8:8 + n], "rest": buf[8 + n:]}


def run(state: dict):
    sims, kind, n = state["sims"], state["kind"], state["steps"]
    if kind == "batch":
        state["batch"].run(n)
        return [_spectra(s, q) for s, q in zip(sims, state["count"])]
    s = sims[0]
    if kind == "resume":
        s.restore(state["saved"])
        s.step(n)
        return _parts(s, s.checkpoint())
    s.step(n)
    if kind == "scene":
        return _spectra(s, state["count"][0])
    if kind == "cavity":
        return {"energy": s.energy(), **_parts(s, s.checkpoint())}
    return {"energy": s.energy(), **_spectra(s, state["count"][0])}


def work(case: dict) -> dict:
    """Compulsory traffic and arithmetic of a pass, as the benchmark counts them: per time step every field, CPML
    auxiliary, Debye current and surface-impedance state read once and written once (float32)."""
    total = dict(bytes=0.0, flops=0.0)
    plans = [_plan(case, n, lay) for n, lay in _members(case)] if case["kind"] == "batch" else None
    if case["kind"] == "board":
        plans = [_plan(case)]
    grids = []
    if plans:
        for p in plans:
            nx, ny, nz = p.meta["dims"]
            grids.append((nx, ny, nz, [p.npml] * 4 + [0, p.npml], 4, 3.0 * nx * ny * p.kl[3]))
    else:
        r = _sims(Recorder(), case, 0)[0]
        nx, ny, nz = (len(v) - 1 for v in r.node)
        deb = [b for b in r.boxes if b[3] is not None]
        nd = 3.0 * sum(float(np.prod([b1 - b0 for b0, b1 in b[0]])) for b in deb)
        grids.append((nx, ny, nz, r.npml, len(r.fp), nd))
    for nx, ny, nz, npml, poles, nd in grids:
        cells, n = nx * ny * nz, (nx, ny, nz)
        psi = sum(4.0 * (npml[2 * a] + npml[2 * a + 1]) * cells / n[a] for a in range(3))
        total["bytes"] += case["steps"] * (48.0 * cells + 8.0 * psi + 8.0 * poles * nd)
        total["flops"] += case["steps"] * (42.0 * cells + 5.0 * psi + 6.0 * poles * nd)
    return total


# ------------------------------------------- the same scenes in float64, torch


class Recorder:
    """Stands in for the library and its Sim: keeps the scene's definition. (Material fits are inputs of a scene and
    come from the library's host side.)"""

    def __init__(self):
        self.npml = [0] * 6
        self.boxes, self.pec, self.sheets, self.planes, self.cells = [], [], [], [], []
        self.ports, self.vp, self.ip, self.fp = [], [], [], []
        self.unknown = False      # surface impedance or mode ports: coefficients not stated here
        self.freq, self.pulse, self.dt = np.array([1e9]), (0, 0.0, 0.0, 1.0), 1.0

    def fitDjordjevicSarkar(self, *a):
        return Courant().fitDjordjevicSarkar(*a)

    def createSim(self, x, y, z):
        r = Recorder()
        r.node = [np.asarray(v, dtype=np.float64) for v in (x, y, z)]
        return r

    def setBoundary(self, face, type_, ncells=0):
        self.npml[face] = ncells if type_ == 1 else 0

    def _range(self, lims):
        out = []
        for v, lo, hi in zip(self.node, lims[0::2], lims[1::2]):
            at = np.nonzero((0.5 * (v[:-1] + v[1:]) >= lo) & (0.5 * (v[:-1] + v[1:]) <= hi))[0]
            out.append((int(at[0]), int(at[-1]) + 1) if len(at) else (0, 0))
        return out

    def materialBox(self, x0, x1, y0, y1, z0, z1, eps, sigma=0.0):
        self.boxes.append((self._range((x0, x1, y0, y1, z0, z1)), eps, sigma, None))

    def materialBoxDebye(self, x0, x1, y0, y1, z0, z1, m, sigma=0.0):
        self.boxes.append((self._range((x0, x1, y0, y1, z0, z1)), m.eps_inf, sigma, list(m.deps)))

    def setDebyePoles(self, fp):
        self.fp = [float(f) for f in fp]

    def setConductorLoss(self, *a):
        self.unknown = True

    def pecBox(self, *lims):
        self.pec.append(self._range(lims))

    def pecSheet(self, axis, pos, a0, a1, b0, b1):
        self.sheets.append((axis, int(np.argmin(np.abs(self.node[axis] - pos))), a0, a1, b0, b1))

    def pecEdgesPlane(self, axis, m, mu, mv):
        self.planes.append((axis, m, mu, mv))

    def pecCells(self, i0, j0, k0, mask):
        self.cells.append((i0, j0, k0, mask))

    def addLumpedPort(self, axis, n1, n2, m0, m1, dir_, R):
        self.ports.append((axis, n1, n2, m0, m1, dir_, R))
        return len(self.ports) - 1

    def setGaussian(self, port, amp, t0, tau):
        self.pulse = (port, amp, t0, tau)

    def addVProbe(self, axis, n1, n2, m0, m1, dir_):
        self.vp.append((axis, n1, n2, m0, m1, dir_))
        return len(self.vp) - 1

    def addIProbe(self, axis, m, u0, u1, v0, v1):
        self.ip.append((axis, m, u0, u1, v0, v1))
        return len(self.ip) - 1

    def addModePort(self, d):
        self.unknown = True
        return 0

    def setModeExcitation(self, *a):
        self.unknown = True

    def setFrequencies(self, f):
        self.freq = np.asarray(f, dtype=np.float64)

    def finalize(self, cfl=0.99):
        d = [np.diff(v).min() for v in self.node]
        self.dt = cfl / (C0 * math.sqrt(sum(1 / v ** 2 for v in d)))


class Exact:
    """The Yee scheme with CPML, dielectric loss, PEC, lumped ports and Debye poles on a recorded scene, float64."""

    def __init__(self, r: Recorder):
        self.r = r
        self.dev = dev = "cuda" if torch.cuda.is_available() else "cpu"
        f64 = dict(dtype=torch.float64, device=dev)
        self.n = n = [len(v) - 1 for v in r.node]
        self.shape = shape = [v + 1 for v in n]
        self.d = [np.diff(v) for v in r.node]
        self.dd = [0.5 * (np.concatenate([[0.0], d]) + np.concatenate([d, [0.0]])) for d in self.d]
        self.E = [torch.zeros(shape, **f64) for _ in range(3)]
        self.H = [torch.zeros(shape, **f64) for _ in range(3)]
        self.t = lambda v, a: torch.as_tensor(v, **f64).reshape([-1 if q == a else 1 for q in range(3)])
        self._cpml()
        self._coefficients(f64)
        self._lines()
        self.rows, self.vold, self.step_no = [], None, 0

    def _cpml(self):
        r, n = self.r, self.n
        self.ide = [1.0 / v for v in self.dd]
        self.idh = [1.0 / v for v in self.d]
        self.slabs = []      # (axis, E side?, first, last + 1, b, c / spacing)
        for a in range(3):
            x = r.node[a]
            for side in range(2):
                m = r.npml[2 * a + side]
                if not m:
                    continue
                xi, L = (x[m], x[m] - x[0]) if side == 0 else (x[n[a] - m], x[n[a]] - x[n[a] - m])
                smax = 0.8 * 4 / (ETA0 * (L / m))
                for e, pos in ((True, x), (False, 0.5 * (x[:-1] + x[1:]))):
                    depth = np.minimum((xi - pos if side == 0 else pos - xi) / L, 1.0)
                    inside = depth > 0
                    u = np.where(inside, depth, 0.0)
                    sg, kp, al = smax * u ** 3, 1 + 4 * u ** 3, 0.05 * (1 - u)
                    b = np.where(inside, np.exp(-(sg / kp + al) * r.dt / EPS0), 0.0)
                    with np.errstate(divide="ignore", invalid="ignore"):
                        cc = np.where(inside & (sg > 0), sg / (sg * kp + kp * kp * al) * (b - 1), 0.0)
                    sp = self.dd[a] if e else self.d[a]
                    inv = self.ide[a] if e else self.idh[a]
                    inv[inside] = 1.0 / (kp * sp)[inside]
                    if e:
                        lo, hi = (1, m + 1) if side == 0 else (n[a] - m, n[a])
                    else:
                        lo, hi = (0, m) if side == 0 else (n[a] - m, n[a])
                    self.slabs.append((a, e, lo, hi, self.t(b[lo:hi], a), self.t((cc / sp)[lo:hi], a)))
        self.psi = {}

    def _average(self, cell, c):
        """Area-weighted mean over the cells around each edge along c of a cell array."""
        ua, va = (c + 1) % 3, (c + 2) % 3
        w = self.t(self.d[ua], ua) * self.t(self.d[va], va) * torch.ones_like(cell)
        num, den = torch.zeros_like(self.E[0]), torch.zeros_like(self.E[0])
        own = self.n[c]
        for du in (0, 1):
            for dv in (0, 1):
                at = [slice(None)] * 3
                at[c] = slice(0, own)
                at[ua] = slice(du, du + self.n[ua])
                at[va] = slice(dv, dv + self.n[va])
                num[tuple(at)] += w * cell
                den[tuple(at)] += w
        return torch.where(den > 0, num / torch.clamp(den, min=1e-300), torch.zeros_like(num))

    def _coefficients(self, f64):
        r, n, dt = self.r, self.n, self.r.dt
        eps, sig = torch.ones(n, **f64), torch.zeros(n, **f64)
        deps = [torch.zeros(n, **f64) for _ in r.fp]
        pec = torch.zeros(n, **f64)
        cut = lambda b: tuple(slice(q0, q1) for q0, q1 in b)   # noqa: E731
        for b, e, s, dp in r.boxes:
            eps[cut(b)] = e
            sig[cut(b)] = s
            for p in range(len(dp) if dp else 0):
                deps[p][cut(b)] = dp[p]
        for b in r.pec:
            pec[cut(b)] = 1.0
        for i, j, k, mask in r.cells:
            m = torch.as_tensor(np.ascontiguousarray(mask), **f64)
            v = pec[i:i + m.shape[0], j:j + m.shape[1], k:k + m.shape[2]]
            v.copy_(torch.maximum(v, (m > 0).to(torch.float64)))
        metal = [self._average(pec, c) > 0 for c in range(3)]
        for axis, m, a0, a1, b0, b1 in r.sheets:
            ua, va = (axis + 1) % 3, (axis + 2) % 3
            U, V = r.node[ua], r.node[va]
            tol = 1e-9 * (U[-1] - U[0] + V[-1] - V[0])
            for along, lo, hi, across, c0, c1 in ((ua, a0, a1, va, b0, b1), (va, b0, b1, ua, a0, a1)):
                X, Y = r.node[along], r.node[across]
                inx = np.append((X[:-1] >= lo - tol) & (X[1:] <= hi + tol), False)
                iny = (Y >= c0 - tol) & (Y <= c1 + tol)
                at = [slice(None)] * 3
                at[axis] = slice(m, m + 1)
                hit = (self.t(inx.astype(float), along) * self.t(iny.astype(float), across)) > 0
                metal[along][tuple(at)] |= hit
        for axis, m, mu, mv in r.planes:
            ua, va = (axis + 1) % 3, (axis + 2) % 3
            for comp, mask, shape in ((ua, mu, (n[ua], n[va] + 1)), (va, mv, (n[ua] + 1, n[va]))):
                if mask is None:
                    continue
                k = torch.as_tensor(np.asarray(mask).reshape(shape) != 0, device=self.dev)
                plane = metal[comp].movedim((ua, va, axis), (0, 1, 2))[:shape[0], :shape[1], m]
                plane |= k
        self.ca, self.cb, self.J, self.beta = [], [], [], []
        tau = [1.0 / (2 * math.pi * f) for f in r.fp]
        self.k = [(1 - dt / (2 * t)) / (1 + dt / (2 * t)) for t in tau]
        for c in range(3):
            er, sg = self._average(eps, c), self._average(sig, c)
            own = (self.t(np.arange(n[c] + 1) < n[c], c) > 0) & ~metal[c]
            beta = [torch.where(own, EPS0 * self._average(dp, c) * dt / (t * (1 + dt / (2 * t))), 0.0)
                    for dp, t in zip(deps, tau)]
            einst = er * EPS0
            ports = [p for p in r.ports if p[0] == c]
            for q in ports:
                for m in range(q[3], q[4]):
                    for b in beta:
                        b[self._edge(c, q[1], q[2], m)] = 0.0
            for b in beta:
                einst = einst + 0.5 * b
            einst = torch.where(own, einst, torch.ones_like(einst))
            h = sg * dt / (2 * einst)
            ca, cb = torch.where(own, (1 - h) / (1 + h), 0.0), torch.where(own, dt / einst / (1 + h), 0.0)
            self.ca.append(ca)
            self.cb.append(cb)
            self.beta.append(beta)
            self.J.append([torch.zeros_like(b) for b in beta])
            for q, p in enumerate(r.ports):
                if p[0] != c:
                    continue
                L = float(self.d[c][p[3]:p[4]].sum())
                for m in range(p[3], p[4]):
                    at = self._edge(c, p[1], p[2], m)
                    ua, va = (c + 1) % 3, (c + 2) % 3
                    area = self.dd[ua][at[ua]] * self.dd[va][at[va]]
                    e, s, dl = float(er[at]) * EPS0, float(sg[at]), self.d[c][m]
                    re = p[6] * dl / L
                    bt = dt * dl / (2 * re * area * e) + s * dt / (2 * e)
                    ca[at], cb[at] = (1 - bt) / (1 + bt), dt / e / (1 + bt)
                    if q == r.pulse[0]:
                        self.drive = getattr(self, "drive", [])
                        self.drive.append((c, at, dt / (re * area * e * (1 + bt)) * (dl / L) * p[5]))

    @staticmethod
    def _edge(axis, n1, n2, m):
        at = [0, 0, 0]
        at[axis], at[(axis + 1) % 3], at[(axis + 2) % 3] = m, n1, n2
        return tuple(at)

    def _lines(self):
        """Edge lists of ports, voltage probes and current probes as (component, flat indices, weights)."""
        r = self.r

        def flat(ats):
            return torch.as_tensor([np.ravel_multi_index(a, self.shape) for a in ats], device=self.dev)

        def column(p):
            ats = [self._edge(p[0], p[1], p[2], m) for m in range(p[3], p[4])]
            return [(p[0], flat(ats), torch.as_tensor(self.d[p[0]][p[3]:p[4]] * p[5], device=self.dev))]

        def ring(p):
            axis, m, u0, u1, v0, v1 = p
            ua, va = (axis + 1) % 3, (axis + 2) % 3
            out = []
            for comp, run, fix, sign in ((ua, range(u0 + 1, u1 + 1), (v0, v1), (1, -1)),
                                         (va, range(v0 + 1, v1 + 1), (u1, u0), (1, -1))):
                other = va if comp == ua else ua
                for f, s in zip(fix, sign):
                    ats = []
                    for q in run:
                        at = [0, 0, 0]
                        at[axis], at[comp], at[other] = m, q, f
                        ats.append(tuple(at))
                    out.append((comp, flat(ats), s * torch.as_tensor(self.dd[comp][list(run)], device=self.dev)))
            return out

        self.lp, self.lv, self.li = ([column(p) for p in r.ports], [column(p) for p in r.vp], [ring(p) for p in r.ip])

    @staticmethod
    def _sum(F, lines):
        return [sum((F[c].reshape(-1)[at] * w).sum() for c, at, w in ln) for ln in lines]

    def _curl(self, F, out, e):
        """out_C += / -= of the curl of F; e: backward differences for E, else forward ones for H."""
        n, dth = self.n, self.r.dt / MU0
        for c in range(3):
            terms = []
            span = [slice(1, n[a]) if e else slice(0, n[a]) for a in range(3)]
            span[c] = slice(0, n[c]) if e else slice(0, n[c] + 1)
            for w, (a, f) in enumerate((((c + 1) % 3, (c + 2) % 3), ((c + 2) % 3, (c + 1) % 3))):
                shift = list(span)
                step = -1 if e else 1
                shift[a] = slice(span[a].start + step, span[a].stop + step)
                diff = (F[f][tuple(span)] - F[f][tuple(shift)]) if e else (F[f][tuple(shift)] - F[f][tuple(span)])
                inv = (self.ide if e else self.idh)[a][span[a]]
                term = diff * self.t(inv, a)
                for q, (sa, se, lo, hi, b, cc) in enumerate(self.slabs):
                    if sa != a or se != e:
                        continue
                    cut = [slice(None)] * 3
                    cut[a] = slice(lo - span[a].start, hi - span[a].start)
                    dv = diff[tuple(cut)]
                    psi = self.psi.get((c, w, q))
                    psi = cc * dv if psi is None else b * psi + cc * dv
                    self.psi[c, w, q] = psi
                    term[tuple(cut)] += psi
                terms.append(term)
            at, curl = tuple(span), terms[0] - terms[1]
            if not e:
                out[c][at] -= dth * curl
                continue
            old = out[c][at].clone() if self.J[c] else None
            for k, J in zip(self.k, self.J[c]):
                curl -= 0.5 * (1 + k) * J[at]
            out[c][at] = self.ca[c][at] * out[c][at] + self.cb[c][at] * curl
            if old is not None:
                self.old = getattr(self, "old", {})
                self.old[c] = (at, old)

    def step(self, steps):
        r = self.r
        port, amp, t0, tau = r.pulse
        for _ in range(steps):
            self._curl(self.E, self.H, False)
            cur = self._sum(self.H, self.li)
            vold = self._sum(self.E, self.lp)
            self._curl(self.H, self.E, True)
            vs = amp * math.exp(-(((self.step_no + 0.5) * r.dt - t0) / tau) ** 2)
            for c, at, w in self.drive:
                self.E[c][at] += w * vs
            for c in range(3):
                if self.J[c]:
                    at, old = self.old[c]
                    de = (self.E[c][at] - old) / r.dt
                    for k, b, J in zip(self.k, self.beta[c], self.J[c]):
                        J[at] = k * J[at] + b[at] * de
            self.rows.append((cur, vold, self._sum(self.E, self.lp), self._sum(self.E, self.lv), vs))
            self.step_no += 1

    def energy(self):
        total = 0.0
        for c in range(3):
            u, v = (c + 1) % 3, (c + 2) % 3
            vol = self.t(np.append(self.d[c], 0.0), c) * self.t(self.dd[u], u) * self.t(self.dd[v], v)
            on = self.cb[c] != 0
            w = torch.where(on, self.r.dt / torch.where(on, self.cb[c], torch.ones_like(self.cb[c])), 0.0)
            total += float((0.5 * w * self.E[c] ** 2 * vol).sum())
            vol = self.t(self.dd[c], c) * self.t(np.append(self.d[u], 0.0), u) * self.t(np.append(self.d[v], 0.0), v)
            total += float((0.5 * MU0 * self.H[c] ** 2 * vol).sum())
        return total

    def spectra(self):
        r, dt = self.r, self.r.dt
        num = lambda k: np.array([[float(v) for v in torch.stack(row[k])] if row[k] else [] for row in self.rows])  # noqa: E731
        n = np.arange(len(self.rows))
        w = 2 * np.pi * r.freq
        ph_h = np.exp(-1j * np.outer((n + 0.5) * dt, w)) * dt
        ph_e = np.exp(-1j * np.outer((n + 1.0) * dt, w)) * dt
        cur, vold, vnew, vp = (num(k) for k in range(4))
        vs = np.array([row[4] for row in self.rows])
        V = 0.5 * (vold + vnew)
        drive = np.zeros_like(V)
        drive[:, r.pulse[0]] = vs
        return {"V": V.T @ ph_h, "I": ((drive - V) / np.array([p[6] for p in r.ports])).T @ ph_h,
                "vprobe": vp.T @ ph_e if r.vp else np.array([]), "iprobe": cur.T @ ph_h if r.ip else np.array([]),
                "source": vs @ ph_h}

    def fields(self):
        return torch.cat([f.reshape(-1) for f in self.E + self.H])


def exact(case: dict, seed: int):
    out = []
    for r in _sims(Recorder(), case, seed):
        if r.unknown:
            return None
        x = Exact(r)
        x.step(case["lead"] + case["steps"])
        out.append(x)
    if case["kind"] == "batch":
        return [x.spectra() for x in out]
    x = out[0]
    if case["kind"] == "resume":
        return {"fields": x.fields(), "rest": None}
    if case["kind"] == "scene":
        return x.spectra()
    if case["kind"] == "cavity":
        return {"energy": x.energy(), "fields": x.fields(), "rest": None}
    return {"energy": x.energy(), **x.spectra()}
