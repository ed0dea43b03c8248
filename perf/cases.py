"""The work that users of this framework have it do, as timed cases.

A case is one pass of one kind of program, written against the Python binding
(bmp-6th-sem_b200/pic_b200.py) as such a program writes it:

run       a short simulation: load the plasma (drawn on the device, or host
          points imported), advance `steps` full PIC steps, read the results
          the way a run does at its print interval.  Loading belongs to the
          pass, so a pass does the same work however often it is repeated.
phase     the particle operators alone in a fixed field (test-particle runs):
          import host points, push them, deposit, read the densities.
poisson   one stand-alone solve: set the charge density, solve from zero, read
          potential and field.
ensemble  many small instances of uneven size advanced together (a parameter
          scan), loading and results included.
deposit   the allocation-free deposit of a host framework's own device array
          of points, in no particular order.
train     one epoch of the learned warm start on pairs recorded before.
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bmp-6th-sem_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

DX = 2.5e-4
DT = 5e-11
QE = 1.602e-19
MASS = (9.109e-31, 6.6335e-26)
CHARGE = (-QE, QE)
TEMP = (2.0, 0.026)
EPS0 = 8.854e-12
N0 = 1e15
DEV = "cuda" if torch.cuda.is_available() else "cpu"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _run(nx, ny, ppc, steps, **kw):
    c = dict(kind="run", nx=nx, ny=ny, ppc=ppc, steps=steps, source="plasma", left=0.0, inner=0.0,
             blob=0.0, b0=0.01, periodic=False, energy=True, bz="uniform", warm="previous", dy=1.0)
    c.update(kw)
    return c


def listed():
    return [
        # the size of the framework's smoke run: every step is launches and latency
        dict(_run(32, 32, 8, 10, source="points", left=20.0), name="run_32"),
        # the 128^2 workload: small-scale research runs
        dict(_run(128, 128, 16, 20), name="run_128"),
        # the 512^2 workload (left electrode at 100 V, 64 particles a cell)
        dict(_run(512, 512, 64, 20, left=100.0), name="run_512"),
        # the 1024^2 headline workload: internal electrode, drifting blob
        dict(_run(1024, 1024, 100, 20, inner=200.0, blob=1000.0, b0=0.02), name="run_1024"),
        # periodic in y, odd width, a Bz profile, no energy diagnostic
        dict(_run(301, 192, 24, 20, periodic=True, energy=False, bz="profile", left=50.0, dy=1.25),
             name="run_periodic"),
        # the solve started from the trained network's guess (inference path)
        dict(_run(256, 256, 32, 10, left=100.0, warm="learned"), name="run_learned"),
        # test particles in a fixed field, odd grid, host points in, densities out
        dict(kind="phase", nx=333, ny=217, ppc=12, steps=10, b0=0.02, energy=True, dy=1.0, name="phase_333x217"),
        # the grid of the reference's own Poisson dumps
        dict(kind="poisson", nx=256, ny=256, inner=0.0, left=100.0, dy=1.0, name="poisson_257"),
        # the headline grid with its electrode
        dict(kind="poisson", nx=1024, ny=1024, inner=200.0, left=0.0, dy=1.0, name="poisson_1025"),
        # the 64-instance parameter scan, 128^2 .. 384^2
        dict(kind="ensemble", count=64, lo=128, hi=384, ppc=32, steps=10, name="ensemble_64"),
        # a framework's own points, unsorted
        dict(kind="deposit", nx=300, ny=280, n=4000000, name="deposit_4m"),
        # one epoch over 8 pairs of the 256^2 workload
        dict(kind="train", nx=256, ny=256, ppc=16, pairs=8, name="train_256"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "phase", "poisson", "poisson", "ensemble", "deposit", "train"])
    if kind == "run":
        nx, ny = _log(rng, 24, 1000), _log(rng, 24, 1000)
        if max(nx, ny) > 8 * min(nx, ny):
            ny = nx
        c = _run(nx, ny, _log(rng, 4, 100), rng.randint(8, 20), left=float(rng.randint(0, 150)),
                 b0=round(rng.uniform(0.0, 0.02), 4), energy=rng.random() < 0.7,
                 bz=rng.choice(["uniform", "uniform", "profile"]), dy=rng.choice([1.0, 1.0, 0.8, 1.3]))
        if rng.random() < 0.25:
            c.update(periodic=True, ny=(ny + 15) // 16 * 16)  # rows that multigrid can halve
        elif min(nx, ny) >= 64 and rng.random() < 0.5:
            c.update(inner=200.0, blob=float(rng.randint(1, 8) * c["ppc"]))
        elif max(nx, ny) <= 300 and rng.random() < 0.3:
            c.update(warm="learned", dy=1.0)
        if nx * ny * c["ppc"] < 400000 and not c["blob"]:
            c["source"] = rng.choice(["plasma", "points"])
        return c
    if kind == "phase":
        nx, ny = _log(rng, 32, 400), _log(rng, 32, 400)
        return dict(kind="phase", nx=nx, ny=ny, ppc=max(2, min(_log(rng, 4, 64), 1200000 // (nx * ny))),
                    steps=rng.randint(4, 12), b0=round(rng.uniform(0.005, 0.02), 4),
                    energy=rng.random() < 0.7, dy=rng.choice([1.0, 0.75]))
    if kind == "poisson":
        nx, ny = _log(rng, 32, 1024), _log(rng, 32, 1024)
        if max(nx, ny) > 4 * min(nx, ny):
            ny = nx
        return dict(kind="poisson", nx=nx, ny=ny, inner=rng.choice([0.0, 200.0]),
                    left=float(rng.randint(0, 200)), dy=rng.choice([1.0, 0.8]))
    if kind == "ensemble":
        lo = _log(rng, 48, 160)
        return dict(kind="ensemble", count=rng.randint(3, 40), lo=lo, hi=2 * lo + rng.randint(0, 60),
                    ppc=_log(rng, 8, 48), steps=rng.randint(3, 6))
    if kind == "deposit":
        return dict(kind="deposit", nx=_log(rng, 32, 700), ny=_log(rng, 32, 700), n=_log(rng, 3000, 4000000))
    n = _log(rng, 64, 256)
    return dict(kind="train", nx=n, ny=n + rng.randint(-8, 8), ppc=8, pairs=rng.randint(2, 8))


# ---------------------------------------------------------------------------
# what a program has in hand
# ---------------------------------------------------------------------------
def _rects(c):
    nx, ny = c["nx"], c["ny"]
    left = c.get("left", 0.0)
    if c.get("periodic"):
        return [(0, 0, 0, ny, left), (nx, 0, nx, ny, 0.0)]
    r = [(0, 0, 0, ny, left), (nx, 0, nx, ny, 0.0), (0, ny, nx, ny, 0.0), (0, 0, nx, 0, 0.0)]
    if c.get("inner"):
        cx, cy, h = nx // 2, ny // 2, max(2, min(nx, ny) // 32)
        r.append((cx - h, cy - h, cx + h, cy + h, c["inner"]))
    return r


def _species(c):
    sim = float(c.get("ppc", 1) * c["nx"] * c["ny"])
    return [(CHARGE[s], MASS[s], sim, N0) for s in range(2)]


def _spacing(c):
    return DX, DX * c.get("dy", 1.0)


def _config(c, **kw):
    import pic_b200 as P
    dx, dy = _spacing(c)
    kw.setdefault("deposit_energy", c.get("energy", True))
    return P.make_config(c["nx"], c["ny"], c["nx"] * dx, c["ny"] * dy, DT, _species(c), _rects(c),
                         b0=c.get("b0", 0.01), epsilon=EPS0, periodic_y=c.get("periodic", False), **kw)


def _bz_profile(c):
    """A Bz that falls off towards the right wall (a magnetic filter)."""
    x = np.linspace(0.0, 1.0, c["nx"] + 1)
    return np.tile(0.004 + 0.016 * np.exp(-((x - 0.3) / 0.2) ** 2), c["ny"] + 1)


def _points(c, s, seed):
    """Maxwellian host points, `ppc` a cell, in cell order."""
    import pic_b200 as P
    rng = np.random.default_rng([seed, s])
    dx, dy = _spacing(c)
    cells = np.repeat(np.arange(c["nx"] * c["ny"]), c["ppc"])
    n = len(cells)
    p = np.zeros(n, P.POINT_DTYPE)
    p["x"] = (cells % c["nx"] + rng.random(n)) * dx
    p["y"] = (cells // c["nx"] + rng.random(n)) * dy
    sig = math.sqrt(QE * TEMP[s] / MASS[s])
    for k in ("vx", "vy", "vz"):
        p[k] = rng.normal(0.0, sig, n)
    p["pointer"] = np.arange(n) & 0x7FFFFFFF
    return p


def _load(pic, c, seed):
    """The plasma of a run: uniform, plus the drifting blob of the large workload."""
    kw = {}
    if c.get("blob"):
        kw = dict(blob_peak_ppc=c["blob"], blob_cx=c["nx"] // 2, blob_cy=c["ny"] // 2,
                  blob_sigma=min(c["nx"], c["ny"]) / 25.6, drift_vx=1e5)
    for s in range(2):
        pic.load_plasma(s, c["ppc"], TEMP[s], seed * 2 + s, **kw)


def _modes(c, seed, amplitude):
    """A smooth random function on the nodes, zero on the four walls."""
    rng = np.random.default_rng([seed, 77])
    x, y = np.linspace(0, 1, c["nx"] + 1), np.linspace(0, 1, c["ny"] + 1)
    f = np.zeros((c["ny"] + 1, c["nx"] + 1))
    for k in range(1, 5):
        for m in range(1, 5):
            f += rng.normal() / (k * m) * np.outer(np.sin(m * np.pi * y), np.sin(k * np.pi * x))
    return amplitude * f.ravel() / np.abs(f).max()


def _scan(c, seed):
    """The instances of a parameter scan: uneven sizes, electrode voltages, Bz, densities."""
    rng = np.random.default_rng(5)  # the scan itself; the seed draws its particles
    out = []
    for _ in range(c["count"]):
        n = int(rng.integers(c["lo"], c["hi"] + 1))
        out.append(_run(n, n, c["ppc"], c["steps"], left=float(rng.uniform(50, 300)),
                        b0=float(rng.uniform(0.0, 0.02))))
    return out


def prepare(case, seed):
    import pic_b200 as P
    c = dict(case)
    k = c["kind"]
    st = dict(case=c, seed=seed)
    if k == "run":
        learned = c["warm"] == "learned"
        pic = st["pic"] = P.Pic(_config(c))
        if c["bz"] == "profile":
            pic.set_bz(_bz_profile(c))
        if learned:
            # a network trained briefly on an earlier run, as such a program keeps it
            _load(pic, c, 1)
            pic.step(0)
            pic.ws_record(8)
            for it in range(8):
                pic.step(it + 1)
            pic.ws_record(0)
            pic.ws_train(2, 1e-3)
            pic.set_poisson(warm=P.WARM_LEARNED)
        if c["source"] == "points":
            st["points"] = [_points(c, s, seed) for s in range(2)]
    elif k == "phase":
        pic = st["pic"] = P.Pic(_config(c))
        pic.set_phi(_modes(c, seed, 40.0))
        pic.update_fields()
        st["points"] = [_points(c, s, seed) for s in range(2)]
    elif k == "poisson":
        st["pic"] = P.Pic(_config(c, warm=P.WARM_ZERO))
        st["rho"] = _charge(c, seed)
    elif k == "ensemble":
        st["cases"] = _scan(c, seed)
        st["ens"] = P.Ensemble([_config(x) for x in st["cases"]])
    elif k == "deposit":
        g = torch.Generator(device=DEV).manual_seed(seed)
        pts = torch.zeros(c["n"], 7, dtype=torch.float64, device=DEV)
        pts[:, 0] = torch.rand(c["n"], generator=g, device=DEV, dtype=torch.float64) * (c["nx"] * DX)
        pts[:, 1] = torch.rand(c["n"], generator=g, device=DEV, dtype=torch.float64) * (c["ny"] * DX)
        ids = torch.arange(c["n"], dtype=torch.int32, device=DEV)
        ids[::97] = -1  # lost particles stay in such an array until it is compacted
        pts.view(torch.int32)[:, 12] = ids
        nodes = (c["nx"] + 1) * (c["ny"] + 1)
        st["points"] = pts
        st["final"] = torch.empty(nodes, dtype=torch.float64, device=DEV)
        st["rho"] = torch.empty(nodes, dtype=torch.float64, device=DEV)
        st["species"] = P.SpeciesDesc(CHARGE[0], MASS[0], float(c["n"]), N0)
    else:
        r = _run(c["nx"], c["ny"], c["ppc"], 0, left=100.0)
        pic = st["pic"] = P.Pic(_config(r))
        _load(pic, r, seed)
        pic.step(0)
        pic.ws_record(c["pairs"])
        for it in range(c["pairs"]):
            pic.step(it + 1)
        pic.ws_record(0)
        rng = np.random.default_rng([seed, 3])
        theta = pic.ws_params()
        st["theta"] = (theta * (1.0 + 0.01 * rng.standard_normal(theta.size))).astype(np.float32)
        st["scales"] = pic.ws_scales()
    return st


def _charge(c, seed):
    """rho of a quasi-neutral plasma with particle noise and a charged region."""
    rng = np.random.default_rng([seed, 9])
    n = (c["nx"] + 1) * (c["ny"] + 1)
    return (0.05 * rng.standard_normal(n) + _modes(c, seed, 0.2)) * (N0 * QE / EPS0)


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _meshes(pic, c):
    out = dict(phi=pic.phi())
    for s in range(2):
        out["density%d" % s] = pic.final_mesh(s)
    return out


def run(st):
    c = st["case"]
    k = c["kind"]
    if k == "run":
        pic = st["pic"]
        if c["source"] == "points":
            for s in range(2):
                pic.import_points(s, st["points"][s])
        else:
            _load(pic, c, st["seed"])
        for it in range(c["steps"]):
            pic.step(it)
        return _meshes(pic, c)
    if k == "phase":
        pic = st["pic"]
        for s in range(2):
            pic.import_points(s, st["points"][s])
        for it in range(c["steps"]):
            pic.particle_phase(it)
        pic.zero_rho()
        out = {}
        for s in range(2):
            pic.charge_deposition(s)
            out["density%d" % s] = pic.final_mesh(s)
            if c["energy"]:
                out["energy%d" % s] = pic.energy_mesh(s)
            out["counts%d" % s] = pic.bin_counts(s)
        out["rho"] = pic.rho()
        return out
    if k == "poisson":
        pic = st["pic"]
        pic.set_rho(st["rho"])
        pic.poisson_solve()
        return dict(phi=pic.phi(), efield=pic.efield())
    if k == "ensemble":
        ens, cases = st["ens"], st["cases"]
        for i, x in enumerate(cases):
            _load(ens[i], x, st["seed"] + i)
        for it in range(c["steps"]):
            ens.step(it)
        return [ens[i].phi() for i in range(len(cases))]
    if k == "deposit":
        import pic_b200 as P
        st["rho"].zero_()
        P._check(P.lib().pic_deposit_points_noalloc(
            st["points"].data_ptr(), c["n"], c["nx"], c["ny"], c["nx"] * DX, c["ny"] * DX,
            ctypes.byref(st["species"]), 0.0, EPS0, st["final"].data_ptr(), st["rho"].data_ptr(),
            torch.cuda.current_stream().cuda_stream))
        return dict(density=st["final"], rho=st["rho"])
    pic = st["pic"]
    pic.ws_set_params(st["theta"], *st["scales"])
    loss = pic.ws_train(1, 1e-3)
    return dict(loss=float(loss), weights=pic.ws_params())


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    c = dict(case)
    k = c["kind"]
    if k == "ensemble":
        each = [work(x) for x in _scan(c, 0)]
        return {q: sum(e[q] for e in each) for q in ("bytes", "flops")}
    nodes = (c["nx"] + 1) * (c["ny"] + 1)
    if k == "poisson":
        # rho in, phi and E out; a few hundred operations a node
        return dict(bytes=nodes * 32.0, flops=nodes * 300.0)
    if k == "deposit":
        return dict(bytes=c["n"] * 56.0 + nodes * 24.0, flops=c["n"] * 20.0)
    if k == "train":
        # forward, data and weight gradients of nine 32->32 convolutions at
        # their three sizes (4 + 4 quarter + 2 sixteenth images, less one) and
        # the two outer layers
        px = ((max(c["nx"], c["ny"]) + 4) // 4 * 4) ** 2
        conv = 2.0 * 9 * 32 * 32 * px * (3 + 4 / 4 + 2 / 16)
        outer = 2.0 * 9 * (3 + 1) * 32 * px
        return dict(bytes=c["pairs"] * nodes * 12.0, flops=c["pairs"] * 3.0 * (conv + outer))
    n = 2.0 * c["ppc"] * c["nx"] * c["ny"]
    if c.get("blob"):
        n += 2.0 * c["blob"] * 2 * math.pi * (min(c["nx"], c["ny"]) / 25.6) ** 2
    # a step reads and writes every particle (20 bytes) once, and phi
    step = n * 40.0 + (nodes * 16.0 if k == "run" else 0.0)
    return dict(bytes=c["steps"] * step + n * 20.0 + nodes * 24.0, flops=c["steps"] * (n * 80.0 + nodes * 300.0))


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _electrodes(c):
    GX, GY = c["nx"] + 1, c["ny"] + 1
    mask, val = np.zeros((GY, GX), bool), np.zeros((GY, GX))
    for x1, y1, x2, y2, v in _rects(c):
        mask[y1:y2 + 1, x1:x2 + 1] = True
        val[y1:y2 + 1, x1:x2 + 1] = v
    return torch.from_numpy(mask).to(DEV), torch.from_numpy(val).to(DEV)


def _solve64(c, rho):
    """phi of  -laplace(phi) = -rho  with the electrodes held (walls all round): CG to rounding."""
    dx, dy = _spacing(c)
    cx, cy = 1.0 / dx ** 2, 1.0 / dy ** 2
    mask, val = _electrodes(c)
    free = (~mask)[1:-1, 1:-1].to(torch.float64)

    def neg_lap(u):
        return (2 * (cx + cy) * u[1:-1, 1:-1] - cx * (u[1:-1, :-2] + u[1:-1, 2:]) -
                cy * (u[:-2, 1:-1] + u[2:, 1:-1])) * free

    x = val.clone()
    r = -rho[1:-1, 1:-1] * free - neg_lap(x)
    p = torch.zeros_like(x)
    p[1:-1, 1:-1] = r
    rr = (r * r).sum()
    stop = 1e-26 * float(rr)
    for it in range(40000):
        q = neg_lap(p)
        a = rr / (p[1:-1, 1:-1] * q).sum()
        x += a * p
        r = r - a * q
        new = (r * r).sum()
        p[1:-1, 1:-1] = r + (new / rr) * p[1:-1, 1:-1]
        rr = new
        if it % 64 == 63 and float(rr) <= stop:
            break
    return x


def _field64(c, phi):
    dx, dy = _spacing(c)
    ex, ey = torch.zeros_like(phi), torch.zeros_like(phi)
    ex[1:-1, 1:-1] = -(phi[1:-1, 2:] - phi[1:-1, :-2]) / (2 * dx)
    ey[1:-1, 1:-1] = -(phi[2:, 1:-1] - phi[:-2, 1:-1]) / (2 * dy)
    for e in (ex, ey):  # wall nodes take the nearest inner node's value
        e[:, 0], e[:, -1] = e[:, 1], e[:, -2]
        e[0], e[-1] = e[1], e[-2]
    return ex, ey


class _Particles64:
    def __init__(self, c, s, pts):
        self.c, self.s = c, s
        t = [torch.from_numpy(np.ascontiguousarray(pts[k])).to(DEV) for k in ("x", "y", "vx", "vy", "vz")]
        self.x, self.y, self.vx, self.vy, self.vz = t

    def corners(self):
        dx, dy = _spacing(self.c)
        GX = self.c["nx"] + 1
        fx, fy = self.x / dx, self.y / dy
        ix, iy = fx.floor().long().clamp(0, self.c["nx"] - 1), fy.floor().long().clamp(0, self.c["ny"] - 1)
        fx, fy = fx - ix, fy - iy
        k = iy * GX + ix
        return ((k, (1 - fx) * (1 - fy)), (k + 1, fx * (1 - fy)), (k + GX, (1 - fx) * fy), (k + GX + 1, fx * fy))

    def push(self, ex, ey, bz):
        c = self.c
        dx, dy = _spacing(c)
        h = 0.5 * CHARGE[self.s] / MASS[self.s] * DT
        at = self.corners()
        gather = lambda f: sum(w * f.reshape(-1)[k] for k, w in at)  # noqa: E731
        ax, ay, t = h * gather(ex), h * gather(ey), h * bz
        s = 2 * t / (1 + t * t)
        vxm, vym = self.vx + ax, self.vy + ay
        vxp, vyp = vxm + vym * t, vym - vxm * t
        self.vx, self.vy = vxm + vyp * s + ax, vym - vxp * s + ay
        self.x, self.y = self.x + self.vx * DT, self.y + self.vy * DT
        live = (self.x >= 0) & (self.x < c["nx"] * dx) & (self.y >= 0) & (self.y < c["ny"] * dy)
        for n in ("x", "y", "vx", "vy", "vz"):
            setattr(self, n, getattr(self, n)[live])

    def mesh(self, energy=False):
        c = self.c
        dx, dy = _spacing(c)
        area = dx * dy
        weight = N0 * (c["nx"] * dx * c["ny"] * dy) / (c["ppc"] * c["nx"] * c["ny"] * area * area) * area
        out = torch.zeros((c["ny"] + 1) * (c["nx"] + 1), dtype=torch.float64, device=DEV)
        ev = 0.5 * (self.vx ** 2 + self.vy ** 2 + self.vz ** 2) * MASS[self.s] / QE if energy else 1.0
        for k, w in self.corners():
            out.index_add_(0, k, w * ev)
        return out * weight


def exact(case, seed):
    c = dict(case)
    k = c["kind"]
    GX, GY = c.get("nx", 0) + 1, c.get("ny", 0) + 1
    if k == "poisson":
        phi = _solve64(c, torch.from_numpy(_charge(c, seed)).to(DEV).view(GY, GX))
        return dict(phi=phi.reshape(-1), efield=torch.stack(_field64(c, phi), -1).reshape(-1, 2))
    if k == "deposit":
        st = prepare(case, seed)
        pts = st["points"]
        pts = pts[pts.view(torch.int32)[:, 12] != -1].cpu().numpy()
        p = _Particles64(dict(c, ppc=1), 0, dict(x=pts[:, 0], y=pts[:, 1], vx=pts[:, 3], vy=pts[:, 4], vz=pts[:, 5]))
        m = p.mesh() * (c["nx"] * c["ny"] / c["n"])
        return dict(density=m, rho=m * (-CHARGE[0] / EPS0))
    if k == "phase":
        mask, val = _electrodes(c)
        phi = torch.from_numpy(_modes(c, seed, 40.0)).to(DEV).view(GY, GX)
        ex, ey = _field64(c, torch.where(mask, val, phi))
        out, rho = {}, 0.0
        for s in range(2):
            p = _Particles64(c, s, _points(c, s, seed))
            for _ in range(c["steps"]):
                p.push(ex, ey, c["b0"])
            out["density%d" % s] = p.mesh()
            if c["energy"]:
                out["energy%d" % s] = p.mesh(True)
            out["counts%d" % s] = None
            rho = rho + out["density%d" % s] * (-CHARGE[s] / EPS0)
        out["rho"] = rho
        return out
    if k == "run" and c["source"] == "points" and not c["periodic"] and c["bz"] == "uniform" and \
            c["nx"] * c["ny"] <= 20000:
        ps = [_Particles64(c, s, _points(c, s, seed)) for s in range(2)]
        for _ in range(c["steps"]):
            mesh = [p.mesh() for p in ps]
            rho = sum(-CHARGE[s] / EPS0 * mesh[s] for s in range(2))
            phi = _solve64(c, rho.view(GY, GX))
            ex, ey = _field64(c, phi)
            for p in ps:
                p.push(ex, ey, c["b0"])
        return dict(phi=phi.reshape(-1), density0=mesh[0], density1=mesh[1])
    return None
