"""Workloads for timing the library: what its users run, from the smallest
systems to the largest, through the public entry points.

Each case names a kind of run (a simulation stepped in one of its ensembles,
a FIRE quench, a batch of systems, sampling of profiles), its size and how
many steps are taken per call. `listed()` gives the standard ones, `draw(rng)`
others of the same ranges; `prepare` makes the inputs and the handle a program
keeps, `run` is one pass, `work` its unavoidable bytes and operations, and
`exact` the same results in 64-bit torch arithmetic.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import md_simulation_cuda_b200 as mdb
from md_simulation_cuda_b200 import workloads as wl

P_EXT = 1.0          # external pressure of the NPH and piston runs
MAX_MD_STEPS = 2_000_000_000  # batches of MD segments are stepped on and on
PAIRS = 11.8         # ordered pairs inside the cutoff per particle at rho = 0.8


def listed():
    return [
        # a driver that takes one step per call (the reference's loop), the
        # smallest system of the tests: launch latency
        dict(name="nve_900_single_steps", kind="nve", n=900, calls=20, steps=1),
        # the NVE configuration, stepped in long calls between saved frames
        dict(name="nve_4096", kind="nve", n=4096, calls=1, steps=200),
        # a small thermostatted run that samples K, U and P as it goes; odd size
        dict(name="nvt_5003_sampled", kind="nvt", n=5003, calls=5, steps=20, sample=True),
        # an interface slab of a size a study runs by the dozen
        dict(name="nvt_slab_60013", kind="slab", n=60013, calls=1, steps=100),
        # walled box under a piston (compression runs), ragged size
        dict(name="piston_20011", kind="piston", n=20011, calls=1, steps=100),
        # constant pressure, middle size
        dict(name="nph_262144", kind="nph", n=262144, calls=1, steps=100),
        # the interface slab at its full size
        dict(name="nvt_slab_1048576", kind="slab", n=1048576, calls=1, steps=200),
        # the largest single system: constant pressure
        dict(name="nph_4194304", kind="nph", n=4194304, calls=1, steps=20),
        # one quench through EnergyMinimizer: the whole call, device memory and all
        dict(name="fire_2048", kind="fire", n=2048, iters=300),
        # the mix of quenches of 256 to 16,384 particles, as one batch
        dict(name="fire_mix_512", kind="fire_batch", systems=512, n_min=256, n_max=16384,
             iters=200),
        # a temperature sweep: many small thermostatted systems as one batch
        dict(name="nvt_batch_64", kind="md_batch", systems=64, n_min=1024, n_max=16384, iters=100),
        # profiles across an interface, sampled between short runs
        dict(name="profiles_slab_131072", kind="profile", n=131072, bins=200, calls=1, steps=20),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["nve", "nvt", "slab", "piston", "nph", "fire", "fire_batch", "md_batch",
                       "profile", "slab", "nph", "nve"])
    if kind == "fire":
        return dict(kind=kind, n=logint(500, 60000), iters=logint(50, 400))
    if kind in ("fire_batch", "md_batch"):
        lo = logint(256, 2048)
        return dict(kind=kind, systems=logint(4, 256), n_min=lo, n_max=lo * rng.randint(2, 8),
                    iters=logint(20, 150))
    if kind == "profile":
        n = logint(2000, 500000)
        return dict(kind=kind, n=n, bins=rng.randint(16, 400), calls=1, steps=rng.randint(1, 30))
    n = logint(500, 3000000)
    most = max(8, min(300, 40000000 // n))
    if n < 100000 and rng.random() < 0.3:
        return dict(kind=kind, n=n, calls=rng.randint(5, 30), steps=rng.randint(1, 3))
    c = dict(kind=kind, n=n, calls=rng.randint(1, 2), steps=rng.randint(4, most))
    if n < 300000 and rng.random() < 0.3 and kind != "piston":
        c["sample"] = True
    return c


# ---------------------------------------------------------------- inputs --

def _one(case, seed):
    """Frame and configuration of a single system."""
    kind, n = case["kind"], case["n"]
    if kind in ("slab", "profile"):
        return wl.nvt_slab(n, seed=seed)
    if kind == "nph":
        return wl.nph_square(n, seed=seed)
    if kind == "piston":
        # an elongated box between soft walls, as in the piston tests
        f, Lx, Ly = wl.lattice_frame(n, 0.6, 2.0, lambda s: np.where(s < 0.5, 0.9, 0.1), 0.9,
                                     seed)
        return f, wl.config_dict(n, Lx, Ly, dt=0.001, T=0.9, barostat_mass=10000.0,
                                 k_piston=100.0)
    if kind == "fire":
        f, Lx, Ly = wl.lattice_frame(n, 0.8, 1.0, 0.65, 0.0, seed)
        f["vel"] = 0.0
        return f, wl.config_dict(n, Lx, Ly, dt=0.001, T=0.0, n_cap=n)
    f, Lx, Ly = wl.lattice_frame(n, 0.8, 1.0, 0.65, 1.0, seed)
    return f, wl.config_dict(n, Lx, Ly, dt=0.001 if kind == "nve" else 0.002, T=1.0)


def _sizes(case):
    """The sizes of a batch's systems: log-uniform, in mixed order, the same for every seed."""
    m, lo, hi = case["systems"], case["n_min"], case["n_max"]
    n = [int(round(lo * (hi / lo) ** ((k + 0.5) / m))) for k in range(m)]
    return [n[k] for k in np.random.default_rng(m).permutation(m)]


def _many(case, seed):
    """Frames and configurations of a batch."""
    rng = np.random.default_rng(seed)
    out = []
    for k, n in enumerate(_sizes(case)):
        if case["kind"] == "fire_batch":
            # the distributions of workloads.fire_mix
            fa, rho = float(rng.uniform(0.2, 0.8)), float(rng.uniform(0.6, 1.0))
            f, L = wl.random_frame(n, rho, fa, seed * 100003 + k)
            out.append((f, wl.config_dict(n, L, L, dt=0.001, T=0.0)))
        else:
            T = float(rng.uniform(0.5, 1.2))
            f, Lx, Ly = wl.lattice_frame(n, 0.8, 1.0, 0.65, T, seed * 1009 + k)
            out.append((f, wl.config_dict(n, Lx, Ly, dt=0.002, T=T)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "fire":
        f, cfg = _one(case, seed)
        s.update(frame=f, minimizer=mdb.EnergyMinimizer(cfg), params=wl.fire_params())
        return s
    if kind in ("fire_batch", "md_batch"):
        systems = _many(case, seed)
        b = mdb.Batch()
        ids = []
        for f, cfg in systems:
            if kind == "fire_batch":
                ids.append(b.add_fire(cfg, f, wl.FIRE_SETTINGS["force_tol"],
                                      wl.FIRE_SETTINGS["max_steps"], wl.fire_params()))
            else:
                ids.append(b.add_md(cfg, f, mdb.JOB_NVT, MAX_MD_STEPS))
        b.run(0)  # device memory, upload, first cell lists
        sizes = [len(f) for f, _ in systems]
        total = sum(sizes)
        s.update(batch=b, ids=ids, sizes=sizes,
                 out={k: np.empty((total, 2)) for k in ("pos", "vel", "acc")})
        return s
    f, cfg = _one(case, seed)
    s["sim"] = mdb.MDSimulation(cfg, frame=f)
    # the frame is read into pinned memory that the program keeps
    pin = torch.empty(len(f) * 64, dtype=torch.uint8, pin_memory=torch.cuda.is_available())
    s["frame"] = pin.numpy().view(mdb._lib.PARTICLE_DTYPE)
    s["pin"] = pin
    return s


# ------------------------------------------------------------------ runs --

def _steps(sim, kind, steps):
    if kind == "nve":
        sim.step_single_NVE(nsteps=steps)
    elif kind == "nph":
        sim.step_single_NPH(P_EXT, nsteps=steps)
    elif kind == "piston":
        sim.step_single_NPH_piston(P_EXT, nsteps=steps)
    else:
        sim.step_single_nose_hoover(nsteps=steps)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "fire":
        r = s["minimizer"].minimize_frame(s["frame"], wl.FIRE_SETTINGS["force_tol"],
                                          case["iters"], s["params"])
        return dict(pos=r.frame["pos"], vel=r.frame["vel"], acc=r.frame["acc"], steps=r.steps,
                    max_force=r.max_force, energy=r.potential_energy, trace=r.energy_trace)
    if kind in ("fire_batch", "md_batch"):
        b, out = s["batch"], s["out"]
        b.run(case["iters"])
        at = 0
        for i, n in zip(s["ids"], s["sizes"]):
            f = b.frame(i)
            for k in out:
                out[k][at:at + n] = f[k]
            at += n
        return out
    sim, f = s["sim"], s["frame"]
    samples = []
    for _ in range(case["calls"]):
        _steps(sim, kind, case["steps"])
        if case.get("sample"):
            samples.append([sim.cal_total_K(), sim.cal_total_U(), sim.cal_instant_pressure()])
    out = {}
    if kind == "profile":
        out["density"] = sim.get_density_profile(case["bins"])
        out["pressure"] = sim.get_pressure_profile(case["bins"])
    if samples:
        out["samples"] = np.array(samples)
    mdb._lib.check(mdb._lib.lib().mdb_sim_get_frame(sim._h, mdb._lib.frame_ptr(f), len(f)))
    o = sim.observables()
    out.update(pos=f["pos"], vel=f["vel"], acc=f["acc"], Lx=o.Lx, Ly=o.Ly, xi=o.xi, t=o.t)
    return out


def work(case):
    """One step of one particle reads its position (as a pair of floats each),
    velocity, acceleration and type and writes position, velocity and
    acceleration: 97 bytes; the pair terms are 24 operations for each ordered
    pair inside the cutoff. The frame leaves at 64 bytes a particle."""
    kind = case["kind"]
    if kind in ("fire_batch", "md_batch"):
        n = sum(_sizes(case))
        steps = case["iters"]
    else:
        n = case["n"]
        steps = case["iters"] if kind == "fire" else case["calls"] * case["steps"]
    return {"bytes": n * (97.0 * steps + 64.0), "flops": 24.0 * PAIRS * n * steps}


# ----------------------------------------------------------- 64-bit model --

class _Model:
    """One system in 64-bit torch arithmetic."""

    SKIN = 0.4
    CHUNK = 1 << 20

    def __init__(self, frame, cfg):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.cfg = cfg
        t = lambda a, d: torch.as_tensor(np.ascontiguousarray(a), device=self.dev).to(d)  # noqa: E731
        self.x = t(frame["pos"], torch.float64)
        self.v = t(frame["vel"], torch.float64)
        self.type = t(frame["type"], torch.int64)
        self.n = len(frame)
        self.L = [float(cfg["box_w_global"]), float(cfg["box_h_global"])]
        self.h0 = self.L[1]
        self.py = True
        self.dt = cfg["dt"]
        c = cfg["cutoff"]
        sig = [cfg["SIGMA_AA"], cfg["SIGMA_BB"], cfg["SIGMA_AB"]]
        eps = [cfg["EPSILON_AA"], cfg["EPSILON_BB"], cfg["EPSILON_AB"]]
        f = lambda a: torch.tensor(a, dtype=torch.float64, device=self.dev)  # noqa: E731
        self.sig2, self.eps = f([s * s for s in sig]), f(eps)
        self.rc2 = f([(c * s) ** 2 for s in sig])
        self.vc = f([4 * e * (c ** -12 - c ** -6) for e in eps])
        self.rc = c * max(sig)
        self.table = None
        self.age = 0
        self.walls = None

    def image(self, d, k):
        if k == 1 and not self.py:
            return d
        return d - self.L[k] * torch.round(d / self.L[k])

    def build(self):
        rl = self.rc + self.SKIN
        nc = [max(1, int(L / rl)) for L in self.L]
        lo = 0.0 if self.py else float(self.x[:, 1].min())
        hy = self.L[1] if self.py else max(self.L[1], float(self.x[:, 1].max())) - lo + 1e-9
        if not self.py:
            nc[1] = max(1, int(hy / rl))
        cx = (self.x[:, 0] / self.L[0] * nc[0]).long().clamp(0, nc[0] - 1)
        cy = ((self.x[:, 1] - lo) / hy * nc[1]).long().clamp(0, nc[1] - 1)
        cell = cy * nc[0] + cx
        order = torch.argsort(cell)
        count = torch.bincount(cell, minlength=nc[0] * nc[1])
        start = torch.cumsum(count, 0) - count
        most = int(count.max())
        k = torch.arange(most, device=self.dev)
        parts, width = [], 1
        for a in range(0, self.n, self.CHUNK):
            i = torch.arange(a, min(a + self.CHUNK, self.n), device=self.dev)
            cand = []
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    yy = cy[i] + dy
                    ok = torch.ones_like(yy, dtype=torch.bool)
                    if self.py:
                        yy = yy % nc[1]
                    else:
                        ok = (yy >= 0) & (yy < nc[1])
                        yy = yy.clamp(0, nc[1] - 1)
                    c = yy * nc[0] + (cx[i] + dx) % nc[0]
                    at = start[c][:, None] + k
                    good = (k < count[c][:, None]) & ok[:, None]
                    j = order[at.clamp(max=self.n - 1)]
                    cand.append(torch.where(good, j, i[:, None]))
            j = torch.cat(cand, 1)
            d0 = self.image(self.x[i, 0][:, None] - self.x[j, 0], 0)
            d1 = self.image(self.x[i, 1][:, None] - self.x[j, 1], 1)
            near = (d0 * d0 + d1 * d1 < rl * rl) & (j != i[:, None])
            m = int(near.sum(1).max())
            pick = torch.sort(near.to(torch.int8), dim=1, descending=True, stable=True)[1][:, :m]
            parts.append(torch.where(near.gather(1, pick), j.gather(1, pick), i[:, None]))
            width = max(width, m)
            del j, d0, d1, near, pick, cand
        self.table = parts
        self.age = 0

    def forces(self, energy=False):
        """Accelerations; with `energy` also U, the virial and the tensor terms."""
        if self.table is None or self.age >= 10:
            self.build()
        self.age += 1
        acc = torch.empty_like(self.x)
        U = W = 0.0
        a = 0
        for j in self.table:
            b = a + len(j)
            d0 = self.image(self.x[a:b, 0][:, None] - self.x[j, 0], 0)
            d1 = self.image(self.x[a:b, 1][:, None] - self.x[j, 1], 1)
            r2 = d0 * d0 + d1 * d1
            ti = self.type[a:b][:, None]
            p = torch.where(self.type[j] == ti, ti, 2)
            inside = (r2 > 0) & (r2 < self.rc2[p])
            i2 = torch.where(inside, 1.0 / r2, 0.0)
            s6 = (self.sig2[p] * i2) ** 3
            f = 24 * self.eps[p] * (2 * s6 * s6 - s6) * i2
            acc[a:b, 0] = (f * d0).sum(1)
            acc[a:b, 1] = (f * d1).sum(1)
            W = W + 0.5 * float((f * r2).sum())
            if energy:
                u = 4 * self.eps[p] * (s6 * s6 - s6) - torch.where(inside, self.vc[p], 0.0)
                U += 0.5 * float(u.sum())
            a = b
        self.W, self.U = W, U
        if self.walls is not None:
            k, y = self.walls, self.x[:, 1]
            up = k * (y - self.L[1]).clamp(min=0)
            acc[:, 1] += k * (-y).clamp(min=0) - up
            self.push = float(up.sum())
        return acc

    def wrap(self):
        for k in (0, 1) if self.py else (0,):
            self.x[:, k] = torch.remainder(self.x[:, k], self.L[k])

    def twice_K(self):
        return float((self.v * self.v).sum())

    def box(self, height):
        c = self.cfg
        lo = c.get("barostat_height_min_ratio", 0.6) * self.h0
        hi = c.get("barostat_height_max_ratio", 1.4) * self.h0
        return min(max(height, lo), hi)

    def start(self, kind):
        self.xi, self.p_area, self.v_piston = 0.0, 0.0, 0.0
        if kind == "piston":
            self.py, self.walls, self.table = False, self.cfg["k_piston"], None
        self.a = self.forces()
        self.k2 = self.twice_K()
        if kind == "nph":
            self.aspect = self.L[0] / self.L[1]
            self.p_now = (self.k2 + self.W) / (2 * self.L[0] * self.L[1])

    def step(self, kind):
        c, dt, h = self.cfg, self.dt, 0.5 * self.dt
        friction = lambda k2: self.xi + h * (k2 - (2.0 * self.n - 2.0) * c["T_target"]) / c["Q"]  # noqa: E731
        if kind in ("slab", "nvt", "profile", "md_batch"):
            self.xi = friction(self.k2)
            self.v += h * (self.a - self.xi * self.v)
            self.x += dt * self.v
            self.xi = friction(self.twice_K())
            self.wrap()
            self.a = self.forces()
            self.v += h * (self.a - self.xi * self.v)
            self.k2 = self.twice_K()
        elif kind == "nve":
            self.v += h * self.a
            self.x += dt * self.v
            self.wrap()
            self.a = self.forces()
            self.v += h * self.a
        elif kind == "nph":
            area = self.L[0] * self.L[1]
            p1 = self.p_area + h * (self.p_now - P_EXT)
            new = area + dt * p1 / c["barostat_mass"]
            ly = self.box(math.sqrt(new / self.aspect))
            self.L = [self.aspect * ly, ly]
            new = self.L[0] * self.L[1]
            lam = math.sqrt(new / area)
            self.v += h * self.a
            self.v /= lam
            self.x = lam * self.x + dt * self.v
            self.wrap()
            self.a = self.forces()
            self.p_area = p1 + h * ((self.twice_K() + self.W) / (2 * new) - P_EXT)
            self.v += h * self.a
            self.p_now = (self.twice_K() + self.W) / (2 * new)
        elif kind == "piston":
            M = c["barostat_mass"]
            v1 = self.v_piston + h * (self.push - P_EXT * self.L[0]) / M
            self.L[1] = self.box(self.L[1] + dt * v1)
            self.v += h * self.a
            self.x += dt * self.v
            self.wrap()
            self.a = self.forces()
            self.v += h * self.a
            self.v_piston = v1 + h * (self.push - P_EXT * self.L[0]) / M

    def sample(self):
        self.forces(energy=True)
        k2 = self.twice_K()
        return [0.5 * k2, self.U, (k2 + self.W) / (2 * self.L[0] * self.L[1])]

    def profiles(self, bins):
        n, (Lx, Ly) = self.n, self.L
        b = (self.x[:, 0] / Lx * bins).long().clamp(0, bins - 1)
        A = torch.bincount(b[self.type == 0], minlength=bins).double()
        B = torch.bincount(b[self.type != 0], minlength=bins).double()
        density = torch.where(A + B > 0, (A - B) / (A + B), 0.0)
        out = torch.zeros(3, bins, dtype=torch.float64, device=self.dev)

        def add(row, y, w):
            k = (torch.remainder(y, Ly) / Ly * bins).long().clamp(0, bins - 1)
            out[row] += torch.bincount(k.reshape(-1), weights=w.reshape(-1), minlength=bins)

        for row, (p, q) in enumerate(((0, 0), (1, 1), (0, 1))):
            add(row, self.x[:, 1], self.v[:, p] * self.v[:, q])
        self.forces()
        a = 0
        for j in self.table:
            e = a + len(j)
            d = [self.image(self.x[a:e, k][:, None] - self.x[j, k], k) for k in (0, 1)]
            r2 = d[0] * d[0] + d[1] * d[1]
            ti = self.type[a:e][:, None]
            p = torch.where(self.type[j] == ti, ti, 2)
            i2 = torch.where((r2 > 0) & (r2 < self.rc2[p]), 1.0 / r2, 0.0)
            s6 = (self.sig2[p] * i2) ** 3
            f = 24 * self.eps[p] * (2 * s6 * s6 - s6) * i2
            mid = self.x[a:e, 1][:, None] - 0.5 * d[1]
            for row, (u, w) in enumerate(((0, 0), (1, 1), (0, 1))):
                add(row, mid, 0.5 * d[u] * f * d[w])
            a = e
        return density, out.reshape(-1) * (bins / (Lx * Ly))

    def quench(self, iters, tol):
        """FIRE; returns (steps, max |a|)."""
        p = wl.FIRE_SETTINGS
        dt, alpha, streak = p["dt_init"], p["alpha0"], 0
        self.v.zero_()
        for it in range(iters):
            self.a = self.forces()
            self.v += dt * self.a
            power = float((self.v * self.a).sum())
            most = float(torch.linalg.vector_norm(self.a, dim=1).max())
            if most < tol:
                return it, most
            stop = power <= 0
            if not stop:
                streak += 1
                if streak > p["N_min"]:
                    dt, alpha = min(dt * p["f_inc"], p["dt_max"]), alpha * 0.99
            else:
                dt, alpha, streak = dt * p["f_dec"], p["alpha0"], 0
            if stop:
                self.v.zero_()
            else:
                nv = torch.linalg.vector_norm(self.v, dim=1, keepdim=True)
                na = torch.linalg.vector_norm(self.a, dim=1, keepdim=True)
                mixed = (1 - alpha) * self.v + alpha * nv / na * self.a
                self.v = torch.where((nv > 0) & (na > 0), mixed, self.v)
            self.x += dt * self.v
            self.wrap()
        return iters, most


def exact(case, seed):
    kind = case["kind"]
    if kind == "fire_batch":
        return None  # random starts with overlapping pairs: no two roundings agree for long
    if kind == "md_batch":
        out = {k: [] for k in ("pos", "vel", "acc")}
        if case["systems"] * case["iters"] > 8000:
            return None  # too long in this form
        for f, cfg in _many(case, seed):
            m = _Model(f, cfg)
            m.start(kind)
            for _ in range(case["iters"]):
                m.step(kind)
            for k, v in (("pos", m.x), ("vel", m.v), ("acc", m.a)):
                out[k].append(v)
        return {k: torch.cat(v) for k, v in out.items()}
    f, cfg = _one(case, seed)
    m = _Model(f, cfg)
    if kind == "fire":
        m.wrap()
        m.forces(energy=True)
        trace = [m.U]
        steps, most = m.quench(case["iters"], wl.FIRE_SETTINGS["force_tol"])
        m.forces(energy=True)
        trace.append(m.U)
        return dict(pos=m.x, vel=m.v, acc=m.a, steps=None, max_force=most, energy=m.U,
                    trace=trace)
    m.start(kind)
    samples = []
    for _ in range(case["calls"]):
        for _ in range(case["steps"]):
            m.step(kind)
        if case.get("sample"):
            samples.append(m.sample())
    out = {}
    if kind == "profile":
        out["density"], out["pressure"] = m.profiles(case["bins"])
    if samples:
        out["samples"] = np.array(samples)
    out.update(pos=m.x, vel=m.v, acc=m.a, Lx=m.L[0], Ly=m.L[1], xi=m.xi,
               t=case["calls"] * case["steps"] * m.dt)
    return out
