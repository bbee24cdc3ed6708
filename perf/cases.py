"""Workloads of the engine as a user's program runs them, for timing.

    listed()              the named cases
    draw(rng)             another case of the same ranges
    prepare(case, seed)   the engines, positions and host buffers a program holds before the call
    run(state)            one pass through the public entry points; returns what the program reads
    work(case)            bytes and flops that one pass cannot do without
    exact(case, seed)     what run returns on a new state, from plain torch in 64 bits

Three ways of use:

    "steps"   a chunk of outer steps on the device, then a frame (positions, velocities, energies of every
              system) read into page-locked buffers: CM3D relinked with the engine's step (a chunk of one
              step), long runs, ensembles in one batch context
    "jobs"    several independent water jobs in flight at once, each in its own context and stream
              (cm3d_nb_step_async, as the serving loop advances them), then a frame of each
    "forces"  a host program that integrates itself: new positions in, nrefsh, force(1), force(2), the
              forces and energies out; one call that has to rebuild the lists and one that has not

The mixed engine forms pair and reciprocal-space terms in single precision behind a double-precision
interface, so its frames and forces are kept as a trajectory file keeps them, in single precision; the plain
FP64 engine's stay in double.
"""
from __future__ import annotations

import dataclasses
import math

import numpy as np
import torch

from cm3d_b200 import _abi, configs
from cm3d_b200.engine import Engine
from cm3d_b200.setup import build_system

ENERGIES = ("vinter", "velec", "vewald", "vbond", "vbend", "zke")


def _case(use, system, size, steps=1, **more):
    case = {"use": use, "system": system, "size": size, "steps": steps, "skin": 0.5, "density": 0.8442,
            "plain": False, "nvt": False, "tune": False}
    case.update(more)
    return case


def listed():
    return [
        # CM3D relinked with the engine's step, 864 argon atoms: every step its own call, the state read
        # back after each; launches and latency are all of it
        _case("steps", "argon", 6, name="argon-864 step"),
        # the same fluid under CM3D's Nose-Hoover chains, 2048 atoms, ten steps to a frame
        _case("steps", "argon", 8, 10, nvt=True, name="argon-2048 nvt x10"),
        # the smallest water box of the serving range, ten steps to a frame
        _case("steps", "water", 6, 10, name="water-648 x10"),
        # 4096 flexible water molecules, RESPA 0.5 / 2 fs: the mid-size single run, tuned once as long runs are
        _case("steps", "water", 16, 10, tune=True, name="water-12288 x10"),
        # 110592 molecules, kmax 21, skin 1.5 A: the largest single run
        _case("steps", "water", 48, 5, skin=1.5, tune=True, name="water-331776 x5"),
        # charged LJ binary, three interactions in one box
        _case("steps", "binary", 2048, 10, density=0.75, name="binary-2048 x10"),
        # 1024 boxes of 64 to 4096 atoms, a quarter of them charged, in one batch: ensemble runs
        _case("steps", "ensemble", 1024, 5, tune=True, name="ensemble-1024 x5"),
        # a small ragged batch
        _case("steps", "ensemble", 37, 10, name="ensemble-37 x10"),
        # four water jobs of the serving range in flight together (of 7, 11, 16 and 20 molecules an edge)
        _case("jobs", "water", 20, 10, name="water jobs x10"),
        # CM3D keeping its own integrator: 3993 atoms, an odd grid
        _case("forces", "water", 11, name="water-3993 forces"),
        # the same call on a larger box
        _case("forces", "water", 24, name="water-41472 forces"),
        # the FP64 engine, for runs that have to follow CM3D's digits
        _case("steps", "water", 8, 5, plain=True, name="water-1536 plain x5"),
    ]


def _spread(rng, lo, hi):
    """an integer of [lo, hi], uniform in its logarithm"""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _water_grid(rng, hi):
    """molecules along an edge: up to 12 placed one by one, larger boxes made of copies"""
    while True:
        n = rng.randint(5, 12) * rng.choice((1, 1, 2, 2, 3))
        if n <= hi:
            return n


def draw(rng):
    what = rng.choice(("argon", "nvt", "water", "water", "binary", "ensemble", "jobs", "forces", "forces", "plain"))
    density = round(rng.uniform(0.6, 0.9), 4)
    steps = rng.randint(2, 12)
    if what in ("argon", "nvt"):
        return _case("steps", "argon", rng.randint(5, 20), rng.choice((1, steps)), density=density, nvt=what == "nvt")
    if what == "water":
        return _case("steps", "water", _water_grid(rng, 33), steps, skin=rng.choice((0.5, 1.0)),
                     tune=rng.random() < 0.5)
    if what == "binary":
        return _case("steps", "binary", 2 * _spread(rng, 200, 5000), steps, density=density)
    if what == "ensemble":
        return _case("steps", "ensemble", _spread(rng, 10, 300), steps, tune=rng.random() < 0.5)
    if what == "jobs":
        return _case("jobs", "water", rng.randint(12, 24), steps)
    if what == "forces":
        return _case("forces", "water", _water_grid(rng, 30), skin=rng.choice((0.5, 1.0)))
    return _case("steps", "water", rng.randint(5, 10), rng.randint(1, 5), plain=True)


# ------------------------------------------------------------------- inputs
def _water(ngrid, seed, skin):
    """ngrid^3 flexible water molecules with the serving jobs' cut-off, alpha and kmax.  A box of more than 12
    molecules an edge repeats a smaller one, every molecule then shifted a little and with its own velocity."""
    L = ngrid * configs.WATER_SPACING
    rc = min(10.0, 0.45 * L)
    base = max(b for b in range(1, 13) if ngrid % b == 0)
    if base < 5:
        base = ngrid
    wl = configs.water_box(ngrid=base, seed=seed, rc=rc, alpha=3.1 / rc, kmax=int(math.ceil(7.0 * L / 49.66)),
                           skin=skin, placement="octant")
    copies = ngrid // base
    if copies == 1:
        return wl
    rng = np.random.default_rng(seed)
    at = np.stack(np.meshgrid(*[np.arange(copies)] * 3, indexing="ij"), -1).reshape(-1, 3) * wl.box
    pos = (at[:, None, :] + wl.pos[None]).reshape(-1, 3, 3)
    pos = pos + np.clip(rng.normal(scale=0.03, size=(len(pos), 1, 3)), -0.08, 0.08)
    mass = np.tile(wl.mass_amu, copies ** 3)
    (name, _, top), = wl.species
    return dataclasses.replace(wl, species=[(name, len(pos), top)], pos=pos.reshape(-1, 3), mass_amu=mass,
                               vel=configs.maxwell_boltzmann(mass, wl.temp, rng), box=L)


def _argon(ncell, density, seed):
    wl = configs.argon_fcc(ncell=ncell, density=density, seed=seed)
    rng = np.random.default_rng(seed)
    return dataclasses.replace(wl, pos=wl.pos + np.clip(rng.normal(scale=0.15, size=wl.pos.shape), -0.4, 0.4))


def _workloads(case, seed):
    """the case's systems as configs.Workload, in order"""
    size = case["size"]
    if case["system"] == "argon":
        return [_argon(size, case["density"], seed)]
    if case["system"] == "binary":
        return [configs.lj_box(size, case["density"], 1.0, seed, charged=True)]
    if case["system"] == "ensemble":
        return [configs.lj_box(m.natoms, m.density, m.tstar, m.seed + seed, charged=m.charged)
                for m in configs.ensemble_plan(size)]
    if case["use"] == "jobs":
        return [_water(n, seed + n, case["skin"]) for n in _job_grids(size)]
    return [_water(size, seed, case["skin"])]


def _job_grids(size):
    return [max(6, size * 7 // 20), size * 11 // 20, size * 16 // 20, size]


def _chains(case, temp, n):
    """one Nose-Hoover chain of three links on all atoms: {ntherm, nchain, mnh, gkt, eta, veta}; a period of
    about 0.5 ps"""
    gkt = np.array([3.0 * n * temp, temp, temp])
    return {"gkt": gkt, "mnh": gkt * 0.08 ** 2, "eta": np.zeros(3), "veta": np.array([0.1, -0.2, 0.3])}


def _system(case, wl):
    sysm = build_system(wl)
    if case["nvt"]:
        c = _chains(case, wl.temp, wl.natoms)
        sysm["iensemble"], sysm["ntherm"], sysm["nchain"] = 1, 1, 3
        sysm["ithm"] = np.zeros(wl.natoms, np.int32)
        sysm["gkt"], sysm["mnh"], sysm["nhc_eta"], sysm["nhc_veta"] = c["gkt"], c["mnh"], c["eta"], c["veta"]
    return sysm


def _moved(wl, seed):
    """Positions that a host integrator brings to two calls: the first has moved by more than half a skin
    somewhere since the call before it, the second has not since the first; two such pairs in turn."""
    rng = np.random.default_rng([seed, 7])
    frames = []
    for far in (0.3, 0.6):
        p = wl.pos.reshape(-1, 3, 3)
        shift = rng.normal(size=(len(p), 1, 3))
        p = p + far * shift / np.linalg.norm(shift, axis=2, keepdims=True)
        pair = [p + np.clip(rng.normal(scale=0.03, size=p.shape), -0.06, 0.06) for _ in range(2)]
        frames.append([np.ascontiguousarray(q.reshape(-1, 3).T) for q in pair])
    return frames


def _pinned(n):
    return torch.empty((3, n), dtype=torch.float64, pin_memory=torch.cuda.is_available())


def prepare(case, seed):
    wls = _workloads(case, seed)
    systems = [_system(case, wl) for wl in wls]
    mode = _abi.PLAIN_FP64 if case["plain"] else _abi.MIXED
    engines = []
    for group in ([[s] for s in systems] if case["use"] == "jobs" else [systems]):
        eng = Engine(group if len(group) > 1 else group[0], mode=mode)
        eng.step_init()
        if case["tune"]:
            eng.autotune()
        engines.append(eng)
    state = {"case": case, "engines": engines, "istep": 1,
             "frames": [(_pinned(e.n), _pinned(e.n)) for e in engines]}
    if case["use"] == "forces":
        state["moved"] = _moved(wls[0], seed)
    elif case["use"] == "steps" and case["steps"] == 1:
        pos, vel = state["frames"][0]
        engines[0].set_host_outputs(pos.numpy(), vel.numpy())
    return state


# --------------------------------------------------------------------- runs
def _kept(case, t):
    return t.clone() if case["plain"] else t.float()


def _energies(case, eng):
    e = eng.energies_table()
    return _kept(case, torch.from_numpy(np.stack([e[k] for k in ENERGIES], axis=1)))


def run(state):
    case, engines, istep = state["case"], state["engines"], state["istep"]
    if case["use"] == "forces":
        return _run_forces(state)
    steps = case["steps"]
    state["istep"] += steps
    if case["use"] == "jobs":
        for eng in engines:
            eng.step_async(istep, steps)
        for eng in engines:
            eng.step_wait()
    else:
        engines[0].step(istep, steps)
    out = []
    for eng, (pos, vel) in zip(engines, state["frames"]):
        if steps > 1 or case["use"] == "jobs":
            eng.positions(out=pos.numpy())
            eng.velocities(out=vel.numpy())
        out.append({"pos": _kept(case, pos), "vel": _kept(case, vel), "energies": _energies(case, eng)})
    return out


def _run_forces(state):
    case, eng = state["case"], state["engines"][0]
    far, near = state["frames"][0]
    frames = state["moved"][state["istep"] // 20 % 2]
    out = []
    for p in frames:
        # ten steps between list tests: no pull-back of atoms that moved early
        state["istep"] += 10
        eng.set_positions(p)
        eng.nrefsh(state["istep"])
        eng.force(1)
        eng.force(2)
        eng.forces(_abi.FXL, out=far.numpy())
        eng.forces(_abi.FXA, out=near.numpy())
        out.append({"fxl": _kept(case, far), "fxa": _kept(case, near), "energies": _energies(case, eng)})
    return out


# --------------------------------------------------------------------- work
def _sizes(case):
    """(atoms, volume, cut-off, kmax or 0, charged) of each system"""
    if case["system"] == "ensemble":
        members = [(m.natoms, m.density, m.charged) for m in configs.ensemble_plan(case["size"])]
    elif case["system"] == "binary":
        members = [(case["size"], case["density"], True)]
    elif case["system"] == "argon":
        members = [(4 * case["size"] ** 3, case["density"], False)]
    else:
        out = []
        for n in (_job_grids(case["size"]) if case["use"] == "jobs" else [case["size"]]):
            L = n * configs.WATER_SPACING
            out.append((3 * n ** 3, L ** 3, min(10.0, 0.45 * L), int(math.ceil(7.0 * L / 49.66)), True))
        return out
    out = []
    for n, density, charged in members:
        vol = n / density * configs.ARGON["sig"] ** 3
        out.append((n, vol, min(2.5 * configs.ARGON["sig"], 0.45 * vol ** (1 / 3)), 5 if charged else 0, charged))
    return out


def work(case):
    """Per step: positions, velocities and masses in, positions and velocities out; every pair inside the
    cut-off once (57 flops of an electrostatic pair, 14 more where it is an LJ pair, 55 of an LJ-only pair); a
    sum over the k-vectors for the structure factors (4 flops) and one for the forces (8 flops) per charge."""
    nbytes = flops = 0.0
    for n, vol, rc, kmax, charged in _sizes(case):
        pairs = 0.5 * n * n / vol * 4.0 / 3.0 * math.pi * rc ** 3
        lj = 1.0 / 9.0 if case["system"] == "water" else 1.0
        kvec = 2.0 / 3.0 * math.pi * kmax ** 3
        flops += pairs * ((57.0 + 14.0 * lj) if charged else 55.0) + 12.0 * kvec * n
        nbytes += 8.0 * 13.0 * n
    calls = 2 if case["use"] == "forces" else case["steps"]
    return {"bytes": calls * nbytes, "flops": calls * flops}


# -------------------------------------------------------------------- exact
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _interp(t, k, p):
    a, b, c = t[k - 1], t[k], t[k + 1]
    return b + 0.5 * p * (c - a + p * (a - 2.0 * b + c))


class _Exact:
    """One system in 64 bits: CM3D's tabulated LJ and erfc terms, its Ewald sum with the excluded-pair
    correction, harmonic bonds and bends, the RESPA step with nrefsh's pull-back and Nose-Hoover chains."""

    def __init__(self, case, wl):
        dev = _device()

        def put(a):
            return torch.tensor(np.asarray(a), dtype=torch.float64, device=dev)

        self.case, self.L = case, float(wl.box)
        self.pos, self.vel = put(wl.pos), put(wl.vel)
        self.n = n = wl.natoms
        self.mass = put(wl.mass_amu) * configs.MCONV
        kw = wl.keywords
        self.dt = float(kw["dt"]) * configs.TCONV
        self.ninner = int(kw["nres_intra"])
        self.skin = float(kw["skin"])
        self.water = case["system"] == "water"
        self.shift = int(kw.get("shift", 0))
        self.ntable = int(kw.get("ntable", 500))
        if self.water:
            w = configs.WATER
            q = np.tile([w["q_o"], w["q_h"], w["q_h"]], n // 3)
            self.mol = torch.arange(n, device=dev) // 3
            self.lj_atom = torch.arange(n, device=dev) % 3 == 0
            eps, sig, rmin = w["eps_oo"], w["sig_oo"], 1.8
        else:
            charge = 0.5 if len(wl.species) == 2 else 0.0
            q = np.concatenate([np.full(m, s * charge) for (_, m, _), s in zip(wl.species, (1.0, -1.0))])
            self.mol = torch.arange(n, device=dev)
            self.lj_atom = torch.ones(n, dtype=torch.bool, device=dev)
            eps, sig = configs.ARGON["eps"], configs.ARGON["sig"]
            rmin = 0.55 * sig
        self.charged = bool(np.any(q))
        self.q = put(q) * math.sqrt(configs.CCONV)
        if self.charged:
            self.rc, self.alpha, self.kmax = float(kw["rcute_max"]), float(kw["alp_ewald"]), int(kw["kmax"])
        else:
            self.rc = 2.5 * sig if case["system"] == "argon" else min(2.5 * sig, 0.45 * self.L)
        # tables uniform in r^2: V and (dV/dr) / r
        self.rmin2_lj, self.dx_lj, r = self._grid(rmin, put)
        s6 = (sig / r) ** 6
        self.v_lj, self.f_lj = 4 * eps * (s6 * s6 - s6), 4 * eps * (6 * s6 - 12 * s6 * s6) / (r * r)
        if self.shift:
            self.v_lj = self.v_lj - self.v_lj[self.ntable - 3]
        if self.charged:
            self.rmin2_el, self.dx_el, r = self._grid(1.0, put)
            erfc = torch.special.erfc(self.alpha * r)
            self.v_el = erfc / r
            self.f_el = (-erfc / (r * r) - 2 * self.alpha / math.sqrt(math.pi) * torch.exp(-(self.alpha * r) ** 2) / r) / r
            if self.shift:
                self.v_el = self.v_el - self.v_el[self.ntable - 3]
        self.energy = {}
        self.chains = {k: v.copy() for k, v in _chains(case, wl.temp, n).items()} if case["nvt"] else None

    def _grid(self, rmin, put):
        dx = (self.ntable - 3.0) / (self.rc ** 2 - rmin ** 2)
        return rmin ** 2, dx, torch.sqrt(put(np.arange(self.ntable)) / dx + rmin ** 2)

    def _near(self):
        """(atoms, candidate neighbours) index tensors that together cover every pair inside the cut-off"""
        nc = int(self.L // self.rc)
        every = torch.arange(self.n, device=self.pos.device)
        if nc < 4 or self.n < 20000:
            for a in range(0, self.n, 2048):
                yield every[a:a + 2048], every
            return
        cell = torch.floor((self.pos / self.L % 1.0) * nc).long().clamp(max=nc - 1)
        cell = (cell[:, 0] * nc + cell[:, 1]) * nc + cell[:, 2]
        order = torch.argsort(cell)
        first = torch.searchsorted(cell[order], torch.arange(nc ** 3 + 1, device=cell.device)).tolist()
        off = [(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1)]
        for c in range(nc ** 3):
            x, y, z = c // (nc * nc), c // nc % nc, c % nc
            around = [((x + i) % nc * nc + (y + j) % nc) * nc + (z + k) % nc for i, j, k in off]
            if first[c + 1] > first[c]:
                yield order[first[c]:first[c + 1]], torch.cat([order[first[k]:first[k + 1]] for k in around])

    def _table(self, r2, rmin2, dx):
        p = (r2 - rmin2) * dx
        low = p < 1.0
        k = torch.where(low, torch.ones_like(p), p.floor()).long().clamp(max=self.ntable - 2)
        return k, torch.where(low, torch.zeros_like(p), p - k)

    def _pairs(self, f):
        vlj = vel = 0.0
        for i, j in self._near():
            d = self.pos[i][:, None] - self.pos[j][None]
            d = d - self.L * torch.round(d / self.L)
            r2 = (d * d).sum(-1)
            a, b = torch.nonzero((r2 < self.rc ** 2) & (self.mol[i][:, None] != self.mol[j][None]), as_tuple=True)
            d, r2, i, j = d[a, b], r2[a, b], i[a], j[b]
            g = torch.zeros_like(r2)
            lj = self.lj_atom[i] & self.lj_atom[j]
            k, p = self._table(r2, self.rmin2_lj, self.dx_lj)
            g = torch.where(lj, _interp(self.f_lj, k, p), g)
            vlj = vlj + 0.5 * torch.where(lj, _interp(self.v_lj, k, p), 0.0).sum()
            if self.charged:
                k, p = self._table(r2, self.rmin2_el, self.dx_el)
                qq = self.q[i] * self.q[j]
                g = g + qq * _interp(self.f_el, k, p)
                vel = vel + 0.5 * (qq * _interp(self.v_el, k, p)).sum()
            f.index_add_(0, i, -d * g[:, None])
        self.energy["vinter"], self.energy["velec"] = float(vlj), float(vel)

    def _ewald(self, f):
        """reciprocal space, background and self terms, and the correction of the excluded pairs"""
        kmax, vol = self.kmax, self.L ** 3
        g = np.arange(-kmax, kmax + 1)
        a, b, c = (t.ravel() for t in np.meshgrid(g[kmax:], g, g, indexing="ij"))
        half = (a * a + b * b + c * c <= kmax * kmax) & ((a > 0) | (b > 0) | ((b == 0) & (c > 0)))
        kv = torch.tensor(np.stack([a[half], b[half], c[half]], 1), dtype=torch.float64, device=self.pos.device)
        kv = kv * (2 * math.pi / self.L)
        g2 = (kv * kv).sum(1)
        pre = torch.exp(-g2 / (4 * self.alpha ** 2)) / (vol * g2)
        tq = self.q * math.sqrt(4 * math.pi)
        vk = 0.0
        step = max(1, int(2e8) // self.n)
        for k0 in range(0, len(kv), step):
            k, w = kv[k0:k0 + step], pre[k0:k0 + step]
            phase = self.pos @ k.T
            cos, sin = torch.cos(phase), torch.sin(phase)
            re, im = tq @ cos, tq @ sin
            vk = vk + (w * (re * re + im * im)).sum()
            f += tq[:, None] * ((sin * (2 * w * re) - cos * (2 * w * im)) @ k)
        ve = vk - self.alpha / math.sqrt(math.pi) * (self.q * self.q).sum() \
            - 0.5 * self.q.sum() ** 2 * math.pi / self.alpha ** 2 / vol
        if self.water:
            p, q = self.pos.view(-1, 3, 3), self.q.view(-1, 3)
            out = f.view(-1, 3, 3)
            for i, j in ((0, 1), (0, 2), (1, 2)):
                d = p[:, i] - p[:, j]
                r = d.norm(dim=1)
                qq = q[:, i] * q[:, j] / r
                erf = torch.special.erf(self.alpha * r)
                ve = ve - (qq * erf).sum()
                dv = -qq * (erf / r - 2 * self.alpha / math.sqrt(math.pi) * torch.exp(-(self.alpha * r) ** 2)) / r
                out[:, i] += dv[:, None] * d
                out[:, j] -= dv[:, None] * d
        self.energy["vewald"] = float(ve)

    def level1(self):
        """accelerations of force(1)"""
        f = torch.zeros_like(self.pos)
        self.energy["vewald"] = 0.0
        self._pairs(f)
        if self.charged:
            self._ewald(f)
        return f / self.mass[:, None]

    def level2(self):
        """accelerations of force(2): bonds and bends; their energies on the side"""
        f = torch.zeros_like(self.pos)
        self.energy["vbond"] = self.energy["vbend"] = 0.0
        if self.water:
            w = configs.WATER
            p, out = self.pos.view(-1, 3, 3), f.view(-1, 3, 3)
            u = [p[:, j] - p[:, 0] for j in (1, 2)]
            r = [x.norm(dim=1) for x in u]
            vb = 0.0
            for j in (0, 1):
                dr = r[j] - w["r0"]
                vb = vb + (0.5 * w["k_bond"] * dr * dr).sum()
                t = (w["k_bond"] * dr / r[j])[:, None] * u[j]
                out[:, j + 1] -= t
                out[:, 0] += t
            cos = (u[0] * u[1]).sum(1) / (r[0] * r[1])
            th = torch.arccos(cos)
            dth = th - math.radians(w["theta0"])
            dudc = (-w["k_bend"] * dth / torch.sqrt(1 - cos * cos))[:, None]
            for j, o in ((0, 1), (1, 0)):
                t = dudc * (cos[:, None] * u[j] / (r[j] ** 2)[:, None] - u[o] / (r[0] * r[1])[:, None])
                out[:, j + 1] += t
                out[:, 0] -= t
            self.energy["vbond"], self.energy["vbend"] = float(vb), float((0.5 * w["k_bend"] * dth * dth).sum())
        return f / self.mass[:, None]

    def _thermostat(self, h):
        c = self.chains
        v, m, g = c["veta"], c["mnh"], c["gkt"]
        self.vel *= math.exp(-h * v[0])
        for i in (0, 1):
            v[i] *= math.exp(-h * v[i + 1])
        force = np.array([(float((self.mass[:, None] * self.vel ** 2).sum()) - g[0]) / m[0],
                          (m[0] * v[0] ** 2 - g[1]) / m[1], (m[1] * v[1] ** 2 - g[2]) / m[2]])
        v += h * force
        v[0] += h * force[0]
        for i in (1, 2):
            v[i] += h * (m[i - 1] * v[i - 1] ** 2 - g[i]) / m[i]
        for i in (1, 0):
            v[i] *= math.exp(-h * v[i + 1])
        self.vel *= math.exp(-h * v[0])

    def steps(self, nsteps):
        """velocity Verlet with force(2) in the inner level, from step_init on"""
        last, listed_at = 0, self.pos.clone()
        fl, fa = self.level1(), self.level2()
        h = 0.5 * self.dt / self.ninner
        for istep in range(1, nsteps + 1):
            self.vel += 0.5 * self.dt * fl
            for _ in range(self.ninner):
                self.vel += h * fa
                self.pos += h * self.vel
                if self.chains:
                    self._thermostat(h)
                self.pos += h * self.vel
                fa = self.level2()
                self.vel += h * fa
            moved = self.pos - listed_at
            d2 = (moved * moved).sum(1)
            far = d2 > 0.25 * self.skin ** 2
            if bool(far.any()):
                if istep - last < 3:
                    pulled = listed_at + moved * (0.25 * self.skin ** 2 / d2)[:, None]
                    self.pos = torch.where(far[:, None], pulled, self.pos)
                last, listed_at = istep, self.pos.clone()
            fl = self.level1()
            self.vel += 0.5 * self.dt * fl

    def energies(self):
        # the bonded energies are those of the positions force(1) saw
        self.level2()
        self.energy["zke"] = 0.5 * float((self.mass[:, None] * self.vel ** 2).sum())
        return [self.energy[k] for k in ENERGIES]


def exact(case, seed):
    wls = _workloads(case, seed)
    if case["use"] == "forces":
        out = []
        x = _Exact(case, wls[0])
        for p in _moved(wls[0], seed)[0]:
            x.pos = torch.tensor(p.T.copy(), dtype=torch.float64, device=x.pos.device)
            fl, fa = x.level1(), x.level2()
            out.append({"fxl": fl.T.cpu(), "fxa": fa.T.cpu(), "energies": torch.tensor([x.energies()], dtype=torch.float64)})
        return out
    found = []
    for wl in wls:
        x = _Exact(case, wl)
        x.steps(case["steps"])
        found.append(x)
    groups = [[x] for x in found] if case["use"] == "jobs" else [found]
    return [{"pos": torch.cat([x.pos for x in g]).T.contiguous().cpu(), "vel": torch.cat([x.vel for x in g]).T.contiguous().cpu(),
             "energies": torch.tensor([x.energies() for x in g], dtype=torch.float64)} for g in groups]
