"""Performance cases of the Lennard-Jones framework: what a simulation program has it do.

Every case goes through the public Python entry points (``MDSystem``, ``Batch``,
``Server``) and returns whole per-atom arrays.  Inputs are made from a seed
alone, with numpy: an fcc lattice of the case's density with every site moved
by a normal displacement, vacancies down to the wanted atom count (so counts
are not multiples of anything), and Maxwell-Boltzmann velocities.  ``order``
says how particles are numbered: "lattice" (neighbours have nearby numbers, as
after a lattice start) or "shuffled" (as in a file, or after long diffusion).

Kinds of case:

  run      whole steps between two trajectory frames, then the frame is read:
           velocity Verlet or the Gaussian thermostat, one LJ type or the
           Kob-Andersen mixture, any box shape
  driver   the reference drivers' loop: one call per phase and the temperature
           read by the host every step
  list     the Verlet neighbour list: rebuild, five steps, rebuild, ...
  energy   single points: cell list, forces and potential energy of a
           configuration, force sums in 32 or 64 bits
  relax    steepest descent of a fresh overlapping random start
  gr       the pair distribution function of a configuration
  batch    many independent systems of uneven size advanced together
  serve    a burst of jobs of different size and length through the job server
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from particlebase_b200 import workloads as W
from particlebase_b200.batch import Batch
from particlebase_b200.md import from_system
from particlebase_b200.serve import Server

DT = 0.005
RC = 2.5
RSTEP = 0.02   # g(r) bin width
SKIN = 0.4     # neighbour-list skin
EVERY = 5      # steps between list rebuilds
ALPHA, MAX_DISP = 1e-3, 0.02  # steepest descent


def listed() -> list[dict]:
    return [
        # the smallest periodic system of interest, NVE: a step is all latency
        dict(name="nve_500", kind="run", n=500, density=0.8442, shape="cube", mixture=False,
             gaussian=False, order="lattice", steps=50),
        # the plain NVE system of the reduced-density benchmark
        dict(name="nve_4000", kind="run", n=4000, density=0.8442, shape="cube", mixture=False,
             gaussian=False, order="lattice", steps=50),
        # a mid-size slab (long in x and y) with vacancies, NVE, particles out of order
        dict(name="nve_slab_131k", kind="run", n=131071, density=0.75, shape="slab",
             mixture=False, gaussian=False, order="shuffled", steps=50),
        # the thermostatted system at scale; a frame every 50 steps
        dict(name="gauss_1m", kind="run", n=1048576, density=0.8442, shape="cube",
             mixture=False, gaussian=True, order="lattice", steps=50),
        # the binary glass former at large N, particles numbered at random
        dict(name="mixture_2m", kind="run", n=2048000, density=1.2, shape="cube",
             mixture=True, gaussian=True, order="shuffled", steps=20),
        # a driver program that calls every phase and watches the temperature
        dict(name="driver_30k", kind="driver", n=30011, density=0.8442, shape="cube",
             gaussian=True, order="lattice", steps=20),
        # neighbour lists kept for five steps at a time
        dict(name="list_108k", kind="list", n=107999, density=0.8442, shape="cube",
             order="lattice", steps=20),
        # potential energy and forces of a configuration, 64-bit force sums
        dict(name="energy_250k", kind="energy", n=250047, density=0.8, shape="rod", acc64=True,
             mixture=False, order="lattice"),
        # relaxation of a random start of the mixture before dynamics
        dict(name="relax_100k", kind="relax", n=100003, density=1.2, steps=20),
        # pair distribution of a frame, out to half the box
        dict(name="gr_32k", kind="gr", n=32000, density=0.8442, order="lattice"),
        # uneven replicas in one batch
        dict(name="replicas_60", kind="batch", count=60, n_lo=500, n_hi=50000, gaussian=True,
             steps=50),
        # a burst of jobs at the server
        dict(name="serve_20", kind="serve", count=20, n_lo=1000, n_hi=50000, s_lo=30, s_hi=100),
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["run", "run", "run", "run", "driver", "list", "energy", "relax", "gr",
                       "batch", "batch", "serve"])
    order = rng.choice(["lattice", "shuffled"])
    shape = rng.choice(["cube", "slab", "rod"])
    rho = round(rng.uniform(0.70, 0.90), 4)
    if kind == "run":
        mixture = rng.random() < 0.3
        return dict(kind=kind, n=_log_int(rng, 1000 if mixture else 500, 1_200_000),
                    density=round(rng.uniform(1.15, 1.25), 4) if mixture else rho,
                    shape=shape, mixture=mixture, gaussian=rng.random() < 0.5, order=order,
                    steps=20 if mixture else 50)
    if kind == "driver":
        return dict(kind=kind, n=_log_int(rng, 500, 200_000), density=rho, shape=shape,
                    gaussian=rng.random() < 0.5, order=order, steps=20)
    if kind == "list":
        return dict(kind=kind, n=_log_int(rng, 2000, 500_000), density=rho, shape="cube",
                    order=order, steps=20)
    if kind == "energy":
        mixture = rng.random() < 0.3
        return dict(kind=kind, n=_log_int(rng, 1000, 1_000_000), density=rho, shape=shape,
                    acc64=rng.random() < 0.5, mixture=mixture, order=order)
    if kind == "relax":
        return dict(kind=kind, n=_log_int(rng, 1000, 300_000), density=1.2, steps=20)
    if kind == "gr":
        return dict(kind=kind, n=_log_int(rng, 1000, 50_000), density=rho, order=order)
    if kind == "batch":
        hi = _log_int(rng, 1000, 50_000)
        return dict(kind=kind, count=rng.randint(2, 60), n_lo=500, n_hi=hi,
                    gaussian=rng.random() < 0.5, steps=50)
    return dict(kind=kind, count=rng.randint(2, 20), n_lo=1000, n_hi=_log_int(rng, 2000, 50_000),
                s_lo=30, s_hi=100)


# ---- inputs ------------------------------------------------------------------


def _cells(n: int, density: float, shape: str, rc: float) -> tuple[tuple[int, int, int], float]:
    """fcc unit cells per axis with at least n sites, every axis at least three
    cutoffs long; "slab" is flat in z, "rod" long in z.  The lattice constant is
    such that n atoms in the box have the wanted density."""
    ax = {"cube": (1.0, 1.0, 1.0), "slab": (2.0, 1.5, 0.5), "rod": (0.7, 0.8, 1.9)}[shape]
    scale = (n / 4.0 / (ax[0] * ax[1] * ax[2])) ** (1.0 / 3.0)
    k = [max(1, int(round(scale * a))) for a in ax]
    least = int(math.ceil(3.02 * rc * (density / 4.0) ** (1.0 / 3.0)))
    k = [max(least, x) for x in k]
    while 4 * k[0] * k[1] * k[2] < n:
        k[int(np.argmin([x / a for x, a in zip(k, ax)]))] += 1
    sites = 4 * k[0] * k[1] * k[2]
    a = (n / density / (sites / 4)) ** (1.0 / 3.0)
    while min(k) * a < 3.02 * rc:  # vacancies shrink the box: fewer of them
        n = min(sites, n + max(1, n // 50))
        a = (n / density / (sites / 4)) ** (1.0 / 3.0)
        if n == sites:
            break
    return (k[0], k[1], k[2]), max(a, 3.02 * rc / min(k))


def _fluid(n: int, density: float, shape: str, mixture: bool, order: str, temperature: float,
           rng: np.random.Generator, cell: float = RC) -> W.LJSystem:
    k, a = _cells(n, density, shape, cell)
    L = np.array([np.float32(x * a) for x in k], np.float64)
    basis = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]]) + 0.25
    g = np.stack(np.meshgrid(*[np.arange(x) for x in k], indexing="ij"), -1).reshape(-1, 1, 3)
    r = ((g + basis) / np.array(k) * L).reshape(-1, 3)
    if len(r) > n:
        r = r[np.sort(rng.permutation(len(r))[:n])]
    if order == "shuffled":
        r = r[rng.permutation(n)]
    r = np.mod(r + rng.normal(0.0, 0.06 if not mixture else 0.03, r.shape), L)
    r = r.astype(np.float32)
    r = np.where(r >= L.astype(np.float32), np.float32(0), r).astype(np.float64)
    types = np.zeros(n, np.uint32)
    if mixture:
        types[rng.permutation(n)[: n // 5]] = 1
    lj = W.kob_andersen_lj() if mixture else W.single_type_lj(RC)
    box = np.array([0, L[0], 0, L[1], 0, L[2]], np.float32)
    return W.LJSystem(box=box, r=r, v=W.maxwell_boltzmann(n, temperature, rng), mass=np.ones(n),
                      types=types, lj=lj, rc=RC, temperature=temperature)


def _sizes(case: dict) -> list[int]:
    """Log-uniform sizes over the case's range, the same for every seed."""
    lo, hi, m = math.log(case["n_lo"]), math.log(case["n_hi"]), case["count"]
    sizes = [int(round(math.exp(lo + (k + 0.5) / m * (hi - lo)))) for k in range(m)]
    random.Random(m).shuffle(sizes)
    return sizes


def _replicas(case: dict, seed: int) -> list[W.LJSystem]:
    rng = np.random.default_rng([seed, case["count"]])
    return [_fluid(n, float(rng.uniform(0.70, 0.90)), "cube", False, "lattice",
                   float(rng.uniform(0.7, 1.5)), rng) for n in _sizes(case)]


def _jobs(case: dict, seed: int) -> list[tuple[W.LJSystem, int]]:
    """Jobs of uneven size, and their step counts."""
    lo, hi = case["s_lo"], case["s_hi"]
    steps = random.Random(case["count"] + 1)
    return [(s, steps.randint(lo, hi)) for s in _replicas(case, seed)]


def _system(case: dict, seed: int) -> W.LJSystem:
    rng = np.random.default_rng([seed, case["n"]])
    kind = case["kind"]
    if kind == "relax":
        return W.kob_andersen_random(case["n"], case["density"], 0.8, int(rng.integers(1 << 31)))
    return _fluid(case["n"], case["density"], case.get("shape", "cube"),
                  case.get("mixture", False), case["order"],
                  0.8 if case.get("mixture", False) else 0.72, rng,
                  cell=RC + SKIN if kind == "list" else RC)


def prepare(case: dict, seed: int):
    kind = case["kind"]
    if kind == "batch":
        systems = _replicas(case, seed)
        return case, Batch.from_systems(systems, gaussian=case["gaussian"], dt=DT)
    if kind == "serve":
        jobs = _jobs(case, seed)
        return case, jobs, Server(hbm_budget=4e9, gaussian=True)
    s = _system(case, seed)
    p = from_system(s, gaussian=case.get("gaussian", False), fp64_forces=case.get("acc64", False),
                    cell_rmax=RC + SKIN if kind == "list" else None)
    if kind == "list":
        p.useNList(SKIN)
    if kind == "relax":
        r4 = np.zeros((s.n, 4), np.float32)
        r4[:, :3] = s.r
        return case, p, r4
    return case, p


def run(state):
    case, kind = state[0], state[0]["kind"]
    p = state[-1]
    if kind == "run":
        p.run(DT, case["steps"])
        if case["gaussian"]:
            return {"r": p.get("r"), "F": p.get("F")}
        return {"r": p.get("r"), "v": p.get("v")}
    if kind == "driver":
        T = np.empty(case["steps"], np.float32)
        for k in range(case["steps"]):
            p.calcBlockID()
            p.calcForce()
            T[k] = p.calcTemp()
            p.TimeEvolution(DT)
            p.treatPeriodicCondition()
        return {"r": p.getPosition(), "F": p.getForce(), "T": T}
    if kind == "list":
        for _ in range(case["steps"] // EVERY):
            p.makeNList()
            p.run(DT, EVERY)
        return {"r": p.get("r"), "v": p.get("v")}
    if kind == "energy":
        p.calcBlockID()
        p.calcForce(energy=True)
        e = p.sums()
        return {"F": p.get("F"), "E": np.array([e["pe"], e["virial"], e["mv2"]], np.float32)}
    if kind == "relax":
        _, p, r4 = state
        p.set("r", r4)
        p.minimize(case["steps"], ALPHA, MAX_DISP)
        return {"r": p.get("r")}
    if kind == "gr":
        return p.gr_counts(RSTEP, 0.5 * float(p.cell[1] - p.cell[0]))
    if kind == "batch":
        p.run(case["steps"])
        return [p.get(k, "r") for k in range(p.nsys)]
    _, jobs, srv = state
    ids = [srv.submit(s, steps, DT) for s, steps in jobs]
    srv.drain()
    out = []
    for i in ids:
        r, _, F = srv.result(i)
        out += [r, F]
        srv.release(i)
    return out


# ---- what a pass cannot do without ----------------------------------------------


def work(case: dict) -> dict:
    """Bytes and operations of one pass.  A step reads and writes positions,
    velocities and both forces of every atom once, and evaluates every pair
    inside the cutoff once (about 8 operations for the distance, 14 for the
    force); a result read back crosses once more."""
    kind = case["kind"]
    if kind == "gr":
        n = case["n"]
        return {"bytes": 16.0 * n, "flops": 12.0 * n * (n - 1) / 2}
    if kind in ("batch", "serve"):
        steps = case["steps"] if kind == "batch" else (case["s_lo"] + case["s_hi"]) / 2
        n, rho, gaussian = sum(_sizes(case)), 0.80, case.get("gaussian", True)
    else:
        n, rho, steps = case["n"], case["density"], case.get("steps", 1)
        gaussian = case.get("gaussian", False)
    near = 4.0 / 3.0 * math.pi * RC ** 3 * rho
    per_step = 2 * 16 + 2 * (24 if gaussian else 16) + 2 * 16
    if kind == "energy":
        per_step = 32
    if kind == "relax":
        per_step = 48
    flops = (22 if kind != "energy" else 28) * near / 2
    return {"bytes": float(n) * (per_step * steps + 32), "flops": float(n) * flops * steps}


# ---- the same in 64 bits ----------------------------------------------------------


class _Exact:
    """One system in 64-bit torch: forces from a pair list with a skin, rebuilt
    when an atom has moved half of it."""

    SKIN = 0.5

    def __init__(self, s: W.LJSystem, capped: bool = False):
        d = "cuda" if torch.cuda.is_available() else "cpu"
        f32 = lambda a: torch.tensor(np.asarray(a, np.float32).astype(np.float64), device=d)  # noqa: E731
        self.n, self.capped = s.n, capped
        self.r = f32(s.r)
        self.v = torch.tensor(s.v, dtype=torch.float64, device=d)
        self.m = torch.tensor(s.mass, dtype=torch.float64, device=d)[:, None]
        box = np.asarray(s.box, np.float32).astype(np.float64)
        self.L = torch.tensor(box[1::2] - box[::2], device=d)
        self.lj = f32(s.lj)
        self.types = torch.tensor(s.types.astype(np.int64), device=d)
        self.rc = float(s.lj[..., 2].max())
        self.F = torch.zeros_like(self.r)
        self.xi = 0.0
        self.at = None

    def image(self, d):
        return d - self.L * torch.round(d / self.L)

    def pairs(self):
        rl = self.rc + self.SKIN
        nc = torch.clamp((self.L / rl).floor(), min=1).long()
        nx, ny, nz = (int(x) for x in nc)
        c = torch.minimum((self.r / self.L * nc).long().clamp(min=0), nc - 1)
        key = (c[:, 0] * ny + c[:, 1]) * nz + c[:, 2]
        order = torch.argsort(key)
        count = torch.bincount(key, minlength=nx * ny * nz)
        start = torch.cumsum(count, 0) - count
        slots = torch.arange(int(count.max()), device=self.r.device)
        found, tried = [], set()
        near = [sorted({x % m for x in (-1, 0, 1)}) for m in (nx, ny, nz)]
        part = max(1, 60_000_000 // max(1, len(slots)))
        for dx in near[0]:
            for dy in near[1]:
                for dz in near[2]:
                    if (dx, dy, dz) in tried:
                        continue
                    tried.add((dx, dy, dz))
                    other = (((c[:, 0] + dx) % nx * ny + (c[:, 1] + dy) % ny) * nz
                             + (c[:, 2] + dz) % nz)
                    for a in range(0, self.n, part):
                        o = other[a:a + part]
                        i = torch.arange(a, min(self.n, a + part), device=self.r.device)
                        ok = slots[None, :] < count[o][:, None]
                        j = order[torch.where(ok, start[o][:, None] + slots, 0)]
                        i, j = i[:, None].expand_as(j)[ok], j[ok]
                        keep = i < j
                        i, j = i[keep], j[keep]
                        keep = (self.image(self.r[i] - self.r[j]) ** 2).sum(1) < rl * rl
                        found.append(torch.stack([i[keep], j[keep]]))
        self.i, self.j = torch.cat(found, 1)
        self.at = self.r.clone()

    def forces(self, energy: bool = False):
        moved = None if self.at is None else self.image(self.r - self.at)
        if moved is None or 2.0 * float((moved ** 2).sum(1).max()) ** 0.5 > self.SKIN:
            self.pairs()
        d = self.image(self.r[self.i] - self.r[self.j])
        r2 = (d ** 2).sum(1)
        sig, eps, rc = self.lj[self.types[self.i], self.types[self.j]].unbind(1)
        inside = r2 < rc * rc
        if self.capped:
            r2 = torch.maximum(r2, 0.25 * sig * sig)
        s6 = (sig * sig / r2) ** 3
        f = torch.where(inside, 24.0 * eps * s6 * (2.0 * s6 - 1.0) / r2, 0.0)
        fd = f[:, None] * d
        F = torch.zeros_like(self.r)
        F.index_add_(0, self.i, fd)
        F.index_add_(0, self.j, -fd)
        if energy:
            return F, float(torch.where(inside, 4.0 * eps * s6 * (s6 - 1.0), 0.0).sum()), \
                float((f * r2).sum())
        return F

    def wrap(self):
        self.r = self.r - self.L * torch.floor(self.r / self.L)

    def step(self, gaussian: bool):
        dt = float(np.float32(DT))
        F = self.forces()
        a = self.v + (F + self.F) * (0.5 * dt / self.m)
        if gaussian:
            a = a - self.v * (0.5 * dt * self.xi)
            c = float((F * a).sum() / (self.m * a * a).sum())
            if self.xi == 0.0:  # the first step ends its solve with v = a
                self.v, self.xi = a, c
            else:
                self.xi = c / (1.0 - 0.5 * dt * c)
                self.v = a / (1.0 + 0.5 * dt * self.xi)
            self.r = (self.r + self.v * (dt - 0.5 * dt * dt * self.xi)
                      + F * (0.5 * dt * dt / self.m))
        else:
            self.v = a
            self.r = self.r + self.v * dt + F * (0.5 * dt * dt / self.m)
        self.F = F
        self.wrap()

    def descend(self):
        F = self.forces()
        size = (F ** 2).sum(1, keepdim=True).sqrt()
        self.r = self.r + F * torch.where(size * ALPHA > MAX_DISP, MAX_DISP / size, ALPHA)
        self.wrap()

    def temperature(self) -> float:
        return float((self.m * self.v * self.v).sum()) / (3 * self.n)


def _four(x: torch.Tensor) -> torch.Tensor:
    return torch.cat([x, torch.zeros_like(x[:, :1])], 1)


def _after(s: W.LJSystem, steps: int, gaussian: bool) -> _Exact:
    if not gaussian:
        s.v = s.v.astype(np.float32).astype(np.float64)
    x = _Exact(s)
    for _ in range(steps):
        x.step(gaussian)
    return x


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "gr":
        return None  # whole numbers
    if kind == "batch":
        systems = _replicas(case, seed)
        return [_four(_after(s, case["steps"], case["gaussian"]).r) for s in systems]
    if kind == "serve":
        out = []
        for s, steps in _jobs(case, seed):
            x = _after(s, steps, True)
            out += [_four(x.r), _four(x.F)]
        return out
    s = _system(case, seed)
    if kind == "energy":
        s.v = s.v.astype(np.float32).astype(np.float64)
        x = _Exact(s)
        F, pe, virial = x.forces(energy=True)
        return {"F": _four(F), "E": np.array([pe, virial, x.temperature() * 3 * x.n])}
    if kind == "relax":
        x = _Exact(s, capped=True)
        for _ in range(case["steps"]):
            x.descend()
        return {"r": _four(x.r)}
    if kind == "driver":
        if not case["gaussian"]:
            s.v = s.v.astype(np.float32).astype(np.float64)
        x, T = _Exact(s), []
        for _ in range(case["steps"]):
            T.append(x.temperature())
            x.step(case["gaussian"])
        return {"r": _four(x.r), "F": _four(x.F), "T": np.array(T)}
    x = _after(s, case["steps"], kind == "run" and case["gaussian"])
    if kind == "run" and case["gaussian"]:
        return {"r": _four(x.r), "F": _four(x.F)}
    return {"r": _four(x.r), "v": _four(x.v)}
