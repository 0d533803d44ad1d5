"""The work a user of dmd_b200 has it do, as cases that can be timed and compared.

Every case goes through the public entry points (``Engine``, ``Batch``): a
frame of a trajectory (``run_n`` and the positions, velocities and energy a
program stores with it), a single-point evaluation, a batch of replicas, a
served wave of jobs.  Systems are the shapes of this repository's workloads
(LJ argon, flexible and rigid 3-site water with SPME, united-atom n-decane),
generated from a seed alone.

Mixed precision computes forces in FP32, so a program keeps its frames in
FP32; frames of the all-FP64 path stay FP64.

``exact`` repeats a case in 64-bit torch: pair sums over a brute-force pair
list, autograd for the bonded terms, SPME as a plain 4x4x4 spread with torch's
FFT, velocity Verlet with the same thermostats.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from dmd_b200.batch import Batch
from dmd_b200.core import Engine, SimulationConfig

KB = 0.008314462618      # kJ mol^-1 K^-1
KE = 138.935456          # kJ mol^-1 nm e^-2
SKIN = 0.15              # nm, the list skin every case asks for

# n-decane: types 0 = CH2, 1 = CH3
DEC_SIG = (0.395, 0.375)
DEC_EPS = (0.382, 0.814)
DEC_DIH = ((1, 2.95, 0.0), (2, -0.567, math.pi), (3, 6.58, 0.0))


# ---------------------------------------------------------------------------
# Cases
# ---------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # a small LJ fluid sampled often: a step is a few short launches, so latency is all
        dict(name="lj-1k-nve", kind="lj", n=1000, rho=0.75, t_star=1.1, steps=100,
             profile="phys", precision="mixed"),
        # argon on an FCC lattice with the engine's default profile (the reference's formulas,
        # list rebuilt every tenth force call)
        dict(name="argon-4k-ref", kind="argon", cells=10, steps=100, profile="ref",
             precision="mixed"),
        # an ordinary LJ fluid of odd size, the largest replica of the batch workload
        dict(name="lj-20k-nvt", kind="lj", n=19997, rho=0.8, t_star=1.0, steps=50,
             thermostat="berendsen", profile="phys", precision="mixed"),
        # rigid water, SHAKE / RATTLE at 2 fs: the shape the reference's own timings are quoted on
        dict(name="water-1.5k-rigid", kind="water", n_mol=522, steps=50, rigid=True,
             thermostat="nose-hoover", profile="phys", precision="mixed"),
        # a solvent box of an everyday study, flexible water, SPME, odd size
        dict(name="water-9k-nvt", kind="water", n_mol=3001, steps=50, thermostat="nose-hoover",
             profile="phys", precision="mixed"),
        # the headline workload (64^3 mesh)
        dict(name="water-30k-nvt", kind="water", n_mol=10000, steps=50, thermostat="nose-hoover",
             profile="phys", precision="mixed"),
        # the same box on the all-FP64 path (a reference run to trust the mixed one by)
        dict(name="water-30k-fp64", kind="water", n_mol=10000, steps=20,
             thermostat="nose-hoover", profile="phys", precision="fp64"),
        # the large box, constant pressure (192^3 mesh)
        dict(name="water-750k-npt", kind="water", n_mol=250000, steps=30, thermostat="berendsen",
             barostat="berendsen", spacing=0.1019, profile="phys", precision="mixed"),
        # a molecular melt without charges: bonds, angles, dihedrals, exclusions
        dict(name="decane-4k-nvt", kind="decane", n_chains=400, steps=100,
             thermostat="berendsen", profile="phys", precision="mixed"),
        # one force evaluation at new positions, as a minimiser or an outer driver asks for it
        dict(name="water-30k-single", kind="water", n_mol=10000, single=True, profile="phys",
             precision="mixed"),
        # replicas of uneven sizes advanced in one launch (48 LJ fluids, 16 decane melts)
        dict(name="batch-64", kind="batch", n_lj=48, n_dec=16, n_lo=500, n_hi=20000, steps=20,
             profile="phys", precision="mixed"),
        # a served wave: jobs of mixed kinds and lengths arrive, run together, leave
        dict(name="serve-8", kind="serve", n_jobs=8, n_lo=1000, n_hi=30000, steps_lo=150,
             steps_hi=450, chunk=50, profile="phys", precision="mixed"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    """One more case of the same ranges."""
    kind = rng.choice(["lj", "lj", "lj", "argon", "water", "water", "water", "water", "fp64",
                       "rigid", "npt", "decane", "single", "single", "batch", "serve"])
    mixed = dict(profile="phys", precision="mixed")
    if kind == "lj":
        return dict(kind="lj", n=_log(rng, 500, 50000), rho=round(rng.uniform(0.6, 0.85), 3),
                    t_star=round(rng.uniform(0.8, 1.5), 3), steps=rng.randint(20, 100),
                    thermostat=rng.choice(["none", "none", "berendsen", "nose-hoover"]), **mixed)
    if kind == "argon":
        return dict(kind="argon", cells=rng.randint(6, 16), steps=rng.randint(20, 100),
                    profile="ref", precision=rng.choice(["mixed", "mixed", "fp64"]))
    if kind == "water":
        return dict(kind="water", n_mol=_log(rng, 600, 32000), steps=rng.randint(20, 50),
                    thermostat=rng.choice(["none", "berendsen", "nose-hoover"]), **mixed)
    if kind == "fp64":
        return dict(kind="water", n_mol=_log(rng, 600, 10000), steps=rng.randint(10, 20),
                    thermostat=rng.choice(["none", "nose-hoover"]), profile="phys",
                    precision="fp64")
    if kind == "rigid":
        return dict(kind="water", n_mol=_log(rng, 522, 4000), steps=rng.randint(20, 50),
                    rigid=True, thermostat=rng.choice(["none", "nose-hoover"]), **mixed)
    if kind == "npt":
        return dict(kind="water", n_mol=_log(rng, 1000, 60000), steps=rng.randint(20, 40),
                    thermostat="berendsen", barostat="berendsen", **mixed)
    if kind == "decane":
        return dict(kind="decane", n_chains=_log(rng, 100, 2000), steps=rng.randint(20, 100),
                    thermostat=rng.choice(["none", "berendsen"]), **mixed)
    if kind == "single":
        what = rng.choice(["lj", "water", "decane"])
        c = dict(kind=what, single=True, **mixed)
        if what == "lj":
            c.update(n=_log(rng, 500, 50000), rho=round(rng.uniform(0.6, 0.85), 3), t_star=1.0)
        elif what == "water":
            c.update(n_mol=_log(rng, 600, 32000))
        else:
            c.update(n_chains=_log(rng, 100, 2000))
        return c
    if kind == "batch":
        return dict(kind="batch", n_lj=rng.randint(6, 48), n_dec=rng.randint(2, 16), n_lo=500,
                    n_hi=_log(rng, 2000, 20000), steps=rng.randint(10, 20), **mixed)
    return dict(kind="serve", n_jobs=rng.randint(3, 8), n_lo=1000, n_hi=_log(rng, 5000, 30000),
                steps_lo=100, steps_hi=rng.randint(200, 400), chunk=rng.choice([25, 50, 100]),
                **mixed)


# ---------------------------------------------------------------------------
# Systems: plain dicts of arrays, made from a seed
# ---------------------------------------------------------------------------
def _maxwell(rng, mass, T):
    v = rng.normal(size=(len(mass), 3)) * np.sqrt(KB * T / mass)[:, None]
    return v - (mass[:, None] * v).sum(0) / mass.sum()


def _base(pos, box, mass, rc, dt, T, rng, **more):
    n = len(mass)
    s = dict(pos=pos, vel=_maxwell(rng, mass, T), box=box, mass=mass, charge=np.zeros(n),
             types=np.zeros(n, np.int32), rc=rc, dt=dt, T=T, sig=np.array([[0.3405]]),
             eps=np.array([[0.996]]), coulomb="cutoff", spacing=0.12, alpha=3.12,
             thermostat="none", barostat="none", tau=0.1)
    s.update(more)
    return s


def _lattice(n, box):
    ns = int(math.ceil(n ** (1.0 / 3.0) - 1e-9))
    g = np.arange(ns)
    sites = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[:n]
    return (sites + 0.5) * (box / ns), box / ns


def _lj(n, rho, t_star, seed):
    rng = np.random.default_rng(seed)
    box = (n * 0.3405 ** 3 / rho) ** (1.0 / 3.0)
    p, a = _lattice(n, box)
    p = p + rng.uniform(-0.05, 0.05, (n, 3)) * a
    return _base(p, box, np.full(n, 39.948), 2.5 * 0.3405, 0.002, t_star * 0.996 / KB, rng)


def _argon(cells, seed):
    rng = np.random.default_rng(seed)
    a = 0.575
    base = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    g = np.arange(cells)
    c = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    p = ((c[:, None, :] + base[None]) * a).reshape(-1, 3) + 0.01 * a * rng.uniform(-1, 1, (4 * cells ** 3, 3))
    return _base(p, cells * a, np.full(len(p), 39.948), 1.0, 0.002, 120.0, rng)


def _water(n_mol, seed, rigid=False, spacing=0.1045):
    rng = np.random.default_rng(seed)
    box = (n_mol / 33.4) ** (1.0 / 3.0)
    o, a = _lattice(n_mol, box)
    o = o + rng.uniform(-0.1, 0.1, (n_mol, 3)) * a
    th = math.radians(109.47)
    q = rng.normal(size=(n_mol, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    rot = np.stack([np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w)], -1),
                    np.stack([2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w)], -1),
                    np.stack([2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)], -1)], 1)
    ref = 0.1 * np.array([[1.0, 0.0, 0.0], [math.cos(th), math.sin(th), 0.0]])
    h = np.einsum("nij,kj->nki", rot, ref) + o[:, None, :]
    pos = np.concatenate([o[:, None, :], h], 1).reshape(-1, 3)
    m = np.arange(n_mol, dtype=np.int32) * 3
    oh = np.stack([np.stack([m, m + 1], 1), np.stack([m, m + 2], 1)], 1).reshape(-1, 2)
    hh = np.stack([np.stack([m, m + 1], 1), np.stack([m, m + 2], 1), np.stack([m + 1, m + 2], 1)], 1).reshape(-1, 2)
    s = _base(pos, box, np.tile([15.9994, 1.008, 1.008], n_mol), 1.0, 0.002 if rigid else 0.0005, 300.0,
              rng, charge=np.tile([-0.8476, 0.4238, 0.4238], n_mol), types=np.tile(np.array([1, 0, 0], np.int32), n_mol),
              sig=np.array([[1.0, 1.0], [1.0, 0.3166]]), eps=np.array([[0.0, 0.0], [0.0, 0.650]]),
              coulomb="pme", spacing=spacing,
              bonds=oh, bond_k=np.full(2 * n_mol, 345000.0), bond_r0=np.full(2 * n_mol, 0.1),
              angles=np.stack([m + 1, m, m + 2], 1), angle_k=np.full(n_mol, 383.0),
              angle_t0=np.full(n_mol, th), excl=hh)
    if rigid:
        s.update(cons=hh, cons_d=np.tile([0.1, 0.1, 0.2 * math.sin(th / 2)], n_mol))
    return s


def _decane(n_chains, seed):
    """All-trans chains on a lattice of parallel sites, slightly jittered."""
    rng = np.random.default_rng(seed)
    b, th, n = 0.154, math.radians(114.0), n_chains
    box = (n / 2.7) ** (1.0 / 3.0)
    fit = []
    for nx in range(1, 16):
        m = math.ceil(math.sqrt(n / nx) - 1e-9)
        fit.append((min((box / nx - 9 * b * math.sin(th / 2)) / 0.38, box / m / 0.44), nx, m))
    _, nx, m = max(fit)
    cell = np.stack(np.meshgrid(np.arange(nx), np.arange(m), np.arange(m), indexing="ij"), -1).reshape(-1, 3)
    cell = cell[np.sort(rng.permutation(len(cell))[:n])]
    k = np.arange(10)
    chain = np.stack([k * b * math.sin(th / 2), (k % 2) * b * math.cos(th / 2), 0 * k], 1)
    pos = (cell * np.array([box / nx, box / m, box / m]))[:, None, :] + chain[None]
    pos = pos + rng.uniform(-0.002, 0.002, pos.shape)
    off = (np.arange(n) * 10)[:, None, None]

    def terms(w):
        t = np.stack([np.arange(10 - w + 1) + i for i in range(w)], 1)
        return (off + t[None]).reshape(-1, w).astype(np.int32)

    quads = terms(4)
    end = np.stack([k[:7], k[:7] + 3], 1)
    pairs = np.concatenate([np.stack([k[:9], k[:9] + 1], 1), np.stack([k[:8], k[:8] + 2], 1), end])
    types = np.tile(np.array([1] + [0] * 8 + [1], np.int32), n)
    cs, ce = 0.5 * sum(DEC_SIG), math.sqrt(DEC_EPS[0] * DEC_EPS[1])
    return _base(pos.reshape(-1, 3), box, np.where(types == 1, 15.035, 14.027), 2.5 * 0.395, 0.002, 300.0,
                 rng, types=types, sig=np.array([[DEC_SIG[0], cs], [cs, DEC_SIG[1]]]),
                 eps=np.array([[DEC_EPS[0], ce], [ce, DEC_EPS[1]]]),
                 bonds=terms(2), bond_k=np.full(9 * n, 200000.0), bond_r0=np.full(9 * n, b),
                 angles=terms(3), angle_k=np.full(8 * n, 520.0), angle_t0=np.full(8 * n, th),
                 dihedrals=np.repeat(quads, 3, axis=0), dih_n=np.tile([d[0] for d in DEC_DIH], len(quads)),
                 dih_k=np.tile([d[1] for d in DEC_DIH], len(quads)),
                 dih_p=np.tile([d[2] for d in DEC_DIH], len(quads)),
                 excl=(off + pairs[None]).reshape(-1, 2).astype(np.int32))


def _system(case, seed):
    if case["kind"] == "lj":
        s = _lj(case["n"], case["rho"], case["t_star"], seed)
    elif case["kind"] == "argon":
        s = _argon(case["cells"], seed)
    elif case["kind"] == "water":
        s = _water(case["n_mol"], seed, bool(case.get("rigid")), case.get("spacing", 0.1045))
    else:
        s = _decane(case["n_chains"], seed)
    s["thermostat"] = case.get("thermostat", "none")
    s["barostat"] = case.get("barostat", "none")
    return s


def _replicas(case, seed):
    """The batch: LJ fluids of uneven sizes, densities and temperatures, and decane melts (the
    case gives the shapes, the seed the configurations)."""
    rng = np.random.default_rng(case["n_hi"])
    out = [_lj(int(rng.integers(case["n_lo"], case["n_hi"] + 1)), rng.uniform(0.6, 0.85), rng.uniform(0.8, 1.5),
               seed + 1 + k) for k in range(case["n_lj"])]
    return out + [_decane(int(rng.integers(100, max(101, case["n_hi"] // 50) + 1)), seed + 1001 + k)
                  for k in range(case["n_dec"])]


def _jobs(case, seed):
    """Served jobs: 70 % LJ, 30 % water, sizes log-uniform, lengths uniform (the case gives
    sizes and lengths, the seed the configurations)."""
    rng = np.random.default_rng(case["n_hi"] + case["steps_hi"])
    jobs = []
    for k in range(case["n_jobs"]):
        n = int(round(math.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))))
        steps = int(rng.integers(case["steps_lo"], case["steps_hi"] + 1))
        jobs.append((_water(max(600, n // 3), seed + 1 + k) if k % 10 in (1, 4, 7)
                     else _lj(n, rng.uniform(0.6, 0.85), rng.uniform(0.8, 1.5), seed + 1 + k), steps))
    return jobs


def _config(s) -> SimulationConfig:
    c = SimulationConfig()
    c.box_size, c.dt, c.init_temperature = s["box"], s["dt"], s["T"]
    c.pos_x, c.pos_y, c.pos_z = s["pos"].T
    c.vel_x, c.vel_y, c.vel_z = s["vel"].T
    c.mass, c.charges, c.atom_types = s["mass"], s["charge"], s["types"]
    c.use_lj, c.lj_sigma, c.lj_epsilon, c.lj_cutoff = True, s["sig"].ravel(), s["eps"].ravel(), s["rc"]
    c.coulomb_type, c.coulomb_cutoff = s["coulomb"], s["rc"]
    c.ewald_coeff, c.pme_grid_spacing = s["alpha"], s["spacing"]
    if "bonds" in s:
        c.bond_i, c.bond_j = s["bonds"].T
        c.bond_k, c.bond_r0 = s["bond_k"], s["bond_r0"]
        c.angle_i, c.angle_j, c.angle_k = s["angles"].T
        c.angle_k_theta, c.angle_theta0 = s["angle_k"], s["angle_t0"]
        c.excl_i, c.excl_j = s["excl"].T
    if "dihedrals" in s:
        c.dihedral_i, c.dihedral_j, c.dihedral_k, c.dihedral_l = s["dihedrals"].T
        c.dihedral_k_phi, c.dihedral_periodicity, c.dihedral_phi0 = s["dih_k"], s["dih_n"], s["dih_p"]
    if "cons" in s:
        c.constraint_type, c.constraint_tolerance = "shake", 1e-8
        c.constraint_i, c.constraint_j = s["cons"].T
        c.constraint_dist = s["cons_d"]
    c.thermostat.type, c.thermostat.temperature, c.thermostat.tau = s["thermostat"], s["T"], s["tau"]
    c.barostat.type = s["barostat"]
    c.checkpoint_interval, c.checkpoint_path = 0, ""
    return c


# ---------------------------------------------------------------------------
# Preparation and one pass
# ---------------------------------------------------------------------------
def prepare(case, seed):
    opt = dict(precision=case["precision"], profile=case["profile"], skin=SKIN)
    keep = np.float32 if case["precision"] == "mixed" else np.float64
    state = dict(case=case, keep=keep)
    if case["kind"] == "batch":
        b = Batch(**opt)
        state["batch"] = b
        state["slots"] = [b.admit(_config(s), 1 << 40) for s in _replicas(case, seed)]
    elif case["kind"] == "serve":
        state["batch"] = Batch(**opt)
        state["jobs"] = [(_config(s), steps) for s, steps in _jobs(case, seed)]
    else:
        s = _system(case, seed)
        state["engine"] = Engine(_config(s), **opt)
        if case.get("single"):
            state["pos"] = s["pos"]
    return state


def run(state):
    case, keep = state["case"], state["keep"]
    if case["kind"] == "batch":
        b = state["batch"]
        b.step(case["steps"])
        return dict(positions=np.concatenate([b.positions(k) for k in state["slots"]]).astype(keep),
                    velocities=np.concatenate([b.velocities(k) for k in state["slots"]]).astype(keep),
                    kinetic=np.array([b.scalars(k).kinetic_energy for k in state["slots"]], keep))
    if case["kind"] == "serve":
        return _serve_wave(state["batch"], state["jobs"], case["chunk"], keep)
    e = state["engine"]
    if case.get("single"):
        e.set_positions(state["pos"])
        f, terms = e.compute_forces()
        return dict(forces=f.astype(keep), terms=np.array(list(terms.values()), keep))
    e.run_n(case["steps"])
    s = e.scalars()
    return dict(positions=e.positions.astype(keep), velocities=e.velocities.astype(keep),
                energy=np.array([s.potential_energy, s.kinetic_energy], keep), box=keep(s.box), step=int(s.step))


def _serve_wave(b, jobs, chunk, keep):
    """Half of the jobs are there at the start, the others arrive one per device call."""
    waiting = list(range(len(jobs)))
    running, out = {}, [None] * len(jobs)
    first = True
    while waiting or running:
        for _ in range(min(len(waiting), (len(jobs) + 1) // 2 if first else 1)):
            j = waiting.pop(0)
            running[b.admit(*jobs[j])] = j
        first = False
        b.step(chunk)
        for slot in b.poll():
            out[running.pop(slot)] = np.concatenate([b.positions(slot), b.velocities(slot)]).astype(keep)
            b.release(slot)
    return np.concatenate(out)


# ---------------------------------------------------------------------------
# Work a pass cannot do without
# ---------------------------------------------------------------------------
def _step_work(s_or_n, rho=None, charged=False, rc=1.0, terms=0.0, mesh=0):
    """Per step: the pairs inside the cutoff once (about 30 flops for an LJ pair, 45 with the
    real-space Ewald term), bonded terms (about 60), mesh points (spread and gather of 64
    points per charge, two real FFTs); the state (positions, velocities, masses, forces) read
    and written once."""
    n = s_or_n
    pairs = 0.5 * n * rho * 4.18879 * rc ** 3
    flops = pairs * (45 if charged else 30) + 60 * terms + 30 * n
    if mesh:
        flops += n * 64 * 20 + 2 * 2.5 * mesh ** 3 * math.log2(mesh ** 3)
    return dict(bytes=144.0 * n + (16.0 * mesh ** 3 if mesh else 0) + 40 * terms, flops=flops)


def _kind_work(kind, n, rho, spacing=0.1045):
    if kind == "water":
        mesh = max(8, int((n / 3 / 33.4) ** (1 / 3) / spacing + 0.5))
        return _step_work(n, 100.2, True, 1.0, 2.0 * n, mesh)
    if kind == "decane":
        return _step_work(n, 27.0, False, 0.9875, 6.2 * n)
    if kind == "argon":
        return _step_work(n, 21.04, False, 1.0)
    return _step_work(n, rho / 0.3405 ** 3, False, 2.5 * 0.3405)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        a = _kind_work("lj", 0.5 * (case["n_lo"] + case["n_hi"]), 0.725)
        d = _kind_work("decane", 10 * 0.5 * (100 + max(101, case["n_hi"] // 50)), 0)
        return {k: case["steps"] * (case["n_lj"] * a[k] + case["n_dec"] * d[k]) for k in a}
    if kind == "serve":
        mean = (case["n_hi"] - case["n_lo"]) / math.log(case["n_hi"] / case["n_lo"])
        a, w = _kind_work("lj", mean, 0.725), _kind_work("water", 3 * int(mean / 3), 0)
        steps = 0.5 * (case["steps_lo"] + case["steps_hi"])
        return {k: case["n_jobs"] * steps * (0.7 * a[k] + 0.3 * w[k]) for k in a}
    n = {"lj": case.get("n"), "argon": 4 * case.get("cells", 0) ** 3, "water": 3 * case.get("n_mol", 0),
         "decane": 10 * case.get("n_chains", 0)}[kind]
    w = _kind_work(kind, n, case.get("rho"), case.get("spacing", 0.1045))
    return {k: v * (1 if case.get("single") else case["steps"]) for k, v in w.items()}


# ---------------------------------------------------------------------------
# The same in 64-bit torch
# ---------------------------------------------------------------------------
class _Exact:
    """Forces and energy terms of one system, and its velocity Verlet steps."""

    def __init__(self, s, phys):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.s, self.phys, self.L = s, phys, s["box"]
        t = lambda a, d=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=d, device=self.dev)  # noqa: E731
        self.x, self.v, self.m, self.q = t(s["pos"]), t(s["vel"]), t(s["mass"]), t(s["charge"])
        self.ty = t(s["types"], torch.int64)
        self.sig, self.eps = t(s["sig"]), t(s["eps"])
        self.charged = phys and bool(np.any(s["charge"]))
        for k in ("bonds", "angles", "dihedrals", "excl"):
            if k in s:
                setattr(self, k, t(s[k], torch.int64))
        for k in ("bond_k", "bond_r0", "angle_k", "angle_t0", "dih_n", "dih_k", "dih_p"):
            if k in s:
                setattr(self, k, t(s[k]))
        self.pairs, self.made_at, self.calls, self.zeta = None, None, 10, 0.0
        self.K = max(8, int(self.L / s["spacing"] + 0.5))

    def wrap(self, d):
        return d - torch.round(d / self.L) * self.L

    def build(self, reach):
        n, out = len(self.x), []
        step = max(1, 40_000_000 // n)
        for i in range(0, n, step):
            d2 = sum(self.wrap(self.x[None, i:, k] - self.x[i:i + step, k, None]) ** 2 for k in range(3))
            a, b = torch.nonzero(torch.triu(d2 < reach * reach, 1), as_tuple=True)
            out.append(torch.stack([a + i, b + i]))
        p = torch.cat(out, 1)
        if self.phys and hasattr(self, "excl"):
            key = lambda u: torch.minimum(u[0], u[1]) * n + torch.maximum(u[0], u[1])  # noqa: E731
            p = p[:, ~torch.isin(key(p), key(self.excl.T))]
        self.pairs, self.made_at = p, self.x.clone()

    def listed_pairs(self):
        if self.phys:
            if self.pairs is None or float(((self.x - self.made_at) ** 2).sum(1).max()) > 0.0099:
                self.build(self.s["rc"] + 0.2)
            return
        if self.calls >= 10:  # the reference's cadence: no skin, every tenth call
            self.build(self.s["rc"])
            self.calls = 0
        self.calls += 1

    def evaluate(self):
        rc2 = self.s["rc"] ** 2
        self.listed_pairs()
        i, j = self.pairs
        d = self.wrap(self.x[j] - self.x[i])
        r2 = (d * d).sum(1)
        keep = r2 < rc2
        i, j, d, r2 = i[keep], j[keep], d[keep], r2[keep]
        sr6 = (self.sig[self.ty[i], self.ty[j]] ** 2 / r2) ** 3
        e4 = 4 * self.eps[self.ty[i], self.ty[j]]
        f = 6 * e4 * (2 * sr6 * sr6 - sr6) / r2
        E = dict(lj=float((e4 * (sr6 * sr6 - sr6)).sum()))
        F = torch.zeros_like(self.x)
        if self.charged:
            a, r = self.s["alpha"], torch.sqrt(r2)
            qq, ec = KE * self.q[i] * self.q[j], torch.erfc(a * r)
            f = f + qq * (ec / (r2 * r) + 2 * a / math.sqrt(math.pi) * torch.exp(-a * a * r2) / r2)
            E["coul_real"] = float((qq * ec / r).sum())
        g = f[:, None] * d
        F.index_add_(0, j, g)
        F.index_add_(0, i, -g)
        if self.charged and self.s["coulomb"] == "pme":
            E["coul_recip"] = self.spme(F)
            E["coul_self"] = -KE * self.s["alpha"] / math.sqrt(math.pi) * float((self.q ** 2).sum())
        if hasattr(self, "excl") and self.charged:
            i, j = self.excl.T
            a, d = self.s["alpha"], self.wrap(self.x[j] - self.x[i])
            r2 = (d * d).sum(1)
            r, qq = torch.sqrt(r2), KE * self.q[i] * self.q[j]
            ef = torch.erf(a * r)
            g = (qq * (2 * a / math.sqrt(math.pi) * torch.exp(-a * a * r2) / r2 - ef / (r2 * r)))[:, None] * d
            F.index_add_(0, j, g)
            F.index_add_(0, i, -g)
            E["coul_excl"] = -float((qq * ef / r).sum())
        if hasattr(self, "bonds"):
            x = self.x.clone().requires_grad_(True)
            E.update(self.bonded(x))
            total = sum(E[k] for k in ("bond", "angle", "dihedral") if k in E)
            F -= torch.autograd.grad(total, x)[0]
            E = {k: float(v) for k, v in E.items()}
        self.F, self.E = F, E
        return F

    def bonded(self, x):
        i, j = self.bonds.T
        r = torch.linalg.norm(self.wrap(x[j] - x[i]), dim=1)
        E = dict(bond=(0.5 * self.bond_k * (r - self.bond_r0) ** 2).sum())
        i, j, k = self.angles.T
        a, b = self.wrap(x[i] - x[j]), self.wrap(x[k] - x[j])
        th = torch.atan2(torch.linalg.norm(torch.linalg.cross(a, b), dim=1), (a * b).sum(1))
        E["angle"] = (0.5 * self.angle_k * (th - self.angle_t0) ** 2).sum()
        if hasattr(self, "dihedrals"):
            i, j, k, l = self.dihedrals.T
            b1, b2, b3 = self.wrap(x[j] - x[i]), self.wrap(x[k] - x[j]), self.wrap(x[l] - x[k])
            n1, n2 = torch.linalg.cross(b1, b2), torch.linalg.cross(b2, b3)
            phi = torch.atan2((torch.linalg.norm(b2, dim=1)) * (b1 * n2).sum(1), (n1 * n2).sum(1))
            E["dihedral"] = (self.dih_k * (1 + torch.cos(self.dih_n * phi - self.dih_p))).sum()
        return E

    def spme(self, F):
        K, L, a = self.K, self.L, self.s["alpha"]
        u = self.x / L
        u = (u - torch.floor(u)) * K
        m0 = torch.floor(u)
        o = torch.arange(-1, 3, device=self.dev, dtype=torch.float64)
        t = u[:, :, None] - (m0[:, :, None] + o)          # n, 3, 4
        b = t.abs()
        w = torch.where(b >= 2, 0 * b, torch.where(b >= 1, (2 - b) ** 3 / 6, (4 - 6 * b * b + 3 * b ** 3) / 6))
        dw = torch.sign(t) * torch.where(b >= 2, 0 * b, torch.where(b >= 1, -(2 - b) ** 2 / 2, (9 * b * b - 12 * b) / 6))
        g = torch.remainder(m0[:, :, None].long() + o.long(), K)
        idx = ((g[:, 2, :, None, None] * K + g[:, 1, None, :, None]) * K + g[:, 0, None, None, :]).reshape(len(u), -1)
        prod = lambda x, y, z: (z[:, :, None, None] * y[:, None, :, None] * x[:, None, None, :]).reshape(len(u), -1)  # noqa: E731
        mesh = torch.zeros(K ** 3, dtype=torch.float64, device=self.dev)
        mesh.index_add_(0, idx.reshape(-1), (self.q[:, None] * prod(w[:, 0], w[:, 1], w[:, 2])).reshape(-1))
        S = torch.fft.rfftn(mesh.reshape(K, K, K))
        m = torch.fft.fftfreq(K, 1.0 / K, device=self.dev, dtype=torch.float64)
        bs = 1 / (2 / 3 + torch.cos(2 * math.pi * m / K) / 3) ** 2
        h = K // 2 + 1
        k2 = 4 * math.pi ** 2 / L ** 2 * (m[:, None, None] ** 2 + m[None, :, None] ** 2 + m[None, None, :h].abs() ** 2)
        G = 4 * math.pi * KE / L ** 3 * torch.exp(-k2 / (4 * a * a)) / k2 * bs[:, None, None] * bs[None, :, None] * bs[None, None, :h]
        G[0, 0, 0] = 0.0
        wt = torch.full((h,), 2.0, dtype=torch.float64, device=self.dev)
        wt[0] = 1.0
        if K % 2 == 0:
            wt[K // 2] = 1.0
        e = 0.5 * float((wt * G * (S.real ** 2 + S.imag ** 2)).sum())
        phi = torch.fft.irfftn(S * G, s=(K, K, K), norm="forward").reshape(-1)[idx]
        f = [(phi * prod(*(dw[:, k] if k == c else w[:, k] for k in range(3)))).sum(1) for c in range(3)]
        F -= (self.q * K / L)[:, None] * torch.stack(f, 1)
        return e

    def steps(self, n):
        s, dt = self.s, self.s["dt"]
        dof = 3 * len(self.m) - 3
        self.evaluate()
        for k in range(n):
            if not self.phys and k:
                self.evaluate()  # the reference evaluates twice per step (its list counts calls)
            self.v = self.v + self.F / self.m[:, None] * (0.5 * dt)
            self.x = self.x + self.v * dt
            self.evaluate()
            self.v = self.v + self.F / self.m[:, None] * (0.5 * dt)
            ke = float((0.5 * self.m * (self.v ** 2).sum(1)).sum())
            T, lam = 2 * ke / (dof * KB), 1.0
            if s["thermostat"] == "berendsen":
                lam = math.sqrt(1 + dt / s["tau"] * (s["T"] / T - 1))
            elif s["thermostat"] == "nose-hoover":
                self.zeta += 0.5 * dt * KB * (T - s["T"]) / (dof * KB * s["T"] * s["tau"] ** 2)
                lam = math.exp(-self.zeta * 0.5 * dt)
            self.v = self.v * lam
            self.ke = ke * lam * lam


_TERMS = ("lj", "coul_real", "coul_recip", "coul_self", "coul_excl", "bond", "angle", "dihedral", "improper")


def exact(case, seed):
    if case["kind"] == "serve" or case.get("rigid") or case.get("barostat", "none") != "none":
        return None
    phys = case["profile"] == "phys"
    if case["kind"] == "batch":
        reps = _replicas(case, seed)
        if sum(len(s["mass"]) for s in reps) > 700_000:
            return None
        sims = []
        for s in reps:
            e = _Exact(s, phys)
            e.steps(case["steps"])
            e.pairs = None
            sims.append(e)
        return dict(positions=torch.cat([e.x for e in sims]), velocities=torch.cat([e.v for e in sims]),
                    kinetic=np.array([e.ke for e in sims]))
    s = _system(case, seed)
    if len(s["mass"]) > 100_000:
        return None
    e = _Exact(s, phys)
    if case.get("single"):
        return dict(forces=e.evaluate(), terms=np.array([e.E.get(k, 0.0) for k in _TERMS]))
    e.steps(case["steps"])
    return dict(positions=e.x, velocities=e.v, energy=np.array([sum(e.E.values()), e.ke]), box=None, step=None)
