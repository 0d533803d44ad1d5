"""Kernel paths that a rule on sizes or shapes selects, each at the sizes where
it can go wrong, against the CPU oracle or the path it replaces."""
import math

import numpy as np
import pytest

from dmd_b200 import workloads as W

pytestmark = pytest.mark.gpu


def rel_rms(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def _engine(cfg, precision, profile, **kw):
    from dmd_b200.core import Engine
    return Engine(cfg, precision=precision, profile=profile, **kw)


def _rigid_water(n_mol, order):
    """Rigid water whose molecules list their constraints in `order` ("tri": the
    register path's (p,q), (p,r), (q,r); "perm": the same three in another order;
    "oh": the two O-H bonds only), or cycle through all three ("mixed")."""
    c = W.water_box(n_mol=n_mol, box=(n_mol / 33.4) ** (1 / 3), seed=11, spacing=0.1).config()
    r0, th = 0.09572, math.radians(104.52)
    ci, cj, cd = [], [], []
    for m in range(n_mol):
        kind = ("tri", "perm", "oh")[m % 3] if order == "mixed" else order
        o, a, b = 3 * m, 3 * m + 1, 3 * m + 2
        hh = 2 * r0 * math.sin(th / 2)
        rows = {"tri": [(o, a, r0), (o, b, r0), (a, b, hh)], "perm": [(a, b, hh), (o, a, r0), (o, b, r0)],
                "oh": [(o, a, r0), (o, b, r0)]}[kind]
        for i, j, d in rows:
            ci.append(i), cj.append(j), cd.append(d)
    c.constraint_type, c.constraint_tolerance, c.dt = "shake", 1e-9, 0.001
    c.constraint_i, c.constraint_j = np.array(ci, np.int32), np.array(cj, np.int32)
    c.constraint_dist = np.array(cd)
    c.thermostat.type = "berendsen"
    return c


@pytest.mark.parametrize("order", ["tri", "perm", "oh", "mixed"])
@pytest.mark.parametrize("n_mol", [64, 65, 130])
def test_constraint_paths(oracle, n_mol, order):
    """Triangles (registers) and other groups (general sweeps) in one launch, at
    block edges, FP64: the oracle sweeps all constraints in the given order.
    Tolerance: that of the constrained FP64 trajectories, 1e-8."""
    c = _rigid_water(n_mol, order)
    oe, eng = oracle.engine(c, "phys"), _engine(c, "fp64", "phys")
    oe.step(6)
    eng.run_n(6)
    assert np.abs(eng.positions - oe.get(0)).max() / c.box_size < 1e-8
    assert rel_rms(eng.velocities, oe.get(1)) < 1e-8


def _lists(cfg, oracle, profile):
    eng = _engine(cfg, "mixed", profile)
    eng.compute_forces()
    got = eng.pair_list()
    return set(zip(*[a.tolist() for a in got])), eng


@pytest.mark.parametrize("profile", ["ref", "phys"])
@pytest.mark.parametrize("n_chains", [9, 26, 40, 130])
def test_pair_set_several_images_and_exclusions(oracle, n_chains, profile):
    """List build in boxes of one to three cutoffs (tile pairs that need several
    periodic images, along one, two or three axes) with chain exclusions that
    reach into neighbouring tiles: the pair set equals a brute-force FP64 one."""
    cfg = W.decane_melt(n_chains, 3).config()
    got, eng = _lists(cfg, oracle, profile)
    x = np.stack([cfg.pos_x, cfg.pos_y, cfg.pos_z], 1)
    L = cfg.box_size
    rc = cfg.lj_cutoff + (0.15 if profile == "phys" else 0.0)
    ex = {(min(i, j), max(i, j)) for i, j in zip(cfg.excl_i, cfg.excl_j)} if profile == "phys" else set()
    want = set()
    for i in range(len(x) - 1):
        dd = x[i + 1:] - x[i]
        q = dd * (1.0 / L)
        dd = dd - np.copysign(np.floor(np.abs(q) + 0.5), q) * L
        r2 = dd[:, 0] * dd[:, 0] + dd[:, 1] * dd[:, 1] + dd[:, 2] * dd[:, 2]
        want.update((i, int(j)) for j in np.nonzero(r2 < rc * rc)[0] + i + 1)
    assert got == want - ex


@pytest.mark.parametrize("alpha", [3.12, 4.2])
@pytest.mark.parametrize("rc_lj", [1.0, 0.85])
@pytest.mark.parametrize("n_mol", [110, 429])
def test_fp64_pair_forms(oracle, n_mol, rc_lj, alpha):
    """FP64 pair forces: Ewald polynomial (alpha rc 3.12) and erfc() (4.2), equal
    and different cutoffs, boxes narrower (1.49 nm) and wider (2.34 nm) than
    twice the list cutoff, with and without energies.  Tolerances: 1e-9 for
    forces (fixed-point step), 1e-8 for a short trajectory."""
    box = (n_mol / 33.43) ** (1 / 3)
    c = W.water_box(n_mol=n_mol, box=box, seed=5, spacing=box / round(box / 0.1)).config()
    c.lj_cutoff, c.ewald_coeff = rc_lj, alpha
    eng = _engine(c, "fp64", "phys")
    f, e = eng.compute_forces()
    f_o, e_o = oracle.forces(c, "phys")
    assert rel_rms(f, f_o) < 1e-9
    oe = oracle.engine(c, "phys")
    oe.step(5)
    run = _engine(c, "fp64", "phys")
    run.run_n(5)
    assert np.abs(run.positions - oe.get(0)).max() < 1e-8
    assert rel_rms(run.velocities, oe.get(1)) < 1e-8
    # energies of the evaluation that ends a call do not change its forces
    one = _engine(c, "fp64", "phys")
    for _ in range(5):
        one.run_n(1)
    assert np.array_equal(one.positions, run.positions)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_mol,spacing", [(130, 0.2), (400, 0.105), (400, 0.022)])
def test_pme_mesh_sizes(oracle, n_mol, spacing, precision):
    """SPME on meshes of 8^3 (one block), 22^3 (a ragged last block) and 104^3 (the
    four-groups-per-thread conversion, above 2^20 points): forces and the
    reciprocal energy against the oracle.  Tolerances: the single-point ones."""
    box = (n_mol / 33.43) ** (1 / 3)
    c = W.water_box(n_mol=n_mol, box=box, seed=9, spacing=spacing).config()
    f, e = _engine(c, precision, "phys").compute_forces()
    f_o, e_o = oracle.forces(c, "phys")
    assert rel_rms(f, f_o) < {"fp64": 1e-9, "mixed": 1e-5}[precision]


def test_energies_of_mixed_blocks(oracle):
    """Bonded energies where a block's terms belong to several replicas: a batch
    of small decane melts gives each the energies it has alone, bit for bit."""
    from dmd_b200.batch import Batch
    cfgs = [W.decane_melt(n, 20 + n).config() for n in (9, 12, 10, 17, 9)]
    b = Batch(precision="mixed", profile="phys")
    slots = [b.admit(c, 3) for c in cfgs]
    b.step(3)
    for c, k in zip(cfgs, slots):
        eng = _engine(c, "mixed", "phys")
        eng.run_n(3)
        assert list(b.scalars(k).e_terms) == list(eng.scalars().e_terms)
        assert np.array_equal(b.positions(k), eng.positions)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [64, 65536, 65537, 140001])
def test_state_rows_and_arrays(n, precision):
    """State copies of one piece, exactly one, just above and several: rows,
    separate arrays and what was set agree bit for bit, and reading velocities
    leaves a pending thermostat scale as it is."""
    import ctypes
    from dmd_b200 import _capi
    c = W.lj_fluid(n, 0.7, 1.0, 3).config()
    c.thermostat.type, c.thermostat.temperature = "berendsen", 90.0
    eng = _engine(c, precision, "phys")
    rng = np.random.default_rng(1)
    x = np.stack([c.pos_x, c.pos_y, c.pos_z], 1)
    v = rng.normal(size=(n, 3))
    eng.set_positions(x)
    eng.set_velocities(v)
    assert np.array_equal(eng.positions, x) and np.array_equal(eng.velocities, v)
    eng.run_n(2)
    for which, rows in ((0, eng.positions), (1, eng.velocities), (2, eng.forces)):
        a = [np.empty(n) for _ in range(3)]
        assert eng._lib.dmdgpu_get_state(eng._h, which, *(_capi.dptr(k) for k in a)) == 0
        assert np.array_equal(np.stack(a, 1), rows)
    other = _engine(c, precision, "phys")
    other.set_positions(x)
    other.set_velocities(np.hstack([v, v])[:, :4])  # more columns: the first three count
    other.run_n(1)
    other.velocities
    other.run_n(1)
    assert np.array_equal(other.velocities, eng.velocities)
    assert eng._lib.dmdgpu_get_state_rows(eng._h, 3, _capi.dptr(np.empty((n, 3)))) == 4  # DMDGPU_ERR_PARM


def _argon(nc, seed=0):
    c = W.argon_fcc(n_cells=nc, a=0.575).config()
    rng = np.random.default_rng(seed)
    n = len(c.masses)
    c.pos_x, c.pos_y, c.pos_z = (p + rng.normal(0, 0.01, n) for p in (c.pos_x, c.pos_y, c.pos_z))
    return c


@pytest.mark.parametrize("calls", [(30,), (1,) * 12, (3, 1, 7, 2, 11), (5, 5, 5), (4, 9)])
def test_ref_cadence_across_calls(oracle, calls):
    """REF: the first evaluation is issued only in the steps whose list cadence
    needs it; calls that end anywhere in the cadence follow the oracle, which
    evaluates twice in every step (FP64, 1e-9), and new positions restart it."""
    c = _argon(4)
    oe, eng = oracle.engine(c, "ref"), _engine(c, "fp64", "ref")
    for n in calls:
        oe.step(n)
        eng.run_n(n)
        assert np.abs(eng.positions - oe.get(0)).max() < 1e-9
        assert rel_rms(eng.velocities, oe.get(1)) < 1e-9


def test_ref_cadence_in_batch(oracle):
    """REF replicas at different points of their cadence in one table (admitted at
    different times, with different targets) follow the oracle (FP64, 1e-9)."""
    from dmd_b200.batch import Batch
    cfgs = [_argon(4, 1), _argon(3, 2), _argon(4, 3)]
    targets = [17, 9, 12]
    b = Batch(precision="fp64", profile="ref")
    slots = [b.admit(cfgs[0], targets[0])]
    b.step(3)
    slots.append(b.admit(cfgs[1], targets[1]))
    b.step(4)
    slots.append(b.admit(cfgs[2], targets[2]))
    for n in (1, 6, 20):
        b.step(n)
    for c, n, k in zip(cfgs, targets, slots):
        oe = oracle.engine(c, "ref")
        oe.step(n)
        assert b.scalars(k).step == n
        assert np.abs(b.positions(k) - oe.get(0)).max() < 1e-9
        assert rel_rms(b.velocities(k), oe.get(1)) < 1e-9


@pytest.mark.parametrize("far", [0, 1000])
@pytest.mark.parametrize("n,d", [(33, 0.34), (64, 0.34), (64, 0.2), (700, 0.3)])
def test_fp64_dense_chunks(oracle, n, d, far):
    """FP64 pair kernel on dense clusters (64 atoms 0.2 nm apart: every pair of a
    chunk within the cutoff, its list full) and with atoms many boxes from the
    origin, where the single-precision distance test must not drop a pair.
    Tolerance: 1e-9 (the fixed-point step); 1,000 boxes out the coordinates hold
    1e-12 nm, on forces that change 14-fold per distance: 1e-9 still."""
    rng = np.random.default_rng(n)
    m = math.ceil(n ** (1 / 3) - 1e-9)
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    w = W.lj_fluid(n, 0.1, 1.0, seed=3)
    w.pos = (g + 0.02 * rng.random((n, 3))) * d + 0.1 + far * w.box * rng.integers(-1, 2, (n, 3))
    c = w.config()
    f, _ = _engine(c, "fp64", "phys").compute_forces()
    f_o, _ = oracle.forces(c, "phys")
    assert rel_rms(f, f_o) < 1e-9


@pytest.mark.parametrize("half", [0.5, 0.4995])
def test_fp64_ref_box_of_two_cutoffs(oracle, half):
    """REF keeps a list without a skin for five steps.  In a box of two cutoffs (or
    just above) the nearest image of a listed pair changes in between (up to 17
    pairs at a time here), and FP64 forces follow it as the oracle's do, over four
    cadences.  Tolerances: 1e-8 for a force component (at most 64 contributions
    to an atom of 8 tiles, each rounded to 2^-32; a pair lost at the cutoff is
    worth 1e-2) and 1e-9 nm."""
    c = _argon(4, 1)
    c.lj_cutoff = half * c.box_size
    oe, eng = oracle.engine(c, "ref"), _engine(c, "fp64", "ref")
    for _ in range(21):
        oe.step(1)
        eng.run_n(1)
        assert np.abs(eng.forces - oe.get(2)).max() < 1e-8
        assert np.abs(eng.positions - oe.get(0)).max() < 1e-9


@pytest.mark.parametrize("profile", ["ref", "phys"])
def test_fp64_pairs_half_a_box_apart(oracle, profile):
    """Lattice sites exactly half a box apart in a box narrower than twice the
    cutoff: the reference rounds the image halfway from zero, and so does the
    FP64 path (the other image would turn the force round).  Every second site is
    displaced, so that the forces do not cancel.  Tolerance: 1e-9."""
    g = np.stack(np.meshgrid(*[np.arange(4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    w = W.lj_fluid(64, 0.7, 1.0, 3)
    w.box, w.lj_cutoff = 2.0, 1.05
    w.pos = 0.5 * g + 0.02 * np.random.default_rng(2).random((64, 3)) * (g.sum(1) % 2)[:, None]
    c = w.config()
    f, _ = _engine(c, "fp64", profile).compute_forces()
    f_o, _ = oracle.forces(c, profile)
    assert rel_rms(f, f_o) < 1e-9


def test_fp64_tables_change_without_refitting():
    """Admitting and releasing one FP64 replica beside 48 charged ones fits no Ewald
    polynomial again: it takes about as long as with an alpha beyond the
    polynomial's reach, which is refused at once (48 fits, twice, are 24 ms or
    more; measured in turn, best of twelve each, 8 ms apart at most)."""
    import time
    from dmd_b200.batch import Batch

    def table(alpha):
        cfgs = [W.water_box(n_mol=60 + k, box=((60 + k) / 33.43) ** (1 / 3) + 1.2, seed=k, spacing=0.3).config()
                for k in range(48)]
        for c in cfgs:
            c.ewald_coeff = alpha
        b = Batch(precision="fp64", profile="phys")
        for c in cfgs:
            b.admit(c, 1 << 40)
        b.step(1)
        return b, cfgs[0]

    def change(b, c):
        t = time.perf_counter()
        k = b.admit(c, 1 << 40)
        b.step(1)
        b.release(k)
        b.step(1)
        return time.perf_counter() - t

    fitted, refused = table(3.12), table(9.0)
    times = [(change(*fitted), change(*refused)) for _ in range(12)]
    assert min(t[0] for t in times) < min(t[1] for t in times) + 0.008


def test_fp64_ewald_polynomials_of_one_table(oracle):
    """Replicas of one FP64 table that share a polynomial, have one of their own (alpha
    or cutoff) or none (alpha rc 4.2), admitted at different times and into a
    released slot: each has the forces it has alone, bit for bit, and the oracle's
    (1e-9)."""
    from dmd_b200.batch import Batch

    def make(k, alpha, rc):
        c = W.water_box(n_mol=429, box=2.34, seed=k, spacing=0.117).config()
        c.ewald_coeff, c.lj_cutoff, c.coulomb_cutoff = alpha, rc, rc
        return c

    kinds = [(3.12, 1.0), (3.12, 1.0), (2.9, 1.0), (3.12, 0.9), (4.2, 1.0), (3.12, 1.0)]
    cfgs = [make(k, a, rc) for k, (a, rc) in enumerate(kinds)]
    b = Batch(precision="fp64", profile="phys")
    first = b.admit(make(9, 3.0, 1.0), 1 << 40)
    slots = [b.admit(c, 1 << 40) for c in cfgs[:3]]
    b.step(1)
    b.release(first)
    slots += [b.admit(c, 1 << 40) for c in cfgs[3:]]
    b.step(1)
    for k, (c, slot) in enumerate(zip(cfgs, slots)):
        eng = _engine(c, "fp64", "phys")
        eng.run_n(1)
        if k < 3:  # in the table when the others came
            eng.repack()
            eng.run_n(1)
        assert np.array_equal(b.forces(slot), eng.forces) and np.array_equal(b.positions(slot), eng.positions)
        assert rel_rms(eng.forces, oracle.forces(c, "phys", pos=eng.positions)[0]) < 1e-9


def test_launch_info_of_the_fp64_path():
    """FP64 tables report the two blocks per SM that their pair kernel is launched
    with, whatever the list's size."""
    for n in (500, 20000):
        eng = _engine(W.lj_fluid(n, 0.8, 1.0, 3).config(), "fp64", "phys")
        eng.run_n(1)
        info = eng.launch_info()
        assert info["nb_blocks_per_sm"] == 2 and info["nb_form"] == "chunk32" and not info["min_image_kernel"]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("start", [5, 7])
def test_timed_ref_steps_are_the_steps_that_run(precision, start):
    """REF: timed steps issue a first evaluation where run_n does, from any point of
    the list cadence, and leave the state and the cadence that run_n leaves."""
    a, b = _engine(_argon(4), precision, "ref"), _engine(_argon(4), precision, "ref")
    a.run_n(start), b.run_n(start)
    n0 = a.kernel_launches()
    a.run_n(20)
    n1 = a.kernel_launches()
    t = b.step_timed(20, 0)
    assert t["kernel_launches"] == n1 - n0 - (precision == "fp64")  # less the mark of the step that is read
    a.run_n(7), b.run_n(7)
    assert np.array_equal(a.positions, b.positions) and np.array_equal(a.velocities, b.velocities)


def _long_cases():
    def lj(thermostat="none"):
        return _set(W.lj_fluid(500, 0.8, 1.0, 3).config(), thermostat)

    def water(barostat="none"):
        c = W.water_box(n_mol=430, box=(430 / 33.43) ** (1 / 3), seed=5, spacing=0.1).config()
        return _set(c, "nose-hoover", barostat)

    return {"lj": (lj, "mixed", "phys"), "lj-nh": (lambda: lj("nose-hoover"), "mixed", "phys"),
            "lj-andersen": (lambda: lj("andersen"), "mixed", "phys"),
            "lj-fp64": (lambda: lj("berendsen"), "fp64", "phys"),
            "water": (water, "mixed", "phys"), "water-fp64": (water, "fp64", "phys"),
            "water-npt": (lambda: water("berendsen"), "mixed", "phys"),
            "rigid": (lambda: _rigid_water(430, "tri"), "mixed", "phys"),
            "argon-ref": (lambda: _argon(4), "mixed", "ref"), "argon-ref-fp64": (lambda: _argon(4), "fp64", "ref"),
            "argon-ref-npt": (lambda: _set(_argon(4), "berendsen", "berendsen"), "mixed", "ref")}


def _set(c, thermostat, barostat="none"):
    c.thermostat.type, c.barostat.type = thermostat, barostat
    if thermostat != "none":
        c.thermostat.temperature = 120.0
    return c


@pytest.mark.parametrize("case", list(_long_cases()))
def test_several_steps_per_launch(case):
    """Tables that keep running take four steps (REF: the five of a list cadence) per
    graph once 256 have run.  Calls of mixed length beyond that point leave the
    state, bit for bit, that calls of three steps leave, which never do."""
    make, precision, profile = _long_cases()[case]
    a, b = _engine(make(), precision, profile), _engine(make(), precision, profile)
    a.run_n(260)
    for n in (9, 4, 1, 7, 3, 16, 5):
        a.run_n(n)
    for _ in range(101):
        b.run_n(3)
    b.run_n(2)
    if precision == "mixed" and case != "argon-ref-npt":
        # the later steps of a graph begin in the update of the one before: fewer launches
        assert a.kernel_launches() < b.kernel_launches()
    assert np.array_equal(a.positions, b.positions) and np.array_equal(a.velocities, b.velocities)
    assert np.array_equal(a.forces, b.forces)
    sa, sb = a.scalars(), b.scalars()
    assert (sa.step, sa.time, sa.box) == (sb.step, sb.time, sb.box)
    assert (sa.kinetic_energy, list(sa.e_terms)) == (sb.kinetic_energy, list(sb.e_terms))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("profile", ["phys", "ref"])
def test_targets_inside_a_launch_of_several_steps(profile, precision):
    """Replicas that reach their targets inside a graph of several steps stop there,
    with their energies, while the others go on: bit for bit as in calls of three."""
    from dmd_b200.batch import Batch
    cfgs = [_argon(3 + k % 2, k) if profile == "ref" else _set(W.lj_fluid(400 + 90 * k, 0.8, 1.0, k).config(), th)
            for k, th in enumerate(("none", "berendsen", "nose-hoover", "none", "berendsen"))]
    targets = [261, 266, 279, 303, 1000]
    out = []
    for calls in ((260, 45), (3,) * 101 + (2,)):
        b = Batch(precision=precision, profile=profile)
        slots = [b.admit(c, n) for c, n in zip(cfgs, targets)]
        for n in calls:
            b.step(n)
        out.append([(b.scalars(k).step, b.scalars(k).kinetic_energy, list(b.scalars(k).e_terms[:]) if n < 1000 else None,
                     b.positions(k).tobytes(), b.velocities(k).tobytes()) for k, n in zip(slots, targets)])
    assert [o[0] for o in out[0]] == [261, 266, 279, 303, 305]
    assert out[0] == out[1]


def _same_energies(e, e_o, tol):
    for k in ("lj", "coul_real", "coul_recip", "total"):
        got = sum(e.values()) if k == "total" else e[k]
        assert abs(got - e_o[k]) <= 10 * tol * max(abs(e_o[k]), 1.0), (k, got, e_o[k])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n_mol,spacing", [(130, 0.2), (400, 0.105), (400, 0.022)])
def test_pme_mesh_energies(oracle, n_mol, spacing, precision):
    """Energies on the meshes of test_pme_mesh_sizes, term by term (single-point
    tolerances)."""
    box = (n_mol / 33.43) ** (1 / 3)
    c = W.water_box(n_mol=n_mol, box=box, seed=9, spacing=spacing).config()
    _, e = _engine(c, precision, "phys").compute_forces()
    _same_energies(e, oracle.forces(c, "phys")[1], {"fp64": 1e-9, "mixed": 1e-5}[precision])


@pytest.mark.parametrize("alpha", [3.12, 4.2])
@pytest.mark.parametrize("rc_lj", [1.0, 0.85])
@pytest.mark.parametrize("n_mol", [110, 429])
def test_fp64_pair_energies(oracle, n_mol, rc_lj, alpha):
    """Energies and the virial of the pair forms of test_fp64_pair_forms: of a single
    point, and of the evaluation that ends a run (1e-7: the positions there agree to
    1e-10 nm or better, on forces of up to 1e4)."""
    box = (n_mol / 33.43) ** (1 / 3)
    c = W.water_box(n_mol=n_mol, box=box, seed=5, spacing=box / round(box / 0.1)).config()
    c.lj_cutoff, c.ewald_coeff = rc_lj, alpha
    eng = _engine(c, "fp64", "phys")
    _same_energies(eng.compute_forces()[1], oracle.forces(c, "phys")[1], 1e-9)
    oe = oracle.engine(c, "phys")
    oe.step(5)
    run = _engine(c, "fp64", "phys")
    run.run_n(5)
    e_o = oe.energy()
    _same_energies(run.energy_terms(), e_o, 1e-8)
    assert abs(run.scalars().virial - e_o["virial"]) <= 1e-7 * abs(e_o["virial"])
