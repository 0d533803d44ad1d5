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
