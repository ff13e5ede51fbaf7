"""Contacts of more spheres than the all-particles search takes (2048), through
the cell list, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from _util import particle_errors, rel_l2
from interparts_mpich_gb300 import IBMSolver
from interparts_mpich_gb300.cases import Case
from oracle.oracle import OracleSolver

pytestmark = pytest.mark.gpu


def crowd_case(unequal):
    """1100 pairs about the sites of a lattice, in all directions, each sphere
    approaching its partner from just outside contact; sites on the periodic edges
    in x and y, the lowest and highest pairs upright next to the walls."""
    h = 1.0 / 96
    m, pitch = np.array([11, 10, 10]), np.array([108 / 11, 9.6, 9.6]) * h
    rng = np.random.default_rng(8)
    ijk = np.stack(np.unravel_index(np.arange(m.prod()), m), 1)
    site = ijk * pitch + np.array([0.0, 0.0, 0.5]) * pitch
    n = len(site)
    r = rng.uniform(1.6, 2.0, (2, n)) * h if unequal else np.full((2, n), 2.0 * h)
    e = rng.standard_normal((n, 3))
    low, high = ijk[:, 2] == 0, ijk[:, 2] == m[2] - 1
    e[low | high] = (0, 0, 1)
    e /= np.linalg.norm(e, axis=1)[:, None]
    half = 0.5 * (r[0] + r[1]) * rng.uniform(1.002, 1.03, n)
    c = np.stack([site - half[:, None] * e, site + half[:, None] * e])
    dz = np.where(low, 1.02 * r[0] - c[0, :, 2], np.where(high, 96 * h - 1.02 * r[1] - c[1, :, 2], 0.0))
    c[:, :, 2] += dz
    # towards each other, or both to the wall beside one of them
    v = 0.2 * np.stack([e, -e]) + rng.uniform(-0.02, 0.02, (2, n, 3))
    v[0, low, 2], v[1, low, 2], v[0, high, 2], v[1, high, 2] = -0.15, -0.35, 0.35, 0.15
    c[:, :, 0] %= 108 * h
    c[:, :, 1] %= 96 * h
    mix = rng.permutation(2 * n)  # partners far apart in the list
    return Case(name="crowd", itot=108, jtot=96, ktot=96, lx=108 * h, ly=96 * h, lz=96 * h, radius=2.0 * h, np=2 * n,
                visc=1.0 / 300.0, ratiorho=8.0, flow="pur", perturb=0.0, centres=c.reshape(-1, 3)[mix],
                velocities=v.reshape(-1, 3)[mix], radii=r.reshape(-1)[mix] if unequal else None)


@pytest.mark.parametrize("unequal", [False, True])
def test_contact_lists_through_the_cell_list(gpu_lib, unequal):
    case = crowd_case(unequal)
    assert case.np == 2200
    ps = case.initial_particles(lagrangian=False)
    # partners listed from before that are far away by now: found by the list, not
    # by the cells, and taken off it
    ps.qmax[::40] = 1
    ps.firstc.reshape(case.np, -1)[::40, 0] = (np.arange(0, case.np, 40) + 1000) % case.np + 1
    g, o = IBMSolver(case), OracleSolver(case)
    for s in (g, o):
        s.setup(particles=ps)
    pairs, walls = set(), set()
    for step in range(6):
        for s in (g, o):
            s.rk3_step(2e-3)
        pg, po = g.get_particles(lagrangian=False), o.get_particles(lagrangian=False)
        assert pg.contact_lists() == po.contact_lists(), step
        for p, c in enumerate(po.contact_lists()):
            pairs |= {(p, q) for q in c if q <= case.np}
            walls |= {(p, q) for q in c if q > case.np}
        e = particle_errors(pg, po)
        assert max(e.values()) < 1e-10, (step, e)
        for f in ("colfx", "colfy", "colfz"):
            assert rel_l2(getattr(pg, f), getattr(po, f)) < 1e-9, (step, f)
    # most of the pairs have touched, some of them across the edges, and both walls
    x, y = case.centres[:, 0], case.centres[:, 1]
    far = [abs(x[p] - x[q - 1]) > 0.5 * case.lx or abs(y[p] - y[q - 1]) > 0.5 * case.ly for p, q in pairs]
    assert len(pairs) > 800 and sum(far) > 50 and {q for _, q in walls} == {case.np + 1, case.np + 2}
    g.close()
    o.close()
