"""The mixed form's shared-memory boxes at the edges of their kinds, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from _util import interior, rel_l2
from interparts_mpich_gb300 import IBM_MODE_MIXED, IBMSolver
from interparts_mpich_gb300.cases import Case
from oracle.oracle import OracleSolver

pytestmark = pytest.mark.gpu

# FP32 delta weights and sums are off by 2^-22 of the velocities; u and w are
# about thirty times smaller than v, which the rotating spheres mix into them,
# and three passes add up
TOL = 2e-5


# diameter in cells, spheres, grid: ordered points in quads (16), rows of single
# cells (grid not a multiple of four), the most points that are ordered (25.5),
# more of them in rows of nine quads (27), a box too large for shared memory
# (40), a box wider than half the period (20 in 40), one sphere
@pytest.mark.parametrize("d,n,grid", [(16.0, 9, (64, 64, 64)), (12.0, 6, (54, 48, 40)), (25.5, 2, (96, 64, 40)),
                                      (27.0, 2, (96, 64, 40)), (40.0, 1, (96, 96, 64)), (20.0, 1, (32, 48, 32)),
                                      (8.0, 1, (24, 24, 24))])
@pytest.mark.parametrize("rotation", [0, 1])
def test_forcing_boxes(gpu_lib, d, n, grid, rotation):
    nx, ny, nz = grid
    h = 1.0 / 64
    rng = np.random.default_rng(5)
    lx, ly, lz = nx * h, ny * h, nz * h
    r = d * h / 2
    # side by side in x and y (periodic images among them), clear of the walls
    m = int(np.ceil(np.sqrt(n)))
    c = np.array([[(q % m + 0.03) * lx / m, (q // m + 0.4) * ly / m, rng.uniform(r + h, lz - r - h)] for q in range(n)])
    case = Case(name="boxes", itot=nx, jtot=ny, ktot=nz, lx=lx, ly=ly, lz=lz, visc=1e-3, radius=r, np=n, centres=c,
                rotation=rotation)
    ps = case.initial_particles(lagrangian=False)
    ps.u[:], ps.v[:], ps.w[:] = rng.uniform(-0.1, 0.1, (3, n))
    if rotation:
        ps.omx[:], ps.omy[:], ps.omz[:] = rng.uniform(-1, 1, (3, n))
    dt = 1e-3
    got = []
    for s in (IBMSolver(case, mode=IBM_MODE_MIXED), OracleSolver(case)):
        s.setup(particles=ps)
        s.rk(1, dt)
        s.forcing_loop(dt, 3)
        f = {q: interior(a) for q, a in s.get_intermediate().items()}
        p = s.get_particles(lagrangian=False)
        f["force"] = np.stack([p.fxltot, p.fyltot, p.fzltot])
        got.append(f)
    for q in got[0]:
        assert rel_l2(got[0][q], got[1][q]) < TOL, q


# the largest boxes: spheres of up to 32 cells (rows padded to quads take more
# cells than the rows), of 34, the last that fit, of 35, and spheres whose boxes
# are far beyond the shared memory beside smaller ones
@pytest.mark.parametrize("d", [(31.5, 24.0), (34.0,), (35.0,), (42.0, 14.0)])
@pytest.mark.parametrize("unequal", [False, True])
def test_forcing_largest_boxes(gpu_lib, d, unequal):
    nx, ny, nz = 144, 96, 64
    h = 1.0 / 64
    rng = np.random.default_rng(6)
    n = len(d)
    d = np.array(d) if unequal else np.full(n, d[0])
    c = np.array([[(q + 0.03) * nx * h / n, (q + 0.4) * ny * h / n, rng.uniform(22.5, 41.5) * h] for q in range(n)])
    case = Case(name="boxes", itot=nx, jtot=ny, ktot=nz, lx=nx * h, ly=ny * h, lz=nz * h, visc=1e-3,
                radius=d[0] * h / 2, np=n, centres=c, radii=d * h / 2 if unequal else None)
    ps = case.initial_particles(lagrangian=False)
    ps.u[:], ps.v[:], ps.w[:] = rng.uniform(-0.1, 0.1, (3, n))
    got = []
    for s in (IBMSolver(case, mode=IBM_MODE_MIXED), OracleSolver(case)):
        s.setup(particles=ps)
        s.rk(1, 1e-3)
        s.forcing_loop(1e-3, 3)
        f = {q: interior(a) for q, a in s.get_intermediate().items()}
        p = s.get_particles(lagrangian=False)
        f["force"] = np.stack([p.fxltot, p.fyltot, p.fzltot])
        got.append(f)
    for q in got[0]:
        assert rel_l2(got[0][q], got[1][q]) < TOL, q
