"""Force and torque totals of the plain form's forcing loop, against the oracle."""
from __future__ import annotations

import math

import numpy as np
import pytest

from interparts_mpich_gb300 import IBMSolver
from interparts_mpich_gb300.cases import Case
from oracle.oracle import OracleSolver

from _util import PLAIN_TOL_CALL

pytestmark = pytest.mark.gpu


# fewer points than a warp, about the four warps that sum them (127, 129), many
# rounds of them; turned spheres, whose torque about the angle takes cos and sin
@pytest.mark.parametrize("r,points", [(1.2, 11), (3.46, 127), (3.485, 129), (8.0, 746)])
@pytest.mark.parametrize("passes", [1, 3])
def test_force_and_torque_sums(gpu_lib, r, points, passes):
    h = 1.0 / 64
    n = 5
    rng = np.random.default_rng(2)
    case = Case(name="sums", itot=48, jtot=64, ktot=32, lx=48 * h, ly=64 * h, lz=32 * h, visc=1e-2, radius=r * h, np=n,
                centres=np.stack([rng.uniform(0, 48 * h, n), rng.uniform(0, 64 * h, n),
                                  rng.uniform(9 * h, 23 * h, n)], 1), rotation=1)
    assert case.nl == points
    ps = case.initial_particles(lagrangian=False)
    ps.u[:], ps.v[:], ps.w[:] = rng.uniform(-0.1, 0.1, (3, n))
    ps.omx[:], ps.omy[:], ps.omz[:] = rng.uniform(-1, 1, (3, n))
    ps.phi[:] = rng.uniform(-3, 3, n)
    got = []
    for s in (IBMSolver(case), OracleSolver(case)):
        s.setup(particles=ps)
        s.rk(1, 1e-3)
        s.forcing_loop(1e-3, passes)
        got.append(s.get_particles())
    a, b = got
    shell = (r - 0.3) * h
    dv = 4.0 / 3.0 * math.pi * ((shell + 0.5 * h) ** 3 - (shell - 0.5 * h) ** 3) / points
    # the point forces agree to the per-call tolerance of their norm, so their
    # sums to that times the root of the number of points
    tol = PLAIN_TOL_CALL * math.sqrt(3 * n * points) * dv * np.linalg.norm([b.fxl, b.fyl, b.fzl])
    for q in ("fxltot", "fyltot", "fzltot"):
        assert np.max(np.abs(getattr(a, q) - getattr(b, q))) <= tol, q
    for q in ("torqxltot", "torqyltot", "torqzltot", "torqtheta"):
        assert np.max(np.abs(getattr(a, q) - getattr(b, q))) <= 2 * shell * tol, q
    assert np.max(np.abs(b.torqtheta)) > 1e6 * shell * tol


# the reference leaves out a point whose periodic image rounds to a cell outside
# the grid: next to the planes half a cell inside the domain and beyond it.  The
# first point of the table lies level with its sphere's centre in y
@pytest.mark.parametrize("ny", [32, 48, 108])
def test_points_at_the_image_planes(gpu_lib, ny):
    h = 1.0 / ny
    half = 0.5 / float(ny)
    y = [np.nextafter(half, 0), half, np.nextafter(half, 1), np.nextafter(1 + half, 0), 1 + half, 0.37, 0.0, 1.0]
    case = Case(name="planes", itot=32, jtot=ny, ktot=24, lx=32 * h, ly=1.0, lz=24 * h, visc=1e-2, radius=3.3 * h,
                np=len(y), centres=np.stack([np.full(len(y), 9.3 * h), y, np.full(len(y), 11.7 * h)], 1))
    got = []
    for s in (IBMSolver(case), OracleSolver(case)):
        s.setup()
        got.append(s.get_particles())
    kept = [int(np.count_nonzero(p.zfp.reshape(len(y), -1)[0])) for p in got]
    assert kept[0] == kept[1] and (ny == 108 or kept[1] == case.nl - 1)
    for q in ("xfp", "yfp", "zfp", "ul"):
        assert np.array_equal(getattr(got[0], q), getattr(got[1], q)), q
