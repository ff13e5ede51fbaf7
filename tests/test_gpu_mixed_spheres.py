"""Sphere integrals of the mixed forms at the edges of their batches, against the
oracle."""
from __future__ import annotations

import numpy as np
import pytest

from interparts_mpich_gb300 import IBM_MODE_MIXED, IBMSolver
from interparts_mpich_gb300.cases import Case
from oracle.oracle import OracleSolver

from test_gpu_plain_kernels import _state

pytestmark = pytest.mark.gpu


# radius in cells, particles, grid, ratio of the sides: below two cells, one
# sphere shared by several blocks, a batch of lines (up to 512) that is not full,
# two batches in a block (24 dx, enough spheres for one block each, the lines not
# a multiple of a batch), many batches, and cells of unequal sides
@pytest.mark.parametrize("r,n,grid,aspect", [(0.8, 3, (24, 24, 12), 1.0), (1.6, 5, (24, 24, 24), 1.0),
                                             (8.0, 1, (32, 32, 32), 1.0), (8.0, 60, (96, 96, 96), 1.0),
                                             (12.0, 60, (108, 108, 108), 1.0), (12.3, 110, (96, 128, 72), 1.0),
                                             (47.0, 1, (128, 108, 104), 1.0), (6.0, 60, (48, 64, 32), 1.7)])
def test_sphere_integrals_mixed(gpu_lib, r, n, grid, aspect):
    nx, ny, nz = grid
    h = 1.0 / 64
    lx, ly, lz = nx * h, ny * h * aspect, nz * h / aspect
    rng = np.random.default_rng(3)
    rad = r * h
    # anywhere in x and y (periodic images), clear of the walls in z
    c = np.stack([rng.uniform(0, lx, n), rng.uniform(0, ly, n), rng.uniform(rad, lz - rad, n)], 1)
    case = Case(name="spheres", itot=nx, jtot=ny, ktot=nz, lx=lx, ly=ly, lz=lz, visc=1e-2, radius=rad, np=n, centres=c)
    fields = _state(case, 11)
    for q in "uvw":  # what the mixed form holds
        fields[q] = np.asfortranarray(fields[q].astype(np.float32).astype(np.float64))
    got = []
    for s in (IBMSolver(case, mode=IBM_MODE_MIXED), OracleSolver(case)):
        vol = s.setup(fields=fields)
        p = s.get_particles(lagrangian=False)
        got.append((vol, np.stack([p.intu, p.intv, p.intw]), np.stack([p.intomx, p.intomy, p.intomz])))
    # FP32 corner distances: three rounded squares and two sums (3 x 2^-24 of the
    # square), an approximate root (2^-23) and the rounded radius (2^-25): 4 x 2^-24
    # of the radius.  A cut cell's fraction is a quotient of sums of eight of them,
    # whose magnitudes add up to three of its smallest sides or more: off by 16
    # distance errors over that.  Cut cells: under 25 (R + 1)^2, by the smallest side
    side = min(h, h * aspect, h / aspect)
    cut = 25 * (rad / side + 1) ** 2
    off = 16 * 4 * 2.0 ** -24 * rad / (3 * side) * cut * h ** 3
    most = max(np.abs(fields[q]).max() for q in "uvw")
    assert abs(got[0][0] - got[1][0]) <= off
    assert np.max(np.abs(got[0][1] - got[1][1])) <= off * most
    assert np.max(np.abs(got[0][2] - got[1][2])) <= 2 * off * most * (rad + 2 * side)
    # (a line of cells through the centre is worth far more)
    assert off * most < 2 * rad / side * h ** 3
