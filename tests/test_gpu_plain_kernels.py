"""Tiled and transform kernels at the edges of their ranges, against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

from interparts_mpich_gb300 import IBMSolver, _abi
from interparts_mpich_gb300.cases import Case, boundp
from oracle.oracle import OracleSolver

from _util import PLAIN_TOL_CALL, interior, rel_l2

pytestmark = pytest.mark.gpu


def _state(case, seed):
    """Random interior fields, walls as bounduvw leaves them."""
    c = Case(name="noise", itot=case.itot, jtot=case.jtot, ktot=case.ktot, lx=case.lx, ly=case.ly, lz=case.lz,
             visc=case.visc, seed=seed, flow="poi", perturb=0.3, bc_top=case.bc_top, bc_bot=case.bc_bot)
    f = c.initial_fields()
    rng = np.random.default_rng(seed)
    for n in ("p", "durk", "dvrk", "dwrk"):
        f[n] = np.asfortranarray(rng.uniform(-1, 1, case.shape))
    boundp(f["p"])
    return f


# one cell beyond, at and below the 32-cell tile width, tiles of unequal
# sides, the smallest grid, more planes than one z chunk
@pytest.mark.parametrize("grid", [(4, 4, 4), (6, 32, 9), (32, 8, 5), (36, 9, 70), (64, 27, 4), (54, 16, 33), (108, 12, 6)])
@pytest.mark.parametrize("buoyancy", [False, True])
def test_predictor_tiles(gpu_lib, grid, buoyancy):
    nx, ny, nz = grid
    case = Case(name="tiles", itot=nx, jtot=ny, ktot=nz, lx=nx / 32, ly=ny / 24, lz=nz / 40, visc=1e-2)
    fields = _state(case, 5)
    dt = 1e-3
    solvers = [IBMSolver(case), OracleSolver(case)]
    out = []
    for s in solvers:
        s.setup(fields=fields)
        if buoyancy:
            rng = np.random.default_rng(9)
            s.set_scalar(np.asfortranarray(rng.uniform(-1, 1, case.shape)), beta=0.3)
        got = []
        for r in (1, 2, 3):
            s.rk(r, dt)
            got.append({n: interior(a).copy() for n, a in s.get_intermediate().items()})
        f = s.get_fields()
        got.append({n: interior(f[n]).copy() for n in ("durk", "dvrk", "dwrk")})
        out.append(got)
    for a, b in zip(*out):
        for n in a:
            assert rel_l2(a[n], b[n]) < PLAIN_TOL_CALL, n


# lengths of two radices (12 x 16 = 192, 9 x 9, 2 x 2, 16 x 16), of three
# (6 x 8 x 8 = 384, 6 x 9 x 9 = 486), of none (2 and 3, left to the general stages)
@pytest.mark.parametrize("grid", [(8, 4, 5), (6, 18, 4), (162, 16, 4), (54, 54, 6), (384, 6, 4), (768, 4, 4), (8, 384, 4),
                                  (16, 486, 4), (512, 12, 4), (4, 6, 8)])
def test_projection_lengths(gpu_lib, grid):
    nx, ny, nz = grid
    case = Case(name="fft", itot=nx, jtot=ny, ktot=nz, lx=nx / 32, ly=ny / 32, lz=nz / 32, visc=1e-2)
    fields = _state(case, 7)
    out = []
    for s in (IBMSolver(case), OracleSolver(case)):
        s.setup(fields=fields)
        s.rk(1, 1e-3)
        s.project(1, 1e-3)
        out.append({n: interior(a) for n, a in s.get_fields().items() if n in "uvwp"})
    for n in "uvw":
        assert rel_l2(out[0][n], out[1][n]) < PLAIN_TOL_CALL, n
    d = out[0]["p"] - out[1]["p"]  # the zero mode is free: its pin differs with the rounding
    assert np.linalg.norm(d - d.mean()) < 10 * PLAIN_TOL_CALL * np.linalg.norm(out[1]["p"])


# odd lengths in y (the oracle's eigenvalue table, as the reference's, covers
# even ones only): the projected velocity is free of divergence, to six
# rounded terms of size 2 x 32 with room for the solve (2^-53 each)
@pytest.mark.parametrize("grid", [(16, 81, 4), (8, 729, 4), (12, 27, 7)])
def test_projection_divergence(gpu_lib, grid):
    nx, ny, nz = grid
    case = Case(name="odd", itot=nx, jtot=ny, ktot=nz, lx=nx / 32, ly=ny / 32, lz=nz / 32, visc=1e-2)
    s = IBMSolver(case)
    s.setup(fields=_state(case, 7))
    s.rk(1, 1e-3)
    s.project(1, 1e-3)
    assert s.chkdiv()[1] < 1e-11


# FP32 transforms: every pair of stages a pass is made of (4x4, 4x2, 4x3, 2x3,
# 3x3, single ones), two and three passes, the four-step lengths, and lengths
# left to the general stages.  Divergence after the projection: terms of up to
# 32 x 2, six a cell, rounded at 2^-24 in about 20 steps: 5e-4 with room for all
# of one sign
@pytest.mark.parametrize("grid", [(32, 16, 4), (64, 256, 4), (128, 64, 4), (512, 128, 4), (16, 12, 4), (48, 36, 5),
                                  (54, 27, 4), (192, 108, 4), (324, 162, 4), (384, 243, 4), (768, 486, 4), (8, 384, 4),
                                  (16, 512, 4), (12, 8, 6)])
def test_projection_fp32(gpu_lib, grid):
    nx, ny, nz = grid
    case = Case(name="fft32", itot=nx, jtot=ny, ktot=nz, lx=nx / 32, ly=ny / 32, lz=nz / 32, visc=1e-2)
    s = IBMSolver(case, mode=_abi.IBM_MODE_MIXED)
    s.setup(fields=_state(case, 7))
    s.rk(1, 1e-3)
    s.project(1, 1e-3)
    assert s.chkdiv()[1] < 5e-4


# radius in cells, particles, grid: below two cells (the reference's inner
# test reaches past the surface), one sphere shared by several blocks, a box
# of one slab, of several, of node planes too large for shared memory, and
# cells of unequal sides
@pytest.mark.parametrize("r,n,grid,aspect", [(0.8, 3, (24, 24, 12), 1.0), (1.6, 5, (24, 24, 24), 1.0),
                                             (8.0, 1, (32, 32, 32), 1.0), (8.0, 40, (96, 96, 96), 1.0),
                                             (14.0, 4, (72, 72, 48), 1.0), (24.0, 2, (108, 54, 64), 1.0),
                                             (47.0, 1, (128, 108, 104), 1.0), (6.0, 7, (48, 64, 32), 1.7)])
def test_sphere_integrals(gpu_lib, r, n, grid, aspect):
    nx, ny, nz = grid
    h = 1.0 / 64
    lx, ly, lz = nx * h, ny * h * aspect, nz * h / aspect
    rng = np.random.default_rng(3)
    rad = r * h
    # anywhere in x and y (periodic images), clear of the walls in z
    c = np.stack([rng.uniform(0, lx, n), rng.uniform(0, ly, n), rng.uniform(rad, lz - rad, n)], 1)
    case = Case(name="spheres", itot=nx, jtot=ny, ktot=nz, lx=lx, ly=ly, lz=lz, visc=1e-2, radius=rad, np=n, centres=c)
    fields = _state(case, 11)
    got = []
    for s in (IBMSolver(case), OracleSolver(case)):
        vol = s.setup(fields=fields)
        p = s.get_particles(lagrangian=False)
        got.append((vol, np.stack([p.intu, p.intv, p.intw]), np.stack([p.intomx, p.intomy, p.intomz])))
    assert abs(got[0][0] - got[1][0]) < PLAIN_TOL_CALL * got[1][0]
    for q in (1, 2):
        assert rel_l2(got[0][q], got[1][q]) < PLAIN_TOL_CALL


# planes below, at and beyond a chunk of 256 cells, more chunks than blocks;
# noise, all at rest (with a viscosity that leaves the limit to the rest
# value), one moving cell in the last chunk, speeds about the rest limit
@pytest.mark.parametrize("grid", [(4, 4, 4), (16, 16, 9), (54, 27, 5), (64, 81, 70)])
@pytest.mark.parametrize("flow", ["noise", "rest", "one", "tiny"])
@pytest.mark.parametrize("mode", [_abi.IBM_MODE_PLAIN_FP64, _abi.IBM_MODE_MIXED])
def test_time_step_control(gpu_lib, grid, flow, mode):
    nx, ny, nz = grid
    case = Case(name="control", itot=nx, jtot=ny, ktot=nz, lx=nx / 32, ly=ny / 24, lz=nz / 40,
                visc=1e-4 if flow == "noise" else 1e-14)
    f = _state(case, 3)
    if flow != "noise":
        for n in "uvw":
            f[n][:] = 0
    if flow == "one":
        f["v"][nx - 1, ny - 1, nz - 1] = 0.7
    if flow == "tiny":
        f["u"][2, 2, 1:nz:2] = 5e-12
        f["w"][3, 1:4, 2] = 0.9e-12
    for n in "uvw":  # what the mixed form holds
        f[n] = np.asfortranarray(f[n].astype(np.float32).astype(np.float64))
    g, o = IBMSolver(case, mode=mode), OracleSolver(case)
    for s in (g, o):
        s.setup(fields=f)
    assert abs(g.chkdt() - o.chkdt()) <= 1e-14 * o.chkdt()
    # a divergence of six terms of size 40 x 2, a sum of n of them: 2^-53 each
    a, b = g.chkdiv(), o.chkdiv()
    assert abs(a[1] - b[1]) <= 1e-13
    # no divergence anywhere: the library names the first cell, the oracle none
    assert tuple(a[2]) == (tuple(b[2]) if b[1] > 0 else (1, 1, 1))
    assert abs(a[0] - b[0]) <= 1e-12 * nx * ny * nz


# rows below, at and beyond a warp's 32 x 4 cells; values of every kind that
# rounds: ties, the largest and smallest of FP32, subnormal, zero of both signs
@pytest.mark.parametrize("grid", [(4, 9, 4), (36, 27, 4), (128, 4, 5), (144, 9, 6), (256, 12, 4)])
@pytest.mark.parametrize("mode", [_abi.IBM_MODE_PLAIN_FP64, _abi.IBM_MODE_MIXED])
def test_field_conversions(gpu_lib, grid, mode):
    nx, ny, nz = grid
    case = Case(name="layout", itot=nx, jtot=ny, ktot=nz, lx=nx / 32, ly=ny / 32, lz=nz / 32, visc=1e-2)
    rng = np.random.default_rng(1)

    def field():
        f = rng.uniform(-1, 1, case.shape) * 10.0 ** rng.integers(-44, 37, case.shape)
        odd = np.array([0.0, -0.0, 1 + 2.0 ** -24, 1 + 3 * 2.0 ** -24, -1 + 2.0 ** -25, 3.4028234e38, 1.1754944e-38,
                        1.17549429e-38, 2.0 ** -149, 2.0 ** -150, 2.0 ** 126, 2 - 2.0 ** -30, -(2.0 ** -74), 2.0 ** -75])
        pick = rng.random(case.shape) < 0.2
        f[pick] = rng.choice(odd, pick.sum())
        return np.asfortranarray(f)

    f = {n: field() for n in ("u", "v", "w", "p", "durk", "dvrk", "dwrk")}
    s = IBMSolver(case, mode=mode)
    s.set_fields(**f)
    got = s.get_fields()
    for n, a in f.items():
        want = a.copy()
        if mode == _abi.IBM_MODE_MIXED:
            hi = a.astype(np.float32)
            want = hi.astype(np.float64)
            if n == "p":
                want += (a - want).astype(np.float32)
        want[0], want[-1] = want[-2], want[1]
        want[:, 0], want[:, -1] = want[:, -2], want[:, 1]
        assert np.array_equal(got[n], want), n
