"""The projection's transforms: the FP32 ones to the bit, both against a 64-bit
restatement at odd lengths and at every kind of pass."""
from __future__ import annotations

import hashlib

import numpy as np
import pytest

from interparts_mpich_gb300 import IBM_MODE_MIXED, IBM_MODE_PLAIN_FP64, IBMSolver
from interparts_mpich_gb300.cases import Case

from _util import PLAIN_TOL_CALL, interior

pytestmark = pytest.mark.gpu

# first digits of the SHA-256 of u, v, w, p after a projection of one and of two
# solves.  From kernels with one pass through shared memory a stage and, at powers
# of two, the four-step scheme: an independent set of kernels with the same stages
# and the same fused products, which the passes in registers stand in for.  Every
# pair of stages a pass is made of, two and three passes, the four-step lengths,
# and lengths left to the general stages
BITS = {
    (32, 16, 4): ("9d25398ed6b9", "f5ce1105bbd1"),
    (64, 256, 4): ("3a01c91d453e", "f37aa3386b75"),
    (128, 64, 4): ("f869aefab259", "da6ca7765f4a"),
    (512, 128, 4): ("b1fac208f455", "1d28d7523a4c"),
    (16, 12, 4): ("474bf65d0b16", "1d5a1c81e016"),
    (48, 36, 5): ("ef178f9019b5", "3f9e13478d63"),
    (54, 27, 4): ("95b87686567b", "24eaef27d35b"),
    (192, 108, 4): ("972353172fbe", "13494dc5f075"),
    (324, 162, 4): ("e5d6944ce4db", "808a76c24acf"),
    (384, 243, 4): ("888e73a39790", "4c58e609317d"),
    (768, 486, 4): ("e1e666309ecb", "7a5dd3bf091c"),
    (8, 384, 4): ("d636a90d7f46", "dfa00d4653e8"),
    (16, 512, 4): ("666e54eb963c", "5c6230253bf8"),
    (12, 8, 6): ("9106337ac233", "f2dfc3bdfd01"),
    (4, 4, 4): ("58a977ec42f6", "37ccb9081022"),
    (256, 192, 5): ("fa5d1644ac80", "e5df0fbe53f0"),
}


def _noise(case):
    rng = np.random.default_rng(7)
    return {n: np.asfortranarray(rng.uniform(-1, 1, case.shape).astype(np.float32).astype(np.float64))
            for n in ("u", "v", "w", "p", "durk", "dvrk", "dwrk")}


@pytest.mark.parametrize("grid", list(BITS))
@pytest.mark.parametrize("solves", [1, 2])
def test_fp32_projection_bits(gpu_lib, grid, solves):
    nx, ny, nz = grid
    case = Case(name="bits", itot=nx, jtot=ny, ktot=nz, lx=nx / 32, ly=ny / 32, lz=nz / 32, visc=1e-2)
    s = IBMSolver(case, mode=IBM_MODE_MIXED)
    s.setup(fields=_noise(case))
    s.set_projection_solves(solves)
    s.rk(1, 2.0 ** -10)
    s.project(1, 2.0 ** -10)
    f = s.get_fields()
    h = hashlib.sha256(b"".join(np.ascontiguousarray(interior(f[n])).tobytes() for n in "uvwp"))
    assert h.hexdigest()[:12] == BITS[grid][solves - 1]


def _restated(du, dx, step):
    """Projected u, v, w, and phi, the right-hand side's norm: rfft2 and a
    tridiagonal solve with Neumann ends a mode (axes i, j, k)."""
    u, v, w = (interior(a) for a in du)
    w = w.copy()
    w[:, :, -1] = 0
    wm = np.concatenate([np.zeros_like(w[:, :, :1]), w[:, :, :-1]], 2)
    rhs = (u - np.roll(u, 1, 0) + v - np.roll(v, 1, 1) + w - wm) / (dx * step)
    nx, ny, nz = rhs.shape
    a2 = 1 / dx ** 2
    lam = -4 * a2 * (np.sin(np.pi * np.arange(nx // 2 + 1) / nx)[:, None] ** 2 + np.sin(np.pi * np.arange(ny) / ny) ** 2)
    x = np.fft.rfft2(rhs, axes=(1, 0))
    cp = np.zeros(lam.shape + (nz,))
    for k in range(nz):
        den = lam - (2 if 0 < k < nz - 1 else 1) * a2 - (a2 * cp[:, :, k - 1] if k else 0)
        inv = np.divide(1.0, den, out=np.zeros_like(den), where=np.abs(den) > 1e-9 * a2)
        x[:, :, k] = (x[:, :, k] - (a2 * x[:, :, k - 1] if k else 0)) * inv
        cp[:, :, k] = a2 * inv
    for k in range(nz - 2, -1, -1):
        x[:, :, k] -= cp[:, :, k] * x[:, :, k + 1]
    phi = np.fft.irfft2(x, s=(ny, nx), axes=(1, 0))
    up = np.concatenate([phi[:, :, 1:], phi[:, :, -1:]], 2)
    f = step / dx
    out = [u - f * (np.roll(phi, -1, 0) - phi), v - f * (np.roll(phi, -1, 1) - phi), w - f * (up - phi)]
    return out, phi - phi.mean(), np.linalg.norm(rhs)


@pytest.mark.parametrize("grid", [(16, 81, 4), (8, 729, 4), (12, 27, 7), (54, 9, 5), (162, 243, 4), *BITS])
@pytest.mark.parametrize("mode", [IBM_MODE_PLAIN_FP64, IBM_MODE_MIXED])
def test_projection_restated(gpu_lib, grid, mode):
    nx, ny, nz = grid
    dx, dt = 1.0 / 32, 2.0 ** -10
    case = Case(name="restated", itot=nx, jtot=ny, ktot=nz, lx=nx * dx, ly=ny * dx, lz=nz * dx, visc=1e-2)
    fields = _noise(case)
    s = IBMSolver(case, mode=mode)
    s.setup(fields=fields)
    s.rk(1, dt)
    du = [s.get_intermediate()[n] for n in ("dudt", "dvdt", "dwdt")]
    s.project(1, dt)
    got = s.get_fields()
    step = 32 * dt / 60
    want, phi, rhs = _restated(du, dx, step)
    # transforms of some 20 roundings in the norm, each way: the right-hand side's
    # error over the smallest eigenvalue (its root for the gradient), the
    # solution's under a difference; and the roundings of the correction
    least = 4 / dx ** 2 * min(np.sin(np.pi / nx), np.sin(np.pi / ny), np.sin(np.pi / (2 * nz))) ** 2
    eps = 20 * (2.0 ** -24 if mode == IBM_MODE_MIXED else 2.0 ** -53)
    tol_phi = eps * (rhs / least + np.linalg.norm(phi))
    tol_u = eps * step * (rhs / least ** 0.5 + 2 / dx * np.linalg.norm(phi)) + eps * np.linalg.norm(want)
    for n, a in zip("uvw", want):
        assert np.linalg.norm(interior(got[n]) - a) <= tol_u, n
    d = interior(got["p"]) - interior(fields["p"])
    assert np.linalg.norm(d - d.mean() - phi) <= tol_phi
    if mode == IBM_MODE_PLAIN_FP64:
        assert np.linalg.norm(interior(got["u"]) - want[0]) < PLAIN_TOL_CALL * np.linalg.norm(want[0])
