"""Workloads that the library is timed on.

Each case is a plain dict.  `listed` names the fixed ones, `draw` gives more
of the same ranges, `prepare` builds what a program holds before the call,
`run` is one pass through the public entry points and `exact` restates the
result in 64 bits with plain torch.

Fields live in device memory in the reference layout (k, j, i with one ghost
layer; the C ABI takes device pointers as they are), the particle state on the
host, all work on one CUDA stream.  The grid spacing is a power of two.
Passes that move the state (time steps, the particle update) start from the
prepared fields and particles again, as a program that hands its own state to
the library and takes it back does.
"""
import ctypes
import math

import numpy as np
import torch

from interparts_mpich_gb300 import _abi
from interparts_mpich_gb300.cases import Case, derived_nl, fibonacci_sphere
from interparts_mpich_gb300.solver import IBMSolver

MODES = {"plain": _abi.IBM_MODE_PLAIN_FP64, "mixed": _abi.IBM_MODE_MIXED, "learned": _abi.IBM_MODE_MIXED_LEARNED}
BC = {"noslip": _abi.IBM_BC_NOSLIP, "freeslip": _abi.IBM_BC_FREESLIP, "periodic": _abi.IBM_BC_PERIODIC}
RK = {1: (32.0, 0.0, 0.0), 2: (8.0, 25.0, 17.0), 3: (20.0, 45.0, 25.0)}  # rk1..rk3 coefficients, in 60ths
RKAB = {1: 32.0 / 60.0, 2: 8.0 / 60.0, 3: 20.0 / 60.0}  # their sum per stage: the projection's step
PRAN, BETA = 0.7, 0.02


def _case(name, kind, form, nx, ny, nz, **kw):
    c = {"kind": kind, "form": form, "nx": nx, "ny": ny, "nz": nz, "bc": "noslip", "spheres": 0, "diameter": 16.0,
         "poly": False, "rotation": False, "scalar": False, "rk": 1, "steps": 1, "batch": 0}
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the time-step control of a small run (chkdiv, chkdt): two reductions
        # whose results the host waits for
        _case("diag_64", "diag", "mixed", 64, 64, 64),
        # the single settling sphere in a triply periodic box, whole steps:
        # small kernels in a row
        _case("settle_64", "steps", "plain", 64, 64, 64, bc="periodic", spheres=1, steps=2),
        # a heated, rotating suspension on a ragged grid through the
        # per-subroutine entry points, one step: every option at once
        _case("scalar_96x108x75", "stages", "plain", 96, 108, 75, bc="freeslip", spheres=60, diameter=11.0,
              rotation=True, scalar=True),
        # the drop-in's momentum predictor on the channel
        _case("predict_plain_256", "predict", "plain", 256, 256, 256, rk=2),
        # the drop-in's projection at lengths with a factor of three
        _case("project_plain_384x192x128", "project", "plain", 384, 192, 128, rk=1),
        # the drop-in's multidirect forcing on the channel with 1000 spheres
        _case("forcing_plain_256", "forcing", "plain", 256, 256, 256, spheres=1000),
        # sphere integrals, collisions and the Newton-Euler update
        _case("particles_plain_256", "particles", "plain", 256, 256, 256, spheres=1000, rk=2),
        # the wide channel's fluid alone in the mixed form: predictor and projection
        _case("fluid_mixed_512x512x256", "project", "mixed", 512, 512, 256, rk=2),
        # the mixed form through the per-subroutine entry points
        _case("step_mixed_256", "stages", "mixed", 256, 256, 256, spheres=1000, steps=3),
        # a settling suspension of unequal spheres in the mixed form, whole steps
        _case("poly_mixed_384x384x192", "steps", "mixed", 384, 384, 192, spheres=1400, diameter=24.0, poly=True,
              steps=2),
        # the headline: mixed form with learned forcing, whole steps
        _case("step_learned_256", "steps", "learned", 256, 256, 256, spheres=1000, steps=4),
        # training of the forcing network on a harvested batch
        _case("train_8192", "train", "learned", 16, 16, 16, batch=8192, steps=100),
    ]


def _smooth(n):
    for q in (2, 3):
        while n % q == 0:
            n //= q
    return n == 1


_XS = [n for n in range(32, 513, 2) if _smooth(n // 2)]
_YS = [n for n in range(27, 513) if _smooth(n)]


def draw(rng):
    kind = rng.choice(["diag", "steps", "steps", "stages", "stages", "predict", "project", "project", "forcing",
                       "particles", "train"])
    if kind == "train":
        return _case(None, kind, "learned", 16, 16, 16, batch=int(math.exp(rng.uniform(math.log(512), math.log(8192)))),
                     steps=rng.randrange(20, 101))
    form = rng.choice(["plain", "mixed"] + (["learned"] if kind in ("steps", "stages") else []))
    most = {"plain": 2.0 ** 23, "mixed": 2.0 ** 24, "learned": 2.0 ** 24}[form] * (2 if kind in ("predict", "project") else 1)
    cells = math.exp(rng.uniform(math.log(2.0 ** 15), math.log(most)))
    side = cells ** (1.0 / 3.0)
    nx = min(_XS, key=lambda n: abs(math.log(n / (side * rng.uniform(0.8, 1.4)))))
    ny = min(_YS, key=lambda n: abs(math.log(n / (side * rng.uniform(0.8, 1.4)))))
    nz = max(32, min(384, int(cells / (nx * ny))))
    c = _case(None, kind, form, nx, ny, nz, rk=rng.choice([1, 2, 3]), bc=rng.choice(["noslip", "freeslip"]),
              steps=rng.choice([1, 2, 3]) if kind in ("steps", "stages") else 1)
    if kind == "forcing":
        c["rk"] = 1  # of the predictor before it
    if kind in ("forcing", "particles") or (kind in ("steps", "stages") and (form == "learned" or rng.random() < 0.8)):
        c["poly"] = kind != "forcing" and form != "learned" and rng.random() < 0.3
        top = min(min(nx, ny, nz) / 2.5, 24.0 if c["poly"] or form == "plain" else 16.0)
        c["diameter"] = round(rng.uniform(9.0, top), 2)
        room = _lattice(c)
        c["spheres"] = max(1, int(room[0] * room[1] * room[2] * rng.uniform(0.1, 0.8)))
        c["rotation"] = rng.random() < 0.5
    if kind == "stages" and rng.random() < 0.3:
        c["scalar"] = True
    if kind == "steps" and form == "plain" and rng.random() < 0.4:
        c.update(bc="periodic", spheres=1, poly=False)
    return c


# ---- inputs ---------------------------------------------------------------------
def _h(c):
    return 2.0 ** -math.ceil(math.log2(c["nz"]))


def _lattice(c):
    """Sites along x, y, z of a lattice that the spheres fit on without overlap."""
    d = c["diameter"] * 1.06
    return int(c["nx"] // d), int(c["ny"] // d), int((c["nz"] - 2.0) // d)


def _geometry(c, seed):
    """The library's Case: spheres at jittered sites of a lattice, seeded."""
    h = _h(c)
    lx, ly, lz = c["nx"] * h, c["ny"] * h, c["nz"] * h
    rng = np.random.default_rng(seed)
    n, d = c["spheres"], c["diameter"] * h
    settle = c["poly"] or c["bc"] == "periodic"
    rho = 2.0 if c["poly"] else (1.5 if settle else 1.0)
    visc = math.sqrt((rho - 1.0) * 9.81 * d ** 3) / 150.0 if settle else lz / 5600.0
    centres = radii = None
    if c["bc"] == "periodic":
        centres = 0.5 * np.array([[lx, ly, lz]]) + rng.uniform(-2 * h, 2 * h, (1, 3))
    elif n:
        m = _lattice(c)
        pitch = np.array([lx / m[0], ly / m[1], (lz - 2 * h) / m[2]])
        site = rng.permutation(m[0] * m[1] * m[2])[:n]
        ijk = np.stack([site % m[0], site // m[0] % m[1], site // (m[0] * m[1])], 1)
        jit = np.maximum(0.0, pitch - 1.02 * d) / 2
        centres = (ijk + 0.5) * pitch + rng.uniform(-1, 1, (n, 3)) * jit + np.array([0.0, 0.0, h])
    if c["poly"]:
        radii = 0.5 * d * rng.uniform(0.5, 1.0, n)
    return Case(name="perf", itot=c["nx"], jtot=c["ny"], ktot=c["nz"], lx=lx, ly=ly, lz=lz, visc=visc, radius=d / 2,
                ratiorho=rho, bc_top=BC[c["bc"]], bc_bot=BC[c["bc"]], np=n, seed=seed, rotation=int(c["rotation"]),
                flow="pur" if settle else "poi", centres=centres, radii=radii)


def _halo(f, sign_bot, sign_top, face):
    """Ghost values of one field: walls (sign 0: periodic copies), x and y periodic."""
    if sign_bot == 0:
        f[0], f[-1] = f[-2], f[1]
    elif face:
        f[0] = 0
        f[-2:] = 0
    else:
        f[0], f[-1] = sign_bot * f[1], sign_top * f[-2]
    f[:, 0], f[:, -1] = f[:, -2], f[:, 1]
    f[:, :, 0], f[:, :, -1] = f[:, :, -2], f[:, :, 1]
    return f


def _walls(c):
    return {"noslip": -1, "freeslip": 1, "periodic": 0}[c["bc"]]


def _fields(c, case, seed):
    """u, v, w, p, three stored right-hand sides and a scalar, each (k, j, i) with ghosts on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    shape = (c["nz"] + 2, c["ny"] + 2, c["nx"] + 2)
    s = _walls(c)
    amp = 0.01 if case.flow == "pur" else 0.05

    def noise(a):
        f = torch.empty(shape, dtype=torch.float32, device="cuda").uniform_(-a, a, generator=g)
        return f

    u, v, w = noise(amp), noise(amp), noise(amp)
    if case.flow == "poi":
        z = (torch.arange(shape[0], device="cuda", dtype=torch.float64) - 0.5) / c["nz"]
        v += (6.0 * z * (1.0 - z)).float()[:, None, None]
    p = noise(0.1 * amp)
    out = [_halo(u.double(), s, s, False), _halo(v.double(), s, s, False), _halo(w.double(), s, s, True),
           _halo(p.double(), abs(s), abs(s), False)]
    if c["kind"] in ("predict", "project"):
        out += [_halo(noise(1.0).double(), 0, 0, False) for _ in range(3)]
    else:
        out += [None] * 3
    out.append(_halo(noise(0.5).double(), 1, 1, False) if c["scalar"] else None)
    return out


def _dt(c, case):
    """Half the stability limit of chkdt for the largest velocities of the inputs."""
    h = _h(c)
    d1 = 1.65 / (4.0 * case.visc * 3.0 / h ** 2)
    d2 = math.sqrt(3.0) * h / (0.03 if case.flow == "pur" else 1.65)
    if case.flow == "pur":
        d2 = min(d2, h / math.sqrt((case.ratiorho - 1.0) * 9.81 * 2 * case.rmax))
    return 0.5 * min(d1, d2)


def _model(seed):
    """Weights of the forcing network (W1 b1 W2 b2 W3 b3) and its standardisation."""
    rng = np.random.default_rng(seed + 17)
    par = np.concatenate([rng.normal(0, math.sqrt(2 / 96), 128 * 96), np.zeros(128),
                          rng.normal(0, math.sqrt(2 / 128), 128 * 128), np.zeros(128),
                          rng.normal(0, 0.1 / math.sqrt(128), 3 * 128), np.zeros(3)]).astype(np.float32)
    norm = np.concatenate([np.zeros(96), np.full(96, 4.0), np.zeros(3), np.full(3, 0.01)]).astype(np.float32)
    return par, norm


_STREAM = None


def _stream():
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def _ptr(t):
    return None if t is None else ctypes.cast(t.data_ptr(), _abi.c_double_p)


def _set_fields(st):
    s = st["solver"]
    s._chk(s.fn["set_fields"](s.ctx, *[_ptr(f) for f in st["fields"][:7]]))


def _get(st, entry, names):
    """Fields by one of the library's getters into the program's own device arrays."""
    s = st["solver"]
    s._chk(s.fn[entry](s.ctx, *[_ptr(st["out"][n]) for n in names]))


def _velocities(ps, case, seed):
    rng = np.random.default_rng(seed + 29)
    z = ps.z / case.lz
    ps.u[:], ps.w[:] = rng.uniform(-0.02, 0.02, (2, case.np))
    ps.v[:] = rng.uniform(-0.02, 0.02, case.np) + (6.0 * z * (1.0 - z) if case.flow == "poi" else 0.0)
    if case.rotation:
        for f in (ps.omx, ps.omy, ps.omz):
            f[:] = rng.uniform(-0.5, 0.5, case.np)


def prepare(case, seed):
    c, st = case, {"case": case}
    if c["kind"] == "train":
        rng = np.random.default_rng(seed)
        st["solver"] = IBMSolver(Case(name="train", itot=16, jtot=16, ktot=16), mode=MODES["learned"])
        st["params"] = _model(seed)[0]
        st["x"] = rng.normal(0, 1, (c["batch"], 96)).astype(np.float32)
        st["t"] = (0.3 * st["x"][:, :3] + 0.2 * rng.normal(0, 1, (c["batch"], 3))).astype(np.float32)
        return st
    geo = _geometry(c, seed)
    solver = IBMSolver(geo, mode=MODES[c["form"]])
    solver.set_stream(_stream().cuda_stream)
    st.update(solver=solver, dt=_dt(c, geo), fields=_fields(c, geo, seed), particles=None)
    torch.cuda.synchronize()
    _set_fields(st)
    if geo.np:
        ps = geo.initial_particles(lagrangian=False)
        _velocities(ps, geo, seed)
        solver.set_particles(ps)
    solver.init_particles()
    if geo.np:
        ps = solver.get_particles(lagrangian=False)
        rng = np.random.default_rng(seed + 31)
        if c["kind"] == "particles":  # force sums of a forcing loop that has run
            scale = 0.05 * geo.visc * geo.radius
            for f in (ps.fxltot, ps.fyltot, ps.fzltot):
                f[:] = rng.uniform(-scale, scale, geo.np)
            for f in (ps.torqxltot, ps.torqyltot, ps.torqzltot):
                f[:] = rng.uniform(-scale, scale, geo.np) * geo.radius
            # the integrals before this substep: those of a slightly slower fluid
            for n in ("intu", "intv", "intw", "intomx", "intomy", "intomz"):
                getattr(ps, n)[:] *= 0.99
        st["particles"] = ps
    names = ("u", "v", "w") if c["kind"] in ("predict", "forcing") else ("u", "v", "w", "p")
    if c["kind"] not in ("diag", "particles"):
        st["out"] = {n: torch.empty_like(st["fields"][0]) for n in names + (("c", "dc") if c["scalar"] else ())}
    if c["form"] == "learned":
        # a model from an earlier training run; one step of calibration loops
        # (the first loop of each stage), a fixed residual reference after
        solver.set_forcing_model(*_model(seed))
        solver.learned_calibration(0)
        solver.learned_config(True, 1.5, 1.0e3)
        solver.rk3_step(st["dt"])
    torch.cuda.synchronize()
    return st


def _values(st, names):
    """The program's arrays, in single precision where the form's state is."""
    plain = st["case"]["form"] == "plain"
    with torch.cuda.stream(_stream()):
        return {n: st["out"][n].clone() if plain else st["out"][n].float() for n in names}


def _particle_values(ps):
    names = ["x", "y", "z", "u", "v", "w", "omx", "omy", "omz", "colfx", "colfy", "colfz", "intu", "intv", "intw"]
    names += ["intomx", "intomy", "intomz"]
    out = {n: getattr(ps, n) for n in names}
    out["qmax"], out["firstc"] = ps.qmax, ps.firstc
    return out


def run(state):
    st, c, s = state, state["case"], state["solver"]
    kind = c["kind"]
    if kind == "train":
        params, losses = s.mlp_fit(st["params"], st["x"], st["t"], c["steps"])
        return {"params": params, "losses": losses}
    dt = st["dt"]
    if kind == "diag":
        # the total divergence is the rounding of a sum that telescopes to zero: not returned
        _, largest, where = s.chkdiv()
        return {"divmax": largest, "where": list(where), "dtmax": s.chkdt()}
    if kind == "predict":
        s.rk(c["rk"], dt)
        _get(st, "get_intermediate", ("u", "v", "w"))
        return _values(st, ("u", "v", "w"))
    if kind == "forcing":
        s.rk(1, dt)
        s.forcing_loop(dt, 3)
        _get(st, "get_intermediate", ("u", "v", "w"))
        return _values(st, ("u", "v", "w"))
    if kind == "particles":
        s.set_particles(st["particles"])
        s.intgr_nwtn_eulr(c["rk"], dt)
        return _particle_values(s.get_particles(lagrangian=False))
    # whole substeps: from the program's own state and back
    _set_fields(st)
    if c["scalar"]:
        sp = _abi.IbmScalarParams(PRAN, BETA, 0.5, -0.5, _abi.IBM_BC_C_DIRICHLET, _abi.IBM_BC_C_NEUMANN)
        s._chk(s.fn["set_scalar"](s.ctx, ctypes.byref(sp), _ptr(st["fields"][7]), None))
    if st["particles"] is not None:
        s.set_particles(st["particles"])
    if kind == "project":
        s.rk(c["rk"], dt)
        s.project(c["rk"], dt)
    elif kind == "stages":
        for _ in range(c["steps"]):
            for r in (1, 2, 3):
                s.rk(r, dt)
                s.forcing_loop(dt, 3)
                s.project(r, dt)
                s.intgr_nwtn_eulr(r, dt)
    else:
        s.run(dt, c["steps"])
    names = ("u", "v", "w", "p")
    s._chk(s.fn["get_fields"](s.ctx, *[_ptr(st["out"][n]) for n in names], None, None, None))
    if c["scalar"]:
        _get(st, "get_scalar", ("c", "dc"))
        names += ("c", "dc")
    out = {"fields": _values(st, names)}
    if st["particles"] is not None:
        out["particles"] = _particle_values(s.get_particles(lagrangian=False))
        if c["form"] != "plain":  # single-precision fields act on them
            for n, a in out["particles"].items():
                if a.dtype == np.float64:
                    out["particles"][n] = a.astype(np.float32)
    return out


# ---- what a pass cannot do without ------------------------------------------------
def work(case):
    c, kind = case, case["kind"]
    if kind == "train":
        par, nb, n = 29315, c["batch"], c["steps"]
        return {"bytes": 4.0 * nb * 99 + n * 4.0 * par * 6, "flops": 6.0 * 29184 * nb * n}
    n = float(c["nx"]) * c["ny"] * c["nz"]
    word = 8 if c["form"] == "plain" else 4
    if kind == "diag":
        return {"bytes": 3 * n * word, "flops": 40 * n}
    d = c["diameter"] * (0.75 if c["poly"] else 1.0)
    points = c["spheres"] * math.pi * (d - 0.6) ** 2
    shell = c["spheres"] * 9.0 * (d - 0.6) ** 2  # cells under the points' stencils
    ball = c["spheres"] * math.pi / 6 * (d + 2) ** 3
    predict = (7 + 3) * n if c["rk"] == 1 else (10 + (6 if c["rk"] == 2 else 3)) * n
    project = 8 * n
    if kind == "predict":
        words, flops = predict, 100 * n
    elif kind == "project":
        words, flops = 8 * n, (100 + 12 * math.log2(n)) * n
    elif kind == "forcing":
        words, flops = 6 * n + 6 * shell, 100 * n + points * 3 * 500
    elif kind == "particles":
        words, flops = 3 * ball, 60 * ball
    else:
        sub = predict + project + 6 * shell + 3 * ball + (4 * n if c["scalar"] else 0)
        words, flops = 3 * c["steps"] * sub, 3 * c["steps"] * ((130 + 12 * math.log2(n)) * n + points * 1500)
        if c["form"] == "learned":
            flops += 3 * c["steps"] * points * 2 * 29184
    return {"bytes": words * float(word), "flops": float(flops)}


# ---- 64-bit restatements ------------------------------------------------------------
def _roll(f, di=0, dj=0, dk=0):
    """f(i+di, j+dj, k+dk) at the interior cells; x and y periodic, z ghosts stored."""
    n = f.shape[0]
    core = f[1 + dk:n - 1 + dk, 1:-1, 1:-1]
    return torch.roll(core, (-dj, -di), (1, 2)) if di or dj else core


def _momentum(u, v, w, p, h, visc):
    """Right-hand sides of the three momentum equations and the pressure gradients."""
    a = 1.0 / h
    U, V, W = u, v, w
    r = _roll

    def lap(f):
        return visc * a * a * (r(f, 1) + r(f, -1) + r(f, 0, 1) + r(f, 0, -1) + r(f, 0, 0, 1) + r(f, 0, 0, -1) - 6 * r(f))

    def flux(x, y):
        return 0.25 * a * x * y

    u0, v0, w0 = r(U), r(V), r(W)
    ru = (flux(r(U, -1) + u0, r(U, -1) + u0) - flux(r(U, 1) + u0, r(U, 1) + u0) +
          flux(r(U, 0, -1) + u0, r(V, 1, -1) + r(V, 0, -1)) - flux(r(U, 0, 1) + u0, r(V, 1) + v0) +
          flux(r(U, 0, 0, -1) + u0, r(W, 1, 0, -1) + r(W, 0, 0, -1)) - flux(r(U, 0, 0, 1) + u0, r(W, 1) + w0) + lap(U))
    rv = (flux(r(U, -1) + r(U, -1, 1), v0 + r(V, -1)) - flux(u0 + r(U, 0, 1), v0 + r(V, 1)) +
          flux(v0 + r(V, 0, -1), v0 + r(V, 0, -1)) - flux(v0 + r(V, 0, 1), v0 + r(V, 0, 1)) +
          flux(r(W, 0, 0, -1) + r(W, 0, 1, -1), r(V, 0, 0, -1) + v0) - flux(w0 + r(W, 0, 1), r(V, 0, 0, 1) + v0) + lap(V))
    rw = (flux(w0 + r(W, -1), r(U, -1) + r(U, -1, 0, 1)) - flux(w0 + r(W, 1), u0 + r(U, 0, 0, 1)) +
          flux(w0 + r(W, 0, -1), r(V, 0, -1) + r(V, 0, -1, 1)) - flux(w0 + r(W, 0, 1), v0 + r(V, 0, 0, 1)) +
          flux(w0 + r(W, 0, 0, -1), w0 + r(W, 0, 0, -1)) - flux(w0 + r(W, 0, 0, 1), w0 + r(W, 0, 0, 1)) + lap(W))
    gp = [-a * (r(p, 1) - r(p)), -a * (r(p, 0, 1) - r(p)), -a * (r(p, 0, 0, 1) - r(p))]
    return [ru, rv, rw], gp


def _predicted(c, f, h, visc, dt):
    """Interior of dudt, dvdt, dwdt after stage rk."""
    rhs, gp = _momentum(f[0], f[1], f[2], f[3], h, visc)
    f1, f2, f3 = (q * dt / 60.0 for q in RK[c["rk"]])
    out = []
    for q in range(3):
        x = _roll(f[q]) + f1 * gp[q]
        if c["rk"] == 1:
            x = x + f1 * rhs[q]
        else:
            x = x + f2 * rhs[q] - f3 * _roll(f[4 + q])
        out.append(x)
    return out


def _framed(x):
    """An interior array in the reference layout: x and y ghosts periodic, z ghosts zero."""
    f = torch.zeros((x.shape[0] + 2, x.shape[1] + 2, x.shape[2] + 2), dtype=x.dtype, device=x.device)
    f[1:-1, 1:-1, 1:-1] = x
    f[:, 0], f[:, -1] = f[:, -2].clone(), f[:, 1].clone()
    f[:, :, 0], f[:, :, -1] = f[:, :, -2].clone(), f[:, :, 1].clone()
    return f


def _projected(c, du, f, h, dt):
    """u, v, w, p in the reference layout after the projection of du."""
    a, s = 1.0 / h, _walls(c)
    step = RKAB[c["rk"]] * dt
    U, V, W = du
    W = W.clone()
    W[-1] = 0
    below = torch.cat([torch.zeros_like(W[:1]), W[:-1]])
    div = a / step * ((W - below) + (V - torch.roll(V, 1, 1)) + (U - torch.roll(U, 1, 2)))
    spec = torch.fft.rfft2(div)
    n, ny, nx = div.shape
    kx = torch.arange(spec.shape[2], device=div.device, dtype=torch.float64)
    ky = torch.arange(ny, device=div.device, dtype=torch.float64)
    lam = (-4 * a * a * torch.sin(math.pi * ky / ny) ** 2)[:, None] + (-4 * a * a * torch.sin(math.pi * kx / nx) ** 2)[None]
    a2 = a * a
    cp = torch.empty((n,) + lam.shape, dtype=torch.float64, device=div.device)
    x = torch.empty_like(spec)
    for k in range(n):
        b = lam - (2 if 0 < k < n - 1 else 1) * a2
        den = b if k == 0 else b - a2 * cp[k - 1]
        inv = torch.where(den == 0, torch.zeros_like(den), 1.0 / den)
        cp[k] = a2 * inv
        x[k] = (spec[k] if k == 0 else spec[k] - a2 * x[k - 1]) * inv
    for k in range(n - 2, -1, -1):
        x[k] -= cp[k] * x[k + 1]
    phi = torch.fft.irfft2(x, s=(ny, nx))
    up = torch.cat([phi[1:], phi[-1:]])
    u = U - step * a * (torch.roll(phi, -1, 2) - phi)
    v = V - step * a * (torch.roll(phi, -1, 1) - phi)
    w = W - step * a * (up - phi)
    return {"u": _halo(_framed(u), s, s, False), "v": _halo(_framed(v), s, s, False),
            "w": _halo(_framed(w), s, s, True), "p": _halo(_framed(phi + _roll(f[3])), 1, 1, False)}


def _delta(r):
    r = r.abs()
    inner = (1 + torch.sqrt((1 - 3 * r * r).clamp(min=0))) / 3
    outer = (5 - 3 * r - torch.sqrt((1 - 3 * (1 - r) ** 2).clamp(min=0))) / 6
    return torch.where(r > 1.5, torch.zeros_like(r), torch.where(r > 0.5, outer, inner))


def _forced(c, du, geo, seed, dt):
    """dudt, dvdt, dwdt (with ghosts) after three passes of the multidirect forcing."""
    h, dev = _h(c), du[0].device
    n = geo.np
    ps = geo.initial_particles(lagrangian=False)
    _velocities(ps, geo, seed)
    theta, phi = fibonacci_sphere(derived_nl(geo.radius, geo.dxi))
    shell = geo.radius - 0.3 * h
    arm = shell * np.stack([np.sin(theta) * np.cos(phi), np.sin(theta) * np.sin(phi), np.cos(theta)], 1)
    x = torch.as_tensor(np.stack([ps.x, ps.y, ps.z], 1)[:, None] + arm[None], device=dev).reshape(-1, 3)
    om = np.stack([ps.omx, ps.omy, ps.omz], 1)
    vel = np.stack([ps.u, ps.v, ps.w], 1)[:, None] + np.cross(om[:, None], arm[None])
    vel = torch.as_tensor(vel, device=dev).reshape(-1, 3)
    dvol = 4.0 / 3.0 * math.pi * ((shell + 0.5 * h) ** 3 - (shell - 0.5 * h) ** 3) / len(theta)
    scale = dvol / h ** 3 * dt
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    g = x / h
    near = torch.floor(g + 0.5)  # nearest face
    low = torch.floor(g)
    three = torch.arange(3, device=dev, dtype=torch.float64)
    base_f = near - 1
    base_f[:, 2].clamp_(min=1)
    base_c = low.clone()
    base_c[:, 2].clamp_(min=1, max=nz - 2)
    wf = _delta(base_f[..., None] + three - g[..., None])
    wc = _delta(base_c[..., None] + three - 0.5 - g[..., None])
    size = (nx, ny)
    index, weight = [], []
    for q in range(3):
        ax, wt = [], []
        for d in range(3):
            b = (base_f if d == q else base_c)[:, d, None] + three
            wt.append((wf if d == q else wc)[:, d])
            b = b.long()
            ax.append(b if d == 2 else torch.remainder(b - 1, size[d]))
        index.append((ax[2][:, :, None, None] * ny + ax[1][:, None, :, None]) * nx + ax[0][:, None, None, :])
        weight.append(wt[2][:, :, None, None] * wt[1][:, None, :, None] * wt[0][:, None, None, :])
    full = []
    for f in du:
        z = torch.zeros((nz + 2, ny, nx), dtype=torch.float64, device=dev)
        z[1:-1] = f
        full.append(z.reshape(-1))
    for _ in range(3):
        for q in range(3):
            slip = vel[:, q] - (full[q][index[q]] * weight[q]).sum((1, 2, 3))
            spread = slip[:, None, None, None] * (scale / dt) * weight[q]
            full[q].index_put_((index[q].reshape(-1),), spread.reshape(-1), accumulate=True)
    out = {}
    for name, f in zip("uvw", full):
        f = f.reshape(nz + 2, ny, nx)
        e = _framed(f[1:-1])
        e[0, 1:-1, 1:-1], e[-1, 1:-1, 1:-1] = f[0], f[-1]
        for k in (0, -1):
            e[k, 0], e[k, -1] = e[k, -2].clone(), e[k, 1].clone()
            e[k, :, 0], e[k, :, -1] = e[k, :, -2].clone(), e[k, :, 1].clone()
        out[name] = e
    return out


def _sphere_integrals(c, f, geo):
    """Volume integrals of u and of r x u over the spheres, cut cells by corner distances."""
    h, dev = _h(c), f[0].device
    ctr = torch.as_tensor(geo.sphere_centres(), device=dev)
    rad = torch.as_tensor(geo.radii if geo.radii is not None else np.full(geo.np, geo.radius), device=dev)
    m = int(2 * geo.rmax / h + 6)
    span = torch.arange(m, device=dev)
    lo = torch.floor((ctr - geo.rmax) / h).long() - 1  # first cell (1-based) of each box
    idx = lo[:, :, None] + span
    n = (c["nx"], c["ny"], c["nz"])
    lin, mom = [], [torch.zeros(geo.np, dtype=torch.float64, device=dev) for _ in range(3)]
    arm = [(idx[:, d] - 0.5) * h - ctr[:, d, None] for d in range(3)]
    for q in range(3):
        sq = []
        for d in range(3):
            left = (idx[:, d] - (0.5 if d == q else 1.0)) * h - ctr[:, d, None]
            sq.append((left ** 2, (left + h) ** 2))
        top = torch.zeros((geo.np, m, m, m), dtype=torch.float64, device=dev)
        bot = torch.zeros_like(top)
        for z in sq[2]:
            for y in sq[1]:
                for x in sq[0]:
                    s = rad[:, None, None, None] - torch.sqrt(z[:, :, None, None] + y[:, None, :, None] + x[:, None, None, :])
                    top += s.clamp(min=0)
                    bot += s.abs()
        ok = ((idx[:, 2] >= 1) & (idx[:, 2] <= n[2]))[:, :, None, None]
        k = idx[:, 2].clamp(1, n[2])
        vals = f[q][k[:, :, None, None], (torch.remainder(idx[:, 1] - 1, n[1]) + 1)[:, None, :, None],
                    (torch.remainder(idx[:, 0] - 1, n[0]) + 1)[:, None, None, :]]
        fw = torch.where(ok, vals * top / bot, torch.zeros_like(top)) * h ** 3
        lin.append(fw.sum((1, 2, 3)))
        rx = (fw * arm[0][:, None, None, :]).sum((1, 2, 3))
        ry = (fw * arm[1][:, None, :, None]).sum((1, 2, 3))
        rz = (fw * arm[2][:, :, None, None]).sum((1, 2, 3))
        if q == 0:
            mom[1] += rz
            mom[2] -= ry
        elif q == 1:
            mom[0] -= rz
            mom[2] += rx
        else:
            mom[0] += ry
            mom[1] -= rx
    return lin, mom


def _trained(c, seed):
    """Full-batch Adam steps of the network from the same weights."""
    rng = np.random.default_rng(seed)
    x = rng.normal(0, 1, (c["batch"], 96)).astype(np.float32)
    t = (0.3 * x[:, :3] + 0.2 * rng.normal(0, 1, (c["batch"], 3))).astype(np.float32)
    x, t = torch.as_tensor(x, device="cuda").double(), torch.as_tensor(t, device="cuda").double()
    p = torch.as_tensor(_model(seed)[0], device="cuda").double()
    m, v, losses = torch.zeros_like(p), torch.zeros_like(p), []
    for step in range(1, c["steps"] + 1):
        q = p.clone().requires_grad_(True)
        w1, b1, w2, b2, w3, b3 = (a.reshape(s) for a, s in zip(
            torch.split(q, [128 * 96, 128, 128 * 128, 128, 384, 3]), [(128, 96), (128,), (128, 128), (128,), (3, 128), (3,)]))
        hid = torch.nn.functional.gelu(x @ w1.T + b1, approximate="tanh")
        hid = torch.nn.functional.gelu(hid @ w2.T + b2, approximate="tanh")
        loss = ((hid @ w3.T + b3 - t) ** 2).sum() / c["batch"]
        (g,) = torch.autograd.grad(loss, q)
        losses.append(loss.detach())
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        p = p - 1e-3 * (m / (1 - 0.9 ** step)) / (torch.sqrt(v / (1 - 0.999 ** step)) + 1e-8)
    return {"params": p, "losses": torch.stack(losses)}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "train":
        return _trained(c, seed) if c["batch"] * c["steps"] <= 1 << 20 else None
    if kind in ("steps", "stages"):
        return None  # many substeps with collisions
    geo = _geometry(c, seed)
    h, dt = _h(c), _dt(c, geo)
    f = _fields(c, geo, seed)
    if kind == "diag":
        u, v, w = (q for q in f[:3])
        r, a = _roll, 1.0 / h
        div = a * ((r(w) - r(w, 0, 0, -1)) + (r(v) - r(v, 0, -1)) + (r(u) - r(u, -1)))
        big = [1.65 / (4.0 * geo.visc * 3 * a * a)]
        for terms in (
            (r(u), 0.25 * (r(v) + r(v, 0, -1) + r(v, 1) + r(v, 1, -1)), 0.25 * (r(w) + r(w, 0, 0, -1) + r(w, 1) + r(w, 1, 0, -1))),
            (0.25 * (r(u) + r(u, 0, 1) + r(u, -1, 1) + r(u, -1)), r(v), 0.25 * (r(w) + r(w, 0, 1) + r(w, 0, 1, -1) + r(w, 0, 0, -1))),
            (0.25 * (r(u) + r(u, -1) + r(u, -1, 0, 1) + r(u, 0, 0, 1)), 0.25 * (r(v) + r(v, 0, -1) + r(v, 0, -1, 1) + r(v, 0, 0, 1)), r(w)),
        ):
            big.append(math.sqrt(3.0) / (a * sum(t.abs() for t in terms)).max().item())
        return {"divmax": div.abs().max().item(), "where": None, "dtmax": min(big)}
    if kind == "particles":
        lin, mom = _sphere_integrals(c, f, geo)
        names = ["x", "y", "z", "u", "v", "w", "omx", "omy", "omz", "colfx", "colfy", "colfz", "qmax", "firstc"]
        out = dict.fromkeys(names)
        out.update(zip(("intu", "intv", "intw"), lin))
        out.update(zip(("intomx", "intomy", "intomz"), mom))
        return out
    du = _predicted(c, f, h, geo.visc, dt)
    if kind == "predict":
        return {n: _framed(x) for n, x in zip("uvw", du)}
    if kind == "project":
        return {"fields": _projected(c, du, f, h, dt)}
    return _forced(c, du, geo, seed, dt)
