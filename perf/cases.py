"""What this framework's users run, as cases that can be timed and compared.

Every case goes through the public entry points (ps3d_b200.model.Model,
ps3d_b200.ensemble.Ensemble and the C ABI of include/ps3d_gpu.h) and returns
the fields a program reads back.  A case is a dict of plain values; its kind
says which part of a program's life it is:

  steps     the main loop between two snapshots: `steps` time steps of the
            resident state, then u, v, w, b and p into page-locked host arrays
  dropin    the Fortran host's loop: parameters set and `integrate` called for
            every single step with the caller's time levels, then the download
  ensemble  `members` eddies of the ensemble's four sizes advanced together,
            then every member read back
  balance   one optimal-balance request: ramped backward and forward runs and
            normal-mode projections, then the balanced fields
  project   the zero-order normal-mode balance of the state and its fields
  pressure  the pressure projection of a caller's own device arrays

Sizes are those of the package's configurations, tests and benchmark and the
ranges between them; all of a grid's lengths factor into 2, 3 and 5 where the
transforms need it, nz is free under a rigid lid.
"""
import ctypes as C
import math
from types import SimpleNamespace

import numpy as np
import torch

from ps3d_b200 import abi
from ps3d_b200 import configs as cf
from ps3d_b200.ensemble import Ensemble
from ps3d_b200.model import Model, PS3DError, load

FIELDS = ("u", "v", "w", "b")
ENSEMBLE_SIZES = ((32, 32, 16), (64, 64, 32), (128, 64, 32), (128, 128, 64))
F64 = torch.float64
DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _steps(name, flow, nx, ny, nz, steps, precision="fp64", friction="harmonic"):
    return {"name": name, "kind": "steps", "flow": flow, "nx": nx, "ny": ny, "nz": nz, "steps": steps,
            "precision": precision, "friction": friction}


def listed():
    return [
        # the smallest call: a host code projects its own device arrays, on a grid that is no power of two
        {"name": "pressure_48x40x24", "kind": "pressure", "nx": 48, "ny": 40, "nz": 24, "rigid": True},
        # a Fortran host's loop on a small test grid, one call per step
        {"name": "dropin_32x32x16", "kind": "dropin", "nx": 32, "ny": 32, "nz": 16, "steps": 24},
        # the plain method's own configuration: a Gaussian eddy, 200 steps
        _steps("eddy_fp64_64x64x32", "eddy", 64, 64, 32, 200),
        # a grid nobody tuned for: lengths with factors 3 and 5, nz no multiple of 16
        _steps("eddy_fp64_96x80x50", "eddy", 96, 80, 50, 120),
        # scale-selective (biharmonic) friction, as many ocean set-ups use it
        _steps("eddy_biharmonic_128x128x64", "eddy", 128, 128, 64, 40, friction="biharmonic"),
        # a medium production grid in mixed precision
        _steps("eddy_mixed_128x128x64", "eddy", 128, 128, 64, 150, precision="mixed"),
        # the benchmark: the jet instability, in both precisions
        _steps("jets_fp64_256x256x128", "jets", 256, 256, 128, 60),
        _steps("jets_mixed_256x256x128", "jets", 256, 256, 128, 60, precision="mixed"),
        # the largest grid: triply periodic lee waves with wavemaker and background flow
        _steps("lee_fp64_512x256x128", "lee", 512, 256, 128, 30, friction="none"),
        # an ensemble of uneven sizes
        {"name": "ensemble_fp64_32", "kind": "ensemble", "members": 32, "steps": 60},
        # an optimal-balance request of the serving mix: 100-step ramps
        {"name": "balance_fp64_64x64x32", "kind": "balance", "nx": 64, "ny": 64, "nz": 32, "ramp": 100, "iterations": 3},
        # the normal-mode projection at the largest serving size
        {"name": "project_fp64_256x256x64", "kind": "project", "nx": 256, "ny": 256, "nz": 64},
    ]


def _smooth(lo, hi):
    """Even lengths in [lo, hi] whose halves factor into 2, 3 and 5."""
    out = []
    for n in range(lo + lo % 2, hi + 1, 2):
        m = n // 2
        for r in (2, 3, 5):
            while m % r == 0:
                m //= r
        if m == 1:
            out.append(n)
    return out


def _near(rng, lo, hi):
    """A smooth even length, spread over the logarithm of [lo, hi]."""
    t = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(_smooth(lo, hi), key=lambda n: abs(n - t))


def _nlog(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("steps", "steps", "steps", "mixed", "mixed", "dropin", "ensemble", "balance", "project", "pressure"))
    if kind == "steps":
        nx, ny, nz = _near(rng, 32, 320), _near(rng, 32, 320), _nlog(rng, 16, 144)
        flow = rng.choice(("eddy", "eddy", "jets", "lee"))
        friction = "none" if flow == "lee" else rng.choice(("harmonic", "harmonic", "biharmonic"))
        if flow == "lee":
            nz = min(_smooth(16, 144), key=lambda n: abs(n - nz))
        return {"kind": "steps", "flow": flow, "nx": nx, "ny": ny, "nz": nz, "precision": "fp64", "friction": friction,
                "steps": max(12, min(200, int((2e8 if friction == "biharmonic" else 4e8) / (nx * ny * nz)) + rng.randrange(5)))}
    if kind == "mixed":
        nx, ny, nz = rng.choice((128, 256, 512)), rng.choice((128, 256)), rng.randrange(64, 161)
        flow = rng.choice(("eddy", "jets", "lee"))
        if flow == "lee":
            nz = min(_smooth(64, 144), key=lambda n: abs(n - nz))
        return {"kind": "steps", "flow": flow, "nx": nx, "ny": ny, "nz": nz, "precision": "mixed",
                "friction": "none" if flow == "lee" else "harmonic",
                "steps": max(12, min(150, int(4e8 / (nx * ny * nz)) + rng.randrange(5)))}
    if kind == "dropin":
        return {"kind": "dropin", "nx": _near(rng, 16, 128), "ny": _near(rng, 16, 128), "nz": _nlog(rng, 8, 48),
                "steps": rng.randrange(12, 40)}
    if kind == "ensemble":
        return {"kind": "ensemble", "members": rng.randrange(8, 41), "steps": rng.randrange(12, 70)}
    if kind == "balance":
        nx = _near(rng, 48, 128)
        return {"kind": "balance", "nx": nx, "ny": _near(rng, 48, 128), "nz": rng.randrange(16, 65), "ramp": rng.randrange(40, 110),
                "iterations": rng.randrange(2, 4)}
    if kind == "project":
        return {"kind": "project", "nx": _near(rng, 64, 256), "ny": _near(rng, 64, 256), "nz": rng.randrange(16, 97)}
    nx, ny, nz = _near(rng, 16, 128), _near(rng, 16, 128), _nlog(rng, 8, 96)
    rigid = rng.random() < 0.7
    if not rigid:
        nz = min(_smooth(8, 96), key=lambda n: abs(n - nz))
    return {"kind": "pressure", "nx": nx, "ny": ny, "nz": nz, "rigid": rigid}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _precision(case):
    return abi.PS3D_MIXED if case.get("precision") == "mixed" else abi.PS3D_FP64


def _params(case):
    n = (case["nx"], case["ny"], case["nz"])
    flow = case.get("flow", "eddy")
    if flow == "jets":
        p = cf.jets_params(*n, precision=_precision(case))
        p.dt = min(p.dt, 0.15 * p.dx / 0.5)
    elif flow == "lee":
        p = cf.lee_wave_params(*n, precision=_precision(case))
    else:
        p = cf.eddy_params(*n, precision=_precision(case), rigid=case.get("rigid", True))
    if case.get("friction") == "biharmonic":
        p.Ah = p.Av = 0.0
        d = min(p.dx, p.dy)
        p.Ahbi = p.Khbi = 0.1 * d ** 4 / (64.0 * p.dt)
        p.Avbi = p.Kvbi = 0.1 * p.dz ** 4 / (16.0 * p.dt)
    return p


def _rand(shape, gen):
    return torch.rand(shape, generator=gen, dtype=F64, device=gen.device) * 2.0 - 1.0


def _axis(n, device, shift=0.0):
    return torch.arange(1, n + 1, dtype=F64, device=device) - shift


def _fields(p, flow, seed):
    """Seeded initial state, interior (nz, ny, nx) on the GPU: the package's eddy, or its jets with an eddy of a fifth of
    their speed between them (a jet that has begun to meander), and white noise in u, v and b."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    dev = gen.device
    shape = (p.nz, p.ny, p.nx)
    if flow == "lee":
        return {n: torch.zeros(shape, dtype=F64, device=dev) for n in FIELDS}
    f = {"u": 0.0, "b": 0.0}
    if flow == "jets":
        y = (_axis(p.ny, dev, 1.0)) * p.dy
        z = (_axis(p.nz, dev, 1.0)) * p.dz
        W = p.Ly / 16.0
        prof = torch.exp(-((y - 0.75 * p.Ly) / W) ** 2) - torch.exp(-((y - 0.25 * p.Ly) / W) ** 2)
        prof = prof * (0.5 * (1.0 + 0.1 * float(_rand((1,), gen))))
        u = prof[None, :] * torch.cos(z / p.Lz * math.pi)[:, None]
        dudz = torch.empty_like(u)
        dudz[1:-1] = (u[2:] - u[:-2]) / (2 * p.dz)
        dudz[0] = (u[1] - u[0]) / p.dz
        dudz[-1] = (u[-1] - u[-2]) / p.dz
        b = torch.cumsum(-p.dy * p.f0 * dudz, 1)
        f = {"u": u[:, :, None], "b": b[:, :, None]}
    amp = 0.05 + 0.075 * (1.0 + float(_rand((1,), gen)))
    R = p.Lx / 8.0
    z = _axis(p.nz, dev, 0.5) * p.dz
    cz, sz = torch.cos(math.pi * z / p.Lz)[:, None, None], torch.sin(math.pi * z / p.Lz)[:, None, None]

    def gauss(sx, sy):
        X = (_axis(p.nx, dev, sx) * p.dx - 0.5 * p.Lx)[None, :]
        Y = (_axis(p.ny, dev, sy) * p.dy - 0.5 * p.Ly)[:, None]
        return X, Y, torch.exp(-(X ** 2 + Y ** 2) / R ** 2)

    X, Y, e = gauss(0.0, 0.5)
    u = (2.0 * Y / R ** 2 * e)[None] * cz
    X, Y, e = gauss(0.5, 0.0)
    v = (-2.0 * X / R ** 2 * e)[None] * cz
    X, Y, e = gauss(0.5, 0.5)
    s = amp / float(u.abs().max())
    f = {"u": f["u"] + u * s, "v": v * s, "b": f["b"] + (-p.f0 * math.pi / p.Lz * s) * e[None] * sz}
    f["w"] = torch.zeros(shape, dtype=F64, device=dev)
    f["b"] = f["b"] + 1e-3 * float(f["b"].abs().max()) * _rand(shape, gen)
    for n in ("u", "v"):
        f[n] = f[n] + 1e-3 * float(f["u"].abs().max()) * _rand(shape, gen)
    return f


def _forcing(p, seed):
    """Background flow and a bottom-localised wavemaker in w with seeded phases."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed + 1000003)
    dev = gen.device
    x, y, z = _axis(p.nx, dev, 0.5) * p.dx, _axis(p.ny, dev, 0.5) * p.dy, _axis(p.nz, dev) * p.dz
    r = torch.rand(24, generator=gen, dtype=F64, device=dev).tolist()
    hr = torch.zeros((p.ny, p.nx), dtype=F64, device=dev)
    hi = hr.clone()
    for m in range(8):
        arg = 2 * math.pi * ((1 + int(4 * r[3 * m])) * x[None, :] / p.Lx + (1 + int(3 * r[3 * m + 1])) * y[:, None] / p.Ly)
        hr += torch.cos(arg + 2 * math.pi * r[3 * m + 2])
        hi += torch.sin(arg + 2 * math.pi * r[3 * m + 2])
    gz = 1e-7 * torch.exp(-((z - p.Lz / 8.0) / (p.Lz / 20.0)) ** 2)[:, None, None]
    return {"omega": 0.5 * p.N0, "w_r": gz * hr, "w_i": gz * hi,
            "u_back": torch.full((p.nz, p.ny, p.nx), 0.1, dtype=F64, device=dev)}


def _halo(f, ghost_levels=False):
    """The reference's halo layout: two periodic points on every side (z levels repeated for p under a rigid lid)."""
    for ax, n in enumerate(f.shape):
        i = torch.arange(-2, n + 2, device=f.device)
        f = f.index_select(ax, i.clamp(0, n - 1) if ghost_levels and ax == 0 else i % n)
    return f


def _pinned(shape):
    return torch.empty(shape, dtype=F64, pin_memory=True).numpy()


def _host(f):
    h = _halo(f)
    out = torch.empty(h.shape, dtype=F64, pin_memory=True)
    out.copy_(h)
    return out.numpy()


def _check(rc, what):
    if rc != 0:
        raise PS3DError(rc, what)


def _members(case, seed):
    """The members' parameters: the four sizes in a fixed seeded order, so that one case is always one amount of work."""
    order = np.random.default_rng(case["members"]).integers(0, len(ENSEMBLE_SIZES), case["members"])
    return [cf.eddy_params(*ENSEMBLE_SIZES[int(k)]) for k in order]


def _pressure_inputs(case, p, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    f = {n: 0.1 * _rand((p.nz, p.ny, p.nx), gen) for n in ("u", "v", "w")}
    if case["rigid"]:
        f["w"][-1] = 0.0
    return f


def prepare(case, seed):
    s = SimpleNamespace(case=case)
    if case["kind"] == "ensemble":
        s.params = _members(case, seed)
        s.handle = Ensemble(s.params)
        s.out = []
        for m, p in enumerate(s.params):
            f = _fields(p, "eddy", seed * 1009 + m)
            s.handle.upload(m, *[_host(f[n]) for n in FIELDS])
            s.out.append(m)
        # one block of page-locked memory for the members of each size
        shapes = sorted(set(abi.halo_shape(p) for p in s.params))
        s.blocks = [_pinned((sum(abi.halo_shape(p) == sh for p in s.params), 5) + sh) for sh in shapes]
        at = {sh: 0 for sh in shapes}
        for m, p in enumerate(s.params):
            sh = abi.halo_shape(p)
            s.out[m] = s.blocks[shapes.index(sh)][at[sh]]
            at[sh] += 1
        return s
    p = s.params = _params(case)
    if case["kind"] == "pressure":
        s.inputs = _pressure_inputs(case, p, seed)
        s.solve = load().ps3d_pressure_solve_noalloc
        s.solve.argtypes = [C.POINTER(abi.Params)] + [C.c_void_p] * 5
        return s
    f = _fields(p, case.get("flow", "eddy"), seed)
    s.model = Model(p)
    s.model.upload(**{n: _host(f[n]) for n in FIELDS})
    if case.get("flow") == "lee":
        g = _forcing(p, seed)
        s.model.set_forcing(abi.PS3D_FORCE_WAVEMAKER | abi.PS3D_FORCE_BACKGROUND, omega=g["omega"],
                            **{n: _host(g[n]) for n in ("w_r", "w_i", "u_back")})
    s.out = {n: _pinned(abi.halo_shape(p)) for n in FIELDS + ("p",)}
    s.levels = [0, 3, 2, 1]   # itt, tau, taum1, taum2 of a host that keeps them itself
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    case, p = s.case, s.params
    kind = case["kind"]
    if kind == "steps":
        s.model.run(case["steps"])
        return s.model.download_into(s.out)
    if kind == "dropin":
        m = s.model
        itt, tau, t1, t2 = s.levels
        for _ in range(case["steps"]):
            m.set_step_params(p.dt, p.Ro)
            m.integrate(itt, tau, t1, t2)
            tau, t1, t2 = tau % 3 + 1, t1 % 3 + 1, t2 % 3 + 1
            itt += 1
        s.levels = [itt, tau, t1, t2]
        return m.download_into(s.out)
    if kind == "ensemble":
        e = s.handle
        e.integrate(case["steps"])
        for m, block in enumerate(s.out):
            _check(e.L.ps3d_ensemble_download(e.h, m, *[abi.dptr(block[q]) for q in range(5)]), "ps3d_ensemble_download")
        return s.blocks
    if kind == "balance":
        s.model.diag_opt_balance(_balance_options(case, p))   # its norm, a difference of nearly equal fields, is not kept
        return _get_fields(s, abi.PS3D_FIELDS_BALANCED)
    if kind == "project":
        s.model.project(abi.PS3D_PROJ_ZERO_ORDER)
        return _get_fields(s, abi.PS3D_FIELDS_ZERO)
    f = {n: a.clone() for n, a in s.inputs.items()}
    f["p"] = torch.empty_like(f["u"])
    _check(s.solve(C.byref(p), *[f[n].data_ptr() for n in ("u", "v", "w", "p")], torch.cuda.current_stream().cuda_stream),
           "ps3d_pressure_solve_noalloc")
    return f


def _balance_options(case, p):
    return abi.OptBal(period=(case["ramp"] - 0.5) * p.dt, average=0.0, max_itts=case["iterations"], average_times=1,
                      tol=1e-30, enable_time_ave=0, adopt=0)


def _get_fields(s, which):
    m = s.model
    _check(m.L.ps3d_get_fields(m.h, which, *[abi.dptr(s.out[n]) for n in FIELDS]), "ps3d_get_fields")
    return {n: s.out[n] for n in FIELDS}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes and operations of one pass.  A step reads u, v, w, b, the pending pressure and two Adams-Bashforth levels
    of four tendencies and writes four tendencies and the state (168 bytes a point; 132 with the mixed path's FP32
    history); the pressure solve reads u, v, w, writes p, and holds one spectral array that three transforms exchange
    (64 bytes a point; mixed, with p read as well, 64).  Every output crosses to the host once."""
    if case["kind"] == "ensemble":
        pts = sum(p.nx * p.ny * p.nz for p in _members(case, 0))
        return {"bytes": pts * (232.0 * case["steps"] + 40.0), "flops": pts * 450.0 * case["steps"]}
    pts = case["nx"] * case["ny"] * case["nz"]
    if case["kind"] == "balance":
        n = 2 * case["ramp"] * case["iterations"]
        return {"bytes": pts * (232.0 * n + 192.0 * (2 * case["iterations"] + 1) + 32.0), "flops": pts * 450.0 * n}
    if case["kind"] == "project":
        return {"bytes": pts * 224.0, "flops": pts * 700.0}
    if case["kind"] == "pressure":
        return {"bytes": pts * 88.0, "flops": pts * 120.0}
    per = 196.0 if case.get("precision") == "mixed" else 232.0
    if case.get("friction") == "biharmonic":
        per += 64.0   # the start-of-step and the friction-updated field of four variables
    if case.get("flow") == "lee":
        per += 32.0   # wavemaker fields of w, background flow and buoyancy
    return {"bytes": pts * (per * case["steps"] + 40.0), "flops": pts * 450.0 * case["steps"]}


# ---------------------------------------------------------------------------
# the same in plain FP64 torch
# ---------------------------------------------------------------------------
def _E(f): return torch.roll(f, -1, 2)   # noqa: E704  the value one point east
def _W(f): return torch.roll(f, 1, 2)    # noqa: E704
def _N(f): return torch.roll(f, -1, 1)   # noqa: E704
def _S(f): return torch.roll(f, 1, 1)    # noqa: E704
def _T(f): return torch.roll(f, -1, 0)   # noqa: E704
def _D(f): return torch.roll(f, 1, 0)    # noqa: E704


class _Plain:
    """The model on one grid, every operator on whole arrays."""

    def __init__(self, p, f, forcing=None, device=DEVICE):
        self.p, self.dev = p, device
        self.f = {n: a.clone() for n, a in f.items()}
        self.pressure = torch.zeros_like(self.f["u"])
        self.forcing = forcing
        self.tend = []
        self.rigid = bool(p.enable_vertical_boundaries)
        self.dt, self.Ro = p.dt, p.Ro

        def wave(n, L, half=False):
            i = torch.arange(n // 2 + 1 if half else n, dtype=F64, device=device)
            if not half:
                i = torch.where(i < (n + 1) // 2, i, i - n)
            return 2 * math.pi * i / L

        def ksqr(k, d): return 2 * (1 - torch.cos(k * d)) / d ** 2   # noqa: E704
        self.kx, self.ky = wave(p.nx, p.Lx, True), wave(p.ny, p.Ly)
        self.hx, self.hy = ksqr(self.kx, p.dx), ksqr(self.ky, p.dy)
        k2 = self.hx[None, :] + self.hy[:, None]
        if self.rigid:
            m = torch.arange(p.nz, dtype=F64, device=device)
            c = torch.cos(math.pi / p.nz * (m[:, None] + 0.5) * m[None, :]) * math.sqrt(2.0 / p.nz)
            c[:, 0] = math.sqrt(1.0 / p.nz)
            self.cz = c.to(torch.complex128)
            lam = 2 * (1 - torch.cos(math.pi * m / p.nz)) / p.dz ** 2 / p.dsqr
            den = lam[:, None, None] + k2
            den[0, 0, 0] = 1.0
            self.inv = -1.0 / den
        else:
            den = ksqr(wave(p.nz, p.Lz), p.dz)[:, None, None] / p.dsqr + k2
            den[0, 0, 0] = 1.0
            self.inv = -1.0 / den
            self.inv[0, 0, 0] = 0.0

    def flux(self, e, n, t):
        p = self.p
        return (e - _W(e)) / p.dx + (n - _S(n)) / p.dy + (t - _D(t)) / p.dz

    def lid(self, f, levels=1):
        if self.rigid:
            f[-levels:] = 0.0
        return f

    def tendencies(self):
        p, (u, v, w, b) = self.p, (self.f[n] for n in FIELDS)
        lid = self.lid
        if p.enable_nonlinear:
            db = -self.Ro * self.flux((b + _E(b)) * u / 2, (b + _N(b)) * v / 2, lid((b + _T(b)) * w / 2))
            du = -self.Ro * self.flux((u + _E(u)) ** 2 / 4, (u + _N(u)) * (v + _E(v)) / 4, lid((u + _T(u)) * (w + _E(w)) / 4))
            dv = -self.Ro * self.flux((v + _E(v)) * (u + _N(u)) / 4, (v + _N(v)) ** 2 / 4, lid((v + _T(v)) * (w + _N(w)) / 4))
            dw = -self.Ro * p.dsqr * self.flux((w + _E(w)) * (u + _T(u)) / 4, (w + _N(w)) * (v + _T(v)) / 4,
                                               lid((w + _T(w)) ** 2 / 4, 2))
        else:
            du, dv, dw, db = (torch.zeros_like(u) for _ in range(4))
        db = db - (w + _D(w)) * p.N0 ** 2 / 2
        du = du + p.f0 / 4 * (v + _S(v) + _E(v) + _E(_S(v)))
        dv = dv - p.f0 / 4 * (u + _W(u) + _N(u) + _N(_W(u)))
        dw = lid(dw + (b + _T(b)) / 2)
        if self.forcing is not None:
            U = self.forcing["u_back"]
            du = du - self.Ro * self.flux((U + _E(U)) * (u + _E(u)) / 2, (U + _N(U)) * (v + _E(v)) / 4, (U + _T(U)) * (w + _E(w)) / 4)
            for n, e in (("v", (v + _E(v)) * (U + _N(U)) / 4), ("w", (w + _E(w)) * (U + _T(U)) / 4), ("b", (b + _E(b)) * U / 2)):
                d = -self.Ro * (e - _W(e)) / p.dx
                if n == "v":
                    dv = dv + d
                elif n == "w":
                    dw = dw + p.dsqr * d
                else:
                    db = db + d
        return {"u": du, "v": dv, "w": dw, "b": db}

    def friction(self, n):
        """The field after the friction that is switched on, in place in the reference's order."""
        p, f = self.p, self.f[n]
        H, V, Hb, Vb = (p.Ah, p.Av, p.Ahbi, p.Avbi) if n != "b" else (p.Kh, p.Kv, p.Khbi, p.Kvbi)
        new = f
        if H > 0 or V > 0:
            new = f + self.dt * self.flux(H * (_E(f) - f) / p.dx, H * (_N(f) - f) / p.dy, self.lid(V * (_T(f) - f) / p.dz))
            if n == "w":
                self.lid(new)
        if Hb > 0:   # beyond the interior the start-of-step values stand
            g = _pad2(f, new, (1, 2))
            d = -Hb * ((g[:, 1:-1, 2:] - 2 * g[:, 1:-1, 1:-1] + g[:, 1:-1, :-2]) / p.dx ** 2
                       + (g[:, 2:, 1:-1] - 2 * g[:, 1:-1, 1:-1] + g[:, :-2, 1:-1]) / p.dy ** 2)
            new = new + self.dt * ((d[:, 1:-1, 2:] - 2 * d[:, 1:-1, 1:-1] + d[:, 1:-1, :-2]) / p.dx ** 2
                                   + (d[:, 2:, 1:-1] - 2 * d[:, 1:-1, 1:-1] + d[:, :-2, 1:-1]) / p.dy ** 2)
        if Vb > 0:
            g = _pad2(f, new, (0,))
            fl = -Vb * (g[1:] - g[:-1]) / p.dz
            if self.rigid:
                fl[:2] = 0.0
                fl[-2:] = 0.0
            d = (fl[1:] - fl[:-1]) / p.dz
            fl = (d[1:] - d[:-1]) / p.dz
            if self.rigid:
                fl[0] = 0.0
                fl[-1] = 0.0
            new = new + self.dt * (fl[1:] - fl[:-1]) / p.dz
            if n == "w":
                self.lid(new)
        return new

    def step(self, itt):
        p = self.p
        t = self.tendencies()
        self.tend = [t] + self.tend[:2]
        if itt == 0:
            c = (1.0,)
        elif itt == 1 or not p.enable_AB_3_order:
            c = (1.5 + p.eps_ab, -0.5 - p.eps_ab)
        else:
            c = (23 / 12, -16 / 12, 5 / 12)
        new = {}
        for n in FIELDS:
            new[n] = self.friction(n)
            if self.forcing is not None and n == "w":
                a = self.forcing["omega"] * p.dt * itt
                new[n] = new[n] + p.dt * (math.cos(a) * self.forcing["w_r"] + math.sin(a) * self.forcing["w_i"])
            h = (self.dt / p.dsqr) if n == "w" else self.dt
            new[n] = new[n] + h * sum(ck * tk[n] for ck, tk in zip(c, self.tend))
        self.f = new
        self.project_pressure()

    def project_pressure(self):
        p, f = self.p, self.f
        q = torch.fft.rfft2(self.flux(f["u"], f["v"], f["w"]) / self.dt)
        if self.rigid:
            s = (self.cz.T @ q.reshape(p.nz, -1)).reshape(q.shape) * self.inv
            s = (self.cz @ s.reshape(p.nz, -1)).reshape(q.shape)
            s[:, 0, 0] = torch.cumsum(torch.cumsum(torch.cat((torch.zeros_like(q[:1, 0, 0]), q[:-1, 0, 0])), 0), 0) * (p.dz ** 2 * p.dsqr)
            pr = torch.fft.irfft2(s, s=(p.ny, p.nx))
        else:
            pr = torch.fft.irfft2(torch.fft.ifft(torch.fft.fft(q, dim=0) * self.inv, dim=0), s=(p.ny, p.nx))
        f["u"] = f["u"] - self.dt * (_E(pr) - pr) / p.dx
        f["v"] = f["v"] - self.dt * (_N(pr) - pr) / p.dy
        f["w"] = self.lid(f["w"] - self.dt / p.dsqr * (_T(pr) - pr) / p.dz)
        self.pressure = pr

    # -- the geostrophic mode under a rigid lid (u, v in cosines, b in sines of the level) -----------
    def _mode(self):
        p, dev = self.p, self.dev
        m = torch.arange(p.nz, dtype=F64, device=dev)
        a = math.pi / p.nz * (m[:, None] + 0.5) * m[None, :]
        phi = math.sqrt(2 / p.Lz) * torch.cos(a)
        phi[:, 0] = math.sqrt(1 / p.Lz)
        psib = math.sqrt(2 / p.Lz) * torch.sin(a)
        half = math.pi * m / p.nz / 2
        lam, carg = (2 * torch.sin(half) / p.dz)[:, None, None], torch.cos(half)[:, None, None]
        ex, ey = torch.exp(1j * self.kx * p.dx)[None, :], torch.exp(1j * self.ky * p.dy)[:, None]
        f2 = p.f0 ** 2 * (0.5 * (1 + torch.cos(self.kx * p.dx)))[None, :] * (0.5 * (1 + torch.cos(self.ky * p.dy)))[:, None]
        kp_x, kp_y = -1j * (ex - 1) / p.dx, -1j * (ey - 1) / p.dy
        safe = torch.where(f2 == 0, torch.ones_like(f2), f2)
        qx = -1j * p.f0 * (ex + 1) / 2 * (ey.conj() + 1) / 2 * kp_y / safe
        qy = 1j * p.f0 * (ex.conj() + 1) / 2 * (ey + 1) / 2 * kp_x / safe
        n2 = p.N0 ** 2 * carg ** 2
        qb = -(lam * carg * p.N0 ** 2 / n2)
        k2 = (self.hx[None, :] + self.hy[:, None])
        dd = k2 * n2 + f2 * lam ** 2
        on = ((f2 != 0) & (k2 > 0))[None] & (dd > 0)
        pc = torch.where(on, f2 * n2 / torch.where(dd > 0, dd, torch.ones_like(dd)), torch.zeros_like(dd))
        return phi.to(torch.complex128), psib.to(torch.complex128), qx, qy, qb, pc

    def geostrophic(self, base=None, only=False):
        """(mode amplitude, the fields of that mode); with `base` the state with its amplitude exchanged for base."""
        p, f = self.p, self.f
        phi, psib, qx, qy, qb, pc = self._mode()
        sh = (p.nz, p.ny, p.nx // 2 + 1)

        def ana(a, m): return (m.T @ torch.fft.rfft2(a).reshape(p.nz, -1)).reshape(sh) * (p.dx * p.dy * p.dz)   # noqa: E704
        def syn(s, m): return torch.fft.irfft2((m @ s.reshape(p.nz, -1)).reshape(sh), s=(p.ny, p.nx)) / (p.dx * p.dy)   # noqa: E704
        g = pc * (qx.conj() * ana(f["u"], phi) + qy.conj() * ana(f["v"], phi) + qb * ana(f["b"], psib) / p.N0 ** 2)
        if only:
            return g, None
        d = g if base is None else base - g
        out = {"u": syn(d * qx, phi), "v": syn(d * qy, phi), "w": torch.zeros_like(f["w"]), "b": syn(d * qb, psib)}
        if base is not None:
            out = {n: f[n] + out[n] for n in FIELDS}
            # b goes through the sine modes 1 .. nz-1 and back, which leaves out its alternating part
            a = 1.0 - 2.0 * (torch.arange(p.nz, device=self.dev) % 2).to(F64)[:, None, None]
            out["b"] = out["b"] - a * (a * f["b"]).mean(0)
        return g, out

    def optimal_balance(self, ramp, iterations):
        p = self.p
        period = (ramp - 0.5) * p.dt
        base, _ = self.geostrophic(only=True)
        keep = (p.Ahbi, p.Avbi, p.Khbi, p.Kvbi)

        def weight(theta):
            t1, t2 = 1.0 / max(1e-32, theta), 1.0 / max(1e-32, 1.0 - theta)
            return math.exp(-t1) / (math.exp(-t1) + math.exp(-t2))

        def ramped(backward):
            self.dt = -p.dt if backward else p.dt
            for s in range(int(period / p.dt) + 1):
                r = weight(s * p.dt / period)
                self.Ro = (1.0 - r if backward else r) * p.Ro
                self.step(0)

        for _ in range(iterations):
            p.Ahbi = p.Avbi = p.Khbi = p.Kvbi = 0.0
            ramped(True)
            p.Ahbi, p.Avbi, p.Khbi, p.Kvbi = keep
            self.f = self.geostrophic()[1]
            ramped(False)
            self.f = self.geostrophic(base)[1]
        return self.f


def _pad2(old, new, axes):
    """`new` with two periodic points of `old` on both sides along the axes."""
    g = old
    for ax in axes:
        i = torch.arange(-2, old.shape[ax] + 2, device=old.device) % old.shape[ax]
        g = g.index_select(ax, i)
    g = g.clone()
    inner = tuple(slice(2, -2) if ax in axes else slice(None) for ax in range(3))
    g[inner] = new
    return g


def _laid_out(m, names):
    out = {n: _halo(m.f[n]).cpu().numpy() for n in names if n != "p"}
    if "p" in names:
        out["p"] = _halo(m.pressure, ghost_levels=m.rigid).cpu().numpy()
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        params = _members(case, seed)
        blocks = {}
        for i, p in enumerate(params):
            m = _Plain(p, _fields(p, "eddy", seed * 1009 + i))
            for itt in range(case["steps"]):
                m.step(itt)
            o = _laid_out(m, FIELDS + ("p",))
            blocks.setdefault(abi.halo_shape(p), []).append(np.stack([o[n] for n in FIELDS + ("p",)]))
        return [np.stack(blocks[sh]) for sh in sorted(blocks)]
    p = _params(case)
    if kind == "pressure":
        f = _pressure_inputs(case, p, seed)
        m = _Plain(p, {**f, "b": torch.zeros_like(f["u"])})
        m.project_pressure()
        return {"u": m.f["u"], "v": m.f["v"], "w": m.f["w"], "p": m.pressure}
    flow = case.get("flow", "eddy")
    m = _Plain(p, _fields(p, flow, seed), _forcing(p, seed) if flow == "lee" else None)
    if kind == "project":
        _, f = m.geostrophic()
        return {n: _halo(f[n]).cpu().numpy() for n in FIELDS}
    if kind == "balance":
        f = m.optimal_balance(case["ramp"], case["iterations"])
        return {n: _halo(f[n]).cpu().numpy() for n in FIELDS}
    for itt in range(case["steps"]):
        m.step(itt)
    return _laid_out(m, FIELDS + ("p",))
