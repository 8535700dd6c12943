"""Performance cases: the work that users of this framework have it do.

A pass is what a program does between two outputs: it advances the resident
state by some steps through the C-ABI's front end and reads the new state
back into its own host arrays (pinned, in the reference's layout with ghost
layers; single precision for a mixed handle, as the reference's default
build has them, double for an FP64 one).  Two kinds of call work on host
arrays by their nature: the PoisSolver replacement and TMarchRK3 on host
arrays.

Kinds of case:
  channel  one domain: rough bottom with the log-law wall model, free-slip
           top, periodic x and y; optionally the temperature (adiabatic or
           over a heated surface), passive scalars with a point source and
           averaged slices, and variable time steps
  cubes    an array of cubes on a stretched grid under a mean pressure
           gradient
  batch    an ensemble of uneven channels stepped together
  poisson  the PoisSolver calls on host arrays, stretched z
  march    TMarchRK3 on host arrays: state in, one step, state out

Initial fields are log profiles with uniform perturbations (and a stratified
temperature, and a Gaussian puff of scalar), projected once, as everywhere
in this repository; they are drawn on the GPU from the seed.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from gpu_elmm_b200 import lib as L
from gpu_elmm_b200.config import FIELD_SCALAR, FIELD_TEMPERATURE, make_config
from gpu_elmm_b200.workloads import CUBES_PR_GRADIENT_X, stretched_zw

KAPPA_Z0, USTAR, AMP = 0.01, 0.3, 0.1
T_REF, GRAV, NU, PRANDTL = 295.0, 9.81, 1.0 / 70000, 0.7
RK_ALPHA = (4.0 / 15.0, 1.0 / 15.0, 1.0 / 6.0)
RK_BETA = (8.0 / 15.0, 5.0 / 12.0, 3.0 / 4.0)
RK_RHO = (0.0, -17.0 / 60.0, -5.0 / 12.0)


# ----------------------------------------------------------------- the cases
def listed():
    return [
        # the small channel of the quickest runs: few cells, a step is bound by
        # latency and launches; on both precision paths
        {"name": "channel-64-mixed", "kind": "channel", "nx": 64, "ny": 64, "nz": 32, "steps": 40, "mixed": True,
         "theta": False, "flux": 0.0, "scalars": 0, "vdt": False},
        {"name": "channel-64-fp64", "kind": "channel", "nx": 64, "ny": 64, "nz": 32, "steps": 40, "mixed": False,
         "theta": False, "flux": 0.0, "scalars": 0, "vdt": False},
        # the benchmark's buoyant channel, both paths
        {"name": "buoyant-256-mixed", "kind": "channel", "nx": 256, "ny": 256, "nz": 128, "steps": 20, "mixed": True,
         "theta": True, "flux": 0.0, "scalars": 0, "vdt": False},
        {"name": "buoyant-256-fp64", "kind": "channel", "nx": 256, "ny": 256, "nz": 128, "steps": 8, "mixed": False,
         "theta": True, "flux": 0.0, "scalars": 0, "vdt": False},
        # a production-size boundary layer
        {"name": "channel-512-mixed", "kind": "channel", "nx": 512, "ny": 512, "nz": 128, "steps": 6, "mixed": True,
         "theta": False, "flux": 0.0, "scalars": 0, "vdt": False},
        # urban flow: a quarter of the benchmark's cube array
        {"name": "cubes-192-mixed", "kind": "cubes", "per_side": 4, "nz": 96, "steps": 20, "mixed": True},
        # a dispersion request: passive scalar, point source, averaged slices
        {"name": "dispersion-128-mixed", "kind": "channel", "nx": 128, "ny": 128, "nz": 64, "steps": 40,
         "mixed": True, "theta": False, "flux": 0.0, "scalars": 1, "vdt": False},
        # an ensemble of uneven small domains
        {"name": "batch-24-mixed", "kind": "batch", "domains": 24, "draw": 1, "steps": 20, "mixed": True},
        # a convective boundary layer on a grid without powers of two, odd in
        # every direction, variable time steps
        {"name": "convective-135-mixed", "kind": "channel", "nx": 135, "ny": 135, "nz": 75, "steps": 20,
         "mixed": True, "theta": True, "flux": 0.1, "scalars": 0, "vdt": True},
        # the same physics in double precision on another common size
        {"name": "convective-160-fp64", "kind": "channel", "nx": 160, "ny": 160, "nz": 80, "steps": 16,
         "mixed": False, "theta": True, "flux": 0.1, "scalars": 0, "vdt": False},
        # a program that uses the Poisson solver alone
        {"name": "poisson-192-fp64", "kind": "poisson", "nx": 192, "ny": 192, "nz": 96, "mixed": False},
        # a host that keeps the state on its side
        {"name": "march-256-mixed", "kind": "march", "nx": 256, "ny": 256, "nz": 128, "mixed": True},
    ]


def _smooth(lo, hi):
    """The lengths in lo..hi that factor into 2, 3 and 5."""
    out = []
    for n in range(lo, hi + 1):
        r = n
        for p in (2, 3, 5):
            while r % p == 0:
                r //= p
        if r == 1:
            out.append(n)
    return out


def _length(rng, lo, hi):
    """A length that the transforms take, spread over the logarithm of lo..hi."""
    target = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(_smooth(lo, hi), key=lambda n: abs(math.log(n / target)))


def draw(rng):
    kind = rng.choice(["channel"] * 7 + ["batch", "poisson", "march", "cubes"])
    mixed = rng.random() < 0.7
    if kind == "cubes":
        return {"kind": kind, "per_side": rng.choice([2, 3, 4]), "nz": rng.randint(40, 96),
                "steps": rng.randint(10, 20), "mixed": mixed}
    if kind == "batch":
        return {"kind": kind, "domains": rng.randint(4, 20), "draw": rng.randint(2, 1 << 20), "steps": 15,
                "mixed": mixed}
    if kind in ("poisson", "march"):
        return {"kind": kind, "nx": _length(rng, 48, 240), "ny": _length(rng, 48, 240), "nz": rng.randint(24, 120),
                "mixed": mixed}
    while True:
        nx, ny, nz = _length(rng, 40, 512), _length(rng, 40, 512), int(math.exp(rng.uniform(math.log(20), math.log(320))))
        cells = nx * ny * nz
        if 1e5 <= cells <= 1.6e7:
            break
    theta = rng.random() < 0.5
    # a pass of about as much work as the listed ones of that size have
    steps = max(3, min(40, int((8e7 if mixed else 3e7) / cells)))
    return {"kind": "channel", "nx": nx, "ny": ny, "nz": nz, "steps": steps, "mixed": mixed, "theta": theta,
            "flux": rng.choice([0.0, 0.05, 0.1]) if theta else 0.0, "scalars": rng.choice([0, 0, 0, 1, 2]),
            "vdt": rng.random() < 0.25}


def _batch_sizes(case):
    """(nx, ny, nz, u*) of each domain of an ensemble."""
    g = np.random.RandomState(case["draw"])
    axes = (32, 48, 64, 96, 128)
    return [tuple(int(axes[q]) for q in g.randint(0, 5, 3)) + (float(g.uniform(0.2, 0.5)),)
            for _ in range(case["domains"])]


# ------------------------------------------------------------- configuration
def _source(nx, ny, nz):
    """The cell (1-based) of the point source and of the slices."""
    return nx // 3 + 1, ny // 2, max(2, nz // 4)


def _config(case):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    ci, cj, ck = _source(nx, ny, nz)
    kw = {}
    if case.get("theta") or case["kind"] == "march":
        kw.update(buoyancy=True, heat_flux=(case.get("flux", 0.0), 0.0))
    if case.get("scalars"):
        kw.update(num_scalars=case["scalars"], point_sources=[(1, (ci - 0.5, cj - 0.5, ck - 0.5), 1.0)],
                  avg_slice_k=ck, avg_slice_j=cj, avg_weight=1.0 / case["steps"])
    if case.get("vdt"):
        kw.update(variable_dt=True, cfl=0.5, dt_max=0.04)
    return make_config(nx, ny, nz, precision=1 if case["mixed"] else 0, **kw)


# -------------------------------------------------------------------- inputs
def _rand(gen, nz, ny, nx):
    """U(-AMP, AMP) on the interior, FP32 values."""
    r = torch.rand((nz, ny, nx), generator=gen, device="cuda", dtype=torch.float32)
    return AMP * (2 * r - 1)


def _interiors(nx, ny, nz, seed, salt=0, ustar=USTAR, zpr=None, theta=False, scalars=0):
    """Interior fields (FP32, on the GPU): U, V, W (nz - 1 levels), and the
    temperature and scalars."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed((seed * 1000003 + salt) & 0x7FFFFFFFFFFF)
    if zpr is None:
        zpr = np.arange(nz) + 0.5
    prof = torch.tensor(ustar / 0.41 * np.log(zpr / KAPPA_Z0), device="cuda", dtype=torch.float32)[:, None, None]
    out = {"U": prof + _rand(gen, nz, ny, nx), "V": _rand(gen, nz, ny, nx), "W": _rand(gen, nz - 1, ny, nx)}
    if theta:
        strat = torch.tensor(T_REF + 0.01 * zpr, device="cuda", dtype=torch.float32)[:, None, None]
        out["T"] = strat + 0.5 * _rand(gen, nz, ny, nx)
    if scalars:
        ci, cj, ck = _source(nx, ny, nz)
        i, j, k = (torch.arange(1, n + 1, device="cuda", dtype=torch.float64) for n in (nx, ny, nz))
        di, dj = (i - ci).abs(), (j - cj).abs()
        di, dj = torch.minimum(di, nx - di), torch.minimum(dj, ny - dj)
        r2 = (k - ck)[:, None, None] ** 2 + dj[None, :, None] ** 2 + di[None, None, :] ** 2
        for s in range(scalars):
            sigma = 2.0 + s
            out["S%d" % (s + 1)] = torch.exp(-r2 / (2 * sigma * sigma)).float()
    return out


def _pinned(shape, dtype):
    return torch.zeros(shape, dtype=dtype, pin_memory=True).numpy()


def _host(shape, interior, dtype=torch.float32, lo=-2):
    """A pinned host array in the reference's layout, zero ghosts."""
    a = torch.zeros(shape, dtype=dtype, pin_memory=True)
    if interior is not None:
        o, (nz, ny, nx) = 1 - lo, interior.shape
        a[o:o + nz, o:o + ny, o:o + nx] = interior.to(dtype).cpu()
    return a.numpy()


@functools.lru_cache(maxsize=4)
def _cube_solids(per_side, nz):
    """The geometry pass of the cube array: once per program, as the mesh of a
    user's city is made once."""
    from gpu_elmm_b200.solids import build_solids, cube_array
    zw = stretched_zw(nz)
    n = 48 * per_side
    cfg = make_config(n, n, nz, zW=zw, pr_gradient_x=CUBES_PR_GRADIENT_X)
    return build_solids(cfg, cube_array(per_side, 16.0, 48.0, float(zw[min(16, nz // 2)]), offset=16.0, depth=5.0))


def _fields_of(case):
    f = ["T"] if case.get("theta") or case["kind"] == "march" else []
    return f + ["S%d" % (s + 1) for s in range(case.get("scalars", 0))]


def _fptr(a):
    return L.fptr(a) if a.dtype == np.float32 else L.ptr(a)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        sizes = _batch_sizes(case)
        b = L.Batch([make_config(nx, ny, nz, precision=1 if case["mixed"] else 0) for nx, ny, nz, _ in sizes])
        # one buffer per field, the domains' arrays one after the other
        shapes = [(g.shape_u(), g.shape_v(), g.shape_w(), g.shape_p()) for g in b.grids]
        flat = {c: _pinned((sum(math.prod(s[q]) for s in shapes),), torch.float64) for q, c in enumerate("UVWP")}
        out, at = [], [0, 0, 0, 0]
        for d, (nx, ny, nz, us) in enumerate(sizes):
            f, arrays = _interiors(nx, ny, nz, seed, d + 1, us), []
            for q, c in enumerate("UVWP"):
                shape = shapes[d][q]
                a = flat[c][at[q]:at[q] + math.prod(shape)].reshape(shape)
                at[q] += a.size
                if c in f:
                    k, j, i = f[c].shape
                    a[3:3 + k, 3:3 + j, 3:3 + i] = f[c].cpu().numpy()
                arrays.append(a)
            b.upload(d, *arrays[:3])
            out.append(arrays)
        b.project(1.0)
        return {"case": case, "batch": b, "out": out, "flat": flat}
    if kind == "poisson":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        s = L.PoissonSolver((nx, ny, nz), L=(float(nx), float(ny)), precision=1 if case["mixed"] else 0,
                            zW=stretched_zw(nz, 0.5, 1.01))
        return {"case": case, "solver": s, "rhs": _host((nz + 2, ny + 2, nx + 2), _poisson_rhs(case, seed), torch.float64, 0),
                "phi": _pinned((nz + 4, ny + 4, nx + 4), torch.float64)}
    if kind == "cubes":
        n, nz = 48 * case["per_side"], case["nz"]
        zw = stretched_zw(nz)
        cfg = make_config(n, n, nz, zW=zw, pr_gradient_x=CUBES_PR_GRADIENT_X, precision=1 if case["mixed"] else 0)
        f = _interiors(n, n, nz, seed, zpr=(zw[:-1] + zw[1:]) / 2)
    else:
        cfg = _config(case)
        f = _interiors(case["nx"], case["ny"], case["nz"], seed, theta="T" in _fields_of(case),
                       scalars=case.get("scalars", 0))
    d = L.Domain(cfg)
    g = d.grid
    shapes = {"U": g.shape_u(), "V": g.shape_v(), "W": g.shape_w(), "P": g.shape_p()}
    host = {c: _host(shapes[c], f.get(c)) for c in "UVWP"}
    d.upload_f32(host["U"], host["V"], host["W"])
    for c in _fields_of(case):
        host[c] = _host(g.shape_t(), f[c])
        if c == "T":
            d.upload_temperature_f32(host[c])
        else:
            d.upload_scalar(int(c[1:]), host[c].astype(np.float64))
    d.project(1.0)
    if kind == "cubes":
        d.set_solids(_cube_solids(case["per_side"], case["nz"]))
    state = {"case": case, "domain": d, "out": host}
    if kind == "march":  # the host holds the state: the projected fields
        L.check(L.lib().elmm_download_state_float(d.h, *[L.fptr(host[c]) for c in "UVWP"]), "download")
        L.check(L.lib().elmm_download_field_float(d.h, FIELD_TEMPERATURE, L.fptr(host["T"])), "download")
    elif not case["mixed"]:  # results in double precision
        state["out"] = {c: _pinned(a.shape, torch.float64) for c, a in host.items()}
    if case.get("scalars"):
        state["xy"] = _pinned((case["ny"], case["nx"]), torch.float64)
        state["xz"] = _pinned((case["nz"], case["nx"]), torch.float64)
    return state


# ---------------------------------------------------------------- one pass
def run(state):
    case, lib = state["case"], L.lib()
    kind = case["kind"]
    if kind == "batch":
        b = state["batch"]
        b.step(case["steps"])
        for d, arrays in enumerate(state["out"]):
            L.check(lib.elmm_batch_download_state(b.h, d, *[L.ptr(a) for a in arrays]), "elmm_batch_download_state")
        return state["flat"]
    if kind == "poisson":
        return state["solver"].execute(state["phi"], state["rhs"])
    d, out = state["domain"], state["out"]
    if kind == "march":
        d.march_host_f32(out["U"], out["V"], out["W"], out["P"], out["T"], n=1)
        return out
    d.step(case["steps"])
    single = case["mixed"]
    down, field = ((lib.elmm_download_state_float, lib.elmm_download_field_float) if single
                   else (lib.elmm_download_state, lib.elmm_download_field))
    L.check(down(d.h, *[_fptr(out[c]) for c in "UVWP"]), "elmm_download_state")
    for c in _fields_of(case):
        L.check(field(d.h, FIELD_TEMPERATURE if c == "T" else FIELD_SCALAR + int(c[1:]) - 1, _fptr(out[c])),
                "elmm_download_field")
    if case.get("scalars"):
        L.check(lib.elmm_download_scalar_slices(d.h, 1, L.ptr(state["xy"]), L.ptr(state["xz"])),
                "elmm_download_scalar_slices")
        return {**out, "xy": state["xy"], "xz": state["xz"]}
    return out


# --------------------------------------------------------------------- work
def _words(case):
    return 4 if case["mixed"] else 8


def work(case):
    """Every stage reads and writes the state (velocity, pressure, scalars)
    and the last stage's tendencies once; a host array crosses once each way
    it goes."""
    kind, w = case["kind"], _words(case)
    if kind == "poisson":
        n = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 2 * 8 * n, "flops": n * (5 * math.log2(case["nx"] * case["ny"]) + 10)}
    if kind == "batch":
        cells = [nx * ny * nz for nx, ny, nz, _ in _batch_sizes(case)]
        n, steps, host, ns = sum(cells), case["steps"], 4 * 8 * sum(cells), 0
        modes = math.log2(64 * 64)
    elif kind == "cubes":
        n = (48 * case["per_side"]) ** 2 * case["nz"]
        steps, host, ns, modes = case["steps"], 4 * w * n, 0, 2 * math.log2(48 * case["per_side"])
    else:
        n = case["nx"] * case["ny"] * case["nz"]
        ns = len(_fields_of(case))
        steps = case.get("steps", 1)
        host = (4 + ns) * w * n * (2 if kind == "march" else 1)
        modes = math.log2(case["nx"] * case["ny"])
    stage = 2 * (4 + ns) + (3 + ns) * 4 / 3
    return {"bytes": 3 * steps * stage * w * n + host,
            "flops": 3 * steps * n * (300 + 100 * ns + 5 * modes + 10)}


# ---------------------------------------------------------------- tolerance
def tolerance(case):
    """About four times the distance to exact() seen at the listed and drawn
    cases.  The pressure is the widest: the projection turns the rounding of
    the velocity's divergence into it, and without a stratification, whose
    hydrostatic part is large, little else stands beside that noise."""
    if not case["mixed"]:
        # march: single-precision host arrays
        return {"rel": 1e-6, "max": 1e-5} if case["kind"] == "march" else {"rel": 3e-11, "max": 1e-9}
    if case["kind"] == "poisson":
        return {"rel": 1e-5, "max": 1e-4}
    if case.get("theta") or case["kind"] == "march":
        return {"rel": 2e-4, "max": 5e-3}
    return {"rel": 6e-3, "max": 1e-1}


# ------------------------------------------------ the same in 64 bits, plainly
def _poisson_rhs(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    r = torch.rand((nz, ny, nx), generator=gen, device="cuda", dtype=torch.float64) - 0.5
    dz = torch.tensor(np.diff(stretched_zw(nz, 0.5, 1.01)), device="cuda")[:, None, None]
    return r - (r * dz).mean() / dz.mean()  # solvable: its integral vanishes


def _xm(a):
    return torch.roll(a, 1, -1)


def _xp(a):
    return torch.roll(a, -1, -1)


def _ym(a):
    return torch.roll(a, 1, -2)


def _yp(a):
    return torch.roll(a, -1, -2)


class _Poisson:
    """Fourier in x and y; in z the eigenvectors of the three-point operator."""

    def __init__(self, nx, ny, zw):
        nz = len(zw) - 1
        self.shape = (nz, ny, nx)
        zp, dz = (zw[:-1] + zw[1:]) / 2, np.diff(zw)
        a = np.zeros((nz, nz))
        for k in range(nz):
            for q in (k - 1, k + 1):
                if 0 <= q < nz:
                    v = 1.0 / (abs(zp[q] - zp[k]) * dz[k])
                    a[k, q] += v
                    a[k, k] -= v
        s = np.sqrt(dz)
        sym = s[:, None] * a / s[None, :]
        mu, q = np.linalg.eigh((sym + sym.T) / 2)
        self.null = int(np.argmax(mu))
        dev = {"device": "cuda", "dtype": torch.float64}
        self.mu, self.q, self.s = (torch.tensor(x, **dev) for x in (mu, q, s))
        kx, ky = np.arange(nx // 2 + 1), np.arange(ny)
        lam = -4 * np.sin(np.pi * ky / ny)[:, None] ** 2 - 4 * np.sin(np.pi * kx / nx)[None, :] ** 2
        self.lam = torch.tensor(lam, **dev)

    def solve(self, r):
        nz, ny, nx = self.shape
        f = torch.fft.rfft2(r)
        den = self.mu[:, None, None] + self.lam
        den[self.null, 0, 0] = float("inf")
        parts = []
        for p in (f.real, f.imag):
            m = (p * self.s[:, None, None]).reshape(nz, -1)
            m = (self.q.T @ m).reshape(den.shape) / den
            parts.append((self.q @ m.reshape(nz, -1)).reshape(den.shape) / self.s[:, None, None])
        x = torch.fft.irfft2(torch.complex(*parts), s=(ny, nx))
        return x - x.mean()


def _kappa(vel, a, b, c, e):
    """The limited flux through the face between cells b and c."""
    pos = vel > 0
    sr, sl = torch.where(pos, c - b, b - c), torch.where(pos, b - a, c - e)
    sg = 1e-8 * torch.copysign(torch.ones_like(sl), sl)
    r = (sr + sg) / (sl + sg)
    lim = torch.clamp(torch.minimum(2 * r, torch.clamp((1 + 2 * r) / 3, max=2.0)), min=0.0)
    return torch.where(pos, vel * (b + (b - a) * lim / 2), vel * (c + (c - e) * lim / 2))


class _Channel:
    """A unit-spaced channel in 64 bits: levels 0..nz+1 (U, V) and 0..nz (W)."""

    def __init__(self, nx, ny, nz, f, flux=0.0, sources=None, vdt=False):
        self.n = (nx, ny, nz)
        self.pois = _Poisson(nx, ny, np.arange(nz + 1.0))
        self.f = {c: a.double() for c, a in f.items() if c not in "UVW"}
        z = torch.zeros((1, ny, nx), device="cuda", dtype=torch.float64)
        self.U, self.V = f["U"].double(), f["V"].double()
        self.W = torch.cat([z, f["W"].double(), z])  # levels 0..nz
        self.P = torch.zeros((nz, ny, nx), device="cuda", dtype=torch.float64)
        self.flux, self.sources, self.vdt, self.dt = flux, sources or {}, vdt, 0.02
        self.us = [torch.ones((ny, nx), device="cuda", dtype=torch.float64) for _ in range(2)]
        self.adv = {}
        self.kappa = NU / PRANDTL
        self._project(1.0)
        self.td = (self._viscosity() - NU) / 0.6 + self.kappa
        self._walls()

    def _ghosts(self, a):  # no-slip bottom, free-slip top
        return torch.cat([-a[:1], a, a[-1:]])

    def _project(self, coef):
        div = (self.U - _xm(self.U)) + (self.V - _ym(self.V)) + (self.W[1:] - self.W[:-1])
        phi = self.pois.solve(div / coef)
        self.U = self.U - coef * (_xp(phi) - phi)
        self.V = self.V - coef * (_yp(phi) - phi)
        self.W[1:-1] -= coef * (phi[1:] - phi[:-1])
        self.P = self.P + phi
        self.P = self.P - self.P[-1].mean()

    def _viscosity(self):
        U, V, W = self._ghosts(self.U), self._ghosts(self.V), self.W
        u, v, w, wb = self.U, self.V, W[1:], W[:-1]
        ua, va = U + _xm(U), V + _ym(V)
        d01 = (_yp(ua) - _ym(ua))[1:-1] / 4 + (_xp(va) - _xm(va))[1:-1] / 4
        d02 = (ua[2:] - ua[:-2]) / 4 + (_xp(w + wb) - _xm(w + wb)) / 4
        d12 = (va[2:] - va[:-2]) / 4 + (_yp(w + wb) - _ym(w + wb)) / 4
        s = (u - _xm(u)) ** 2 + (v - _ym(v)) ** 2 + (w - wb) ** 2 + (d01 ** 2 + d02 ** 2 + d12 ** 2) / 2
        return torch.sqrt(2 * s) * 0.1 ** 2 + NU

    def _walls(self):
        """u*^2 over the wind speed times each component, at the lowest level."""
        u, v = self.U[0], self.V[0]
        vu = (_xp(v) + v + _xp(_ym(v)) + _ym(v)) / 4
        uv = (_yp(u) + u + _yp(_xm(u)) + _xm(u)) / 4
        out = []
        for q, (a, b) in enumerate(((u, vu), (v, uv))):
            vel = torch.sqrt(a * a + b * b)
            lam = torch.sqrt(NU * vel / 0.5)
            rough = vel * 0.41 / math.log(0.5 / KAPPA_Z0)
            us = torch.where(0.5 * lam / NU < 11.225 * 1.1, lam, rough)
            if self.flux > 0:
                us = self._obukhov(self.us[q], vel)
            us = torch.clamp(torch.where(vel != 0, us, self.us[q] if self.flux <= 0 else 0 * us), min=0)
            self.us[q] = us
            out.append(torch.where(vel > 1.5e-8, a / vel * us * us, 0 * us))
        return out

    def _obukhov(self, us, vel):
        us, zl, psi = us.clone(), torch.zeros_like(us), torch.zeros_like(us)
        live = torch.ones_like(us, dtype=torch.bool)
        done = torch.zeros_like(us)
        f32 = lambda x: float(np.float32(x))
        for _ in range(50):
            old = us
            arg = torch.clamp(0.5 / KAPPA_Z0 - psi, min=f32(1e-5))
            us = us + (torch.clamp(vel * 0.4 / torch.log(arg), min=0) - us) / 2
            zl2 = 0.5 * (0.4 * (GRAV / T_REF) * self.flux) / (-(us ** 3))
            zl = torch.where(us < f32(1e-4), -10000.0 + 0 * zl, zl + (zl2 - zl) / 2)
            x = torch.clamp(1 - 15 * zl, min=0) ** 0.25
            neg = torch.log((1 + x * x) / 2 * ((1 + x) / 2) ** 2) - 2 * torch.atan(x) + math.pi / 2
            psi = torch.where(zl < 0, neg, -4.8 * zl)
            stop = live & ((us - old).abs() / torch.clamp(us.abs(), min=1e-3) < f32(1e-3))
            done = torch.where(stop, us, done)
            live = live & ~stop
            if not bool(live.any()):
                break
        return done

    def _scalar(self, c, beta, rho, stage):
        s, W, k0 = self.f[c], self.W, self.td
        sg = torch.cat([s[:1], s[:1], s, s[-1:], s[-1:]])
        kg = torch.cat([k0[:1], k0, k0[-1:]])
        fx = _kappa(self.U, _xm(s), s, _xp(s), _xp(_xp(s)))
        fy = _kappa(self.V, _ym(s), s, _yp(s), _yp(_yp(s)))
        fz = _kappa(W, sg[:-3], sg[1:-2], sg[2:-1], sg[3:])
        a = (_xm(fx) - fx) + (_ym(fy) - fy) + (fz[:-1] - fz[1:])
        a = a + (_xp(k0) + k0) * (_xp(s) - s) / 2 - (k0 + _xm(k0)) * (s - _xm(s)) / 2
        a = a + (_yp(k0) + k0) * (_yp(s) - s) / 2 - (k0 + _ym(k0)) * (s - _ym(s)) / 2
        a = a + (kg[2:] + k0) * (sg[3:-1] - s) / 2 - (k0 + kg[:-2]) * (s - sg[1:-3]) / 2
        for (i, j, k), q in self.sources.get(c, {}).items():
            a[k - 1, j - 1, i - 1] += q
        div = (self.U[0] - _xm(self.U[0])) + (self.V[0] - _ym(self.V[0])) + (W[1] - W[0])
        a[0] += (self.flux if c == "T" else 0.0) + div * s[0]
        new = s + beta * self.dt * a
        if stage:
            new = new + rho * self.dt * self.adv[c]
        self.adv[c] = a
        return new

    def _tendencies(self, nu):
        U, V, W, N = self._ghosts(self.U), self._ghosts(self.V), self.W, torch.cat([nu[:1], nu, nu[-1:]])
        u, v = self.U, self.V
        w, wb = W[1:], W[:-1]
        ut, ub, vt, vb = U[2:], U[:-2], V[2:], V[:-2]
        nt, nb = N[2:], N[:-2]
        fu, fv = self._walls()
        out = []
        # along x: the component u (across y and z), then v by exchange of x and y
        for (c, o, ct, cb, xp, xm, yp, ym, wall) in ((u, v, ut, ub, _xp, _xm, _yp, _ym, fu),
                                                    (v, u, vt, vb, _yp, _ym, _xp, _xm, fv)):
            ce, cw, cn, cs = xp(c), xm(c), yp(c), ym(c)
            oe, os_, ose = xp(o), ym(o), xp(ym(o))
            we, wbe = xp(w), xp(wb)
            a = -(((ce + c) ** 2 - (c + cw) ** 2) + ((cn + c) * (oe + o) - (c + cs) * (ose + os_)) +
                  ((ct + c) * (we + w) - (c + cb) * (wbe + wb))) / 4
            a = a - ((ce - cw) * c / 2 + (cn - cs) * (o + oe + os_ + ose) / 8 + (ct - cb) * (w + we + wb + wbe) / 8)
            a = a / 2
            ne, nn, nne, ns, nse = xp(nu), yp(nu), xp(yp(nu)), ym(nu), xp(ym(nu))
            a = a + ne * (ce - c) - nu * (c - cw)
            a = a + (nne + ne + nn + nu) * (cn - c) / 4 - (ne + nse + nu + ns) * (c - cs) / 4
            top = (xp(nt) + ne + nt + nu) * (ct - c) / 4
            bot = (ne + xp(nb) + nu + nb) * (c - cb) / 4
            bot[0] = wall  # the wall model's stress in the place of the ground's diffusive flux
            out.append(a + top - bot)
        w, wt, wb = W[1:-1], W[2:], W[:-2]
        n0, n1 = nu[:-1], nu[1:]
        u0, u1, v0, v1 = u[:-1], u[1:], v[:-1], v[1:]
        we, ww, wn, ws = _xp(w), _xm(w), _yp(w), _ym(w)
        a = -(((wt + w) ** 2 - (w + wb) ** 2) + ((wn + w) * (v1 + v0) - (w + ws) * (_ym(v0) + _ym(v1))) +
              ((we + w) * (u1 + u0) - (w + ww) * (_xm(u1) + _xm(u0)))) / 4
        ua, va = u0 + u1 + _xm(u0) + _xm(u1), v0 + v1 + _ym(v0) + _ym(v1)
        a = (a - ((we - ww) * ua / 8 + (wn - ws) * va / 8 + (wt - wb) * w / 2)) / 2
        if "T" in self.f:
            th = self.f["T"]
            a = a + GRAV / T_REF / 2 * (th[1:] + th[:-1]) - GRAV
        ns_ = n0 + n1
        a = a + (_xp(ns_) + ns_) * (we - w) / 4 - (ns_ + _xm(ns_)) * (w - ww) / 4
        a = a + (_yp(ns_) + ns_) * (wn - w) / 4 - (ns_ + _ym(ns_)) * (w - ws) / 4
        bot = n0 * (w - wb)
        bot[0] = 0  # at the ground: no normal stress of the wall model
        out.append(a + n1 * (wt - w) - bot)
        return out

    def step(self):
        if self.vdt:
            big = torch.maximum
            cfl = (big(self.U.abs(), _xm(self.U).abs()) + big(self.V.abs(), _ym(self.V).abs()) +
                   big(self.W[1:].abs(), self.W[:-1].abs())).max()
            self.dt = min(0.5 / float(cfl), 0.04)
        for stage in range(3):
            beta, rho, coef = RK_BETA[stage], RK_RHO[stage], 2 * RK_ALPHA[stage] * self.dt
            nu = self._viscosity()
            if "T" in self.f:
                self.td = (nu - NU) / 0.6 + self.kappa
            tend = self._tendencies(nu)
            new = {c: self._scalar(c, beta, rho, stage) for c in self.f}
            star = getattr(self, "star", None)
            p = self.P
            grads = (_xp(p) - p, _yp(p) - p, p[1:] - p[:-1])
            inc = [beta * self.dt * t + (rho * self.dt * star[q] if stage else 0) - coef * grads[q]
                   for q, t in enumerate(tend)]
            self.star = tend
            self.U, self.V = self.U + inc[0], self.V + inc[1]
            self.W = self.W.clone()
            self.W[1:-1] += inc[2]
            self.f = new
            self._project(coef)

    # the arrays a host reads back, ghosts included
    def _wrap(self, a, deep):
        a = torch.cat([a[..., -deep:], a, a[..., :deep]], -1)
        return torch.cat([a[..., -deep:, :], a, a[..., :deep, :]], -2)

    def host(self):
        out, (nx, ny, nz) = {}, self.n
        for c, a in (("U", self.U), ("V", self.V)):
            out[c] = self._wrap(torch.cat([-a[2:3], -a[1:2], -a[:1], a, a[-1:], a[-1:], a[-1:]]), 3)
        w = self.W
        out["W"] = self._wrap(torch.cat([-w[2:3], -w[1:2], w, -w[-2:-1], -w[-3:-2]]), 3)
        p = torch.zeros((nz + 4, ny + 4, nx + 4), device="cuda", dtype=torch.float64)
        a, z, y, x = self.P, slice(2, nz + 2), slice(2, ny + 2), slice(2, nx + 2)
        p[z, y, x] = a
        p[z, y, :2], p[z, y, -2:] = a[..., -2:], a[..., :2]
        p[z, :2, x], p[z, -2:, x] = a[:, -2:], a[:, :2]
        p[1, y, x], p[0, y, x] = a[2] - 3 * (a[1] - a[0]), a[1]
        p[-2, y, x], p[-1, y, x] = a[-3] - 3 * (a[-2] - a[-1]), a[-2]
        out["P"] = p
        for c, a in self.f.items():
            out[c] = self._wrap(torch.cat([a[:1]] * 3 + [a] + [a[-1:]] * 3), 3)
        return out


def _marched(nx, ny, nz, f, steps, flux=0.0, scalars=0, vdt=False):
    src = _source(nx, ny, nz)
    ch = _Channel(nx, ny, nz, f, flux, {"S1": {src: 1.0}} if scalars else {}, vdt)
    xy = xz = 0.0
    for _ in range(steps):
        ch.step()
        if scalars:
            w = ch.dt / 0.02 / steps if vdt else 1.0 / steps
            xy, xz = xy + w * ch.f["S1"][src[2] - 1], xz + w * ch.f["S1"][:, src[1] - 1]
    out = ch.host()
    if scalars:
        out.update(xy=xy, xz=xz)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "cubes":
        return None  # the immersed boundary's geometry pass has no short plain form
    if kind == "poisson":
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        phi = torch.zeros((nz + 4, ny + 4, nx + 4), dtype=torch.float64)
        phi[2:-2, 2:-2, 2:-2] = _Poisson(nx, ny, stretched_zw(nz, 0.5, 1.01)).solve(_poisson_rhs(case, seed)).cpu()
        return phi
    if kind == "batch":
        parts = []
        for d, (nx, ny, nz, us) in enumerate(_batch_sizes(case)):
            parts.append(_marched(nx, ny, nz, _interiors(nx, ny, nz, seed, d + 1, us), case["steps"]))
        return {c: torch.cat([p[c].reshape(-1) for p in parts]) for c in "UVWP"}
    f = _interiors(case["nx"], case["ny"], case["nz"], seed, theta="T" in _fields_of(case),
                   scalars=case.get("scalars", 0))
    return _marched(case["nx"], case["ny"], case["nz"], f, case.get("steps", 1), case.get("flux", 0.0),
                    case.get("scalars", 0), case.get("vdt", False))
