"""Workloads of the boundary-layer solver as its users run them.

A pass of a flow case is one leg of a run between two checkpoints: the state
goes up from pinned host arrays (the FP64 Fortran layout of the C ABI), the
solver advances a few tens of steps, and the new state comes down, through the
public calls a host program makes (`Solver.upload_state_async`, `advance`,
`download_state_async`, `sync`; `Ensemble.advance` for a set of boxes).  With
a recycled inflow the leg starts as a restart does, with the running means set
from the uploaded field.  The network case is one training leg of the learned
wall model.

`exact` restates the same leg in FP64 with plain torch operations from the
scheme's formulas (staggered second-order RHS, RK3, boundary pass, DCT/DFT/
tridiagonal Poisson solve, Smagorinsky and dynamic Smagorinsky viscosity, law
of the wall, Lund rescaling, statistics).
"""
import functools
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "boundary-layer-gpu_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import blgpu  # noqa: E402
from blgpu import cases as bl  # noqa: E402

DEV = "cuda:0"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _flow(kind, nx, ny, nz, precision, steps, lund=0, les=0, rk=3, stats=False):
    return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "precision": precision, "steps": steps, "lund": lund,
            "les": les, "rk": rk, "stats": stats}


def listed():
    def named(name, c):
        return dict(c, name=name)

    return [
        # laminar flat plate at the size of a quick validation run: a step is a chain of
        # small launches, so latency and launch counts decide; both precisions
        named("plate_fp64_128x64x32", _flow("plate", 128, 64, 32, "fp64", 30, stats=True)),
        named("plate_mixed_128x64x32", _flow("plate", 128, 64, 32, "mixed", 30)),
        # transition run: Blasius plate forced by temporal inflow modes (a long box with an x
        # transform of 1022 = 2 7 73), checked through its z-averaged statistics at the end
        named("modes_mixed_1024x129x128", _flow("modes", 1024, 129, 128, "mixed", 40, stats=True)),
        # the turbulent boundary layer the benchmark runs (RK3 at a CFL number, Lund inflow), in
        # the mixed form and in the bit-faithful FP64 form
        named("turbulent_mixed_814x257x193", _flow("turbulent", 814, 257, 193, "mixed", 60, lund=3)),
        named("turbulent_fp64_814x257x193", _flow("turbulent", 814, 257, 193, "fp64", 30, lund=3)),
        # smaller turbulent boxes with odd sizes (x lengths 299 = 13 23 and 385 = 5 7 11, prime z
        # lengths), as a grid-refinement study has them
        named("turbulent_fp64_301x98x75", _flow("turbulent", 301, 98, 75, "fp64", 30, lund=5)),
        named("turbulent_mixed_387x121x151", _flow("turbulent", 387, 121, 151, "mixed", 40)),
        # wall-modelled LES: constant-coefficient Smagorinsky with the law of the wall
        named("wmles_mixed_512x96x256", _flow("wmles", 512, 96, 256, "mixed", 30, les=1, stats=True)),
        # LES with the dynamic Smagorinsky model: coefficient averaged in z (FP64, a moderate
        # box) and pointwise (mixed, the size of the wall-modelled LES)
        named("dynamic_fp64_256x97x66", _flow("wmles", 256, 97, 66, "fp64", 12, les=2)),
        named("dynamic_mixed_512x96x256", _flow("wmles", 512, 96, 256, "mixed", 8, les=3)),
        # training-data ensemble: uneven boxes of about a million cells advanced together
        named("ensemble_mixed_16", {"kind": "ensemble", "boxes": 16, "ny": 65, "precision": "mixed", "steps": 20}),
        # a training leg of the wall-stress network on wall samples held on the device
        named("net_train_100000", {"kind": "net", "rows": 100000, "batch": 8192, "steps": 400}),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same kinds: box sides between those of the smallest and
    the largest listed case, any parity, at most the largest one's cells."""
    kind = rng.choice(["plate", "modes", "turbulent", "turbulent", "turbulent", "wmles", "dynamic", "ensemble", "net"])
    if kind == "net":
        return {"kind": "net", "rows": _log_int(rng, 20000, 250000), "batch": _log_int(rng, 1024, 16384),
                "steps": rng.randint(100, 400)}
    precision = rng.choice(["fp64", "mixed"])
    if kind == "ensemble":
        return {"kind": "ensemble", "boxes": rng.randint(4, 16), "ny": rng.randint(33, 65), "precision": precision,
                "steps": rng.randint(5, 20)}
    les = {"wmles": 1, "dynamic": rng.choice([2, 3])}.get(kind, 0)
    most = 6.0e6 if kind == "dynamic" else 1.3e7 if kind == "wmles" else 4.0e7
    while True:
        nx, ny, nz = _log_int(rng, 64, 1024), _log_int(rng, 32, 257), _log_int(rng, 20, 256)
        if nx * ny * nz <= most and nx >= 2 * nz // 3:
            break
    steps = rng.randint(4, 8) if kind == "dynamic" else rng.randint(10, 30)
    lund = rng.choice([0, 3, 5]) if kind == "turbulent" else 0
    return _flow("wmles" if kind == "dynamic" else kind, nx, ny, nz, precision, steps, lund=lund, les=les,
                 rk=rng.choice([3, 3, 3, 2]) if kind in ("plate", "turbulent") else 3,
                 stats=kind != "dynamic" and rng.random() < 0.3)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _lerp(a, dim, pos, wrap=False):
    """Linear interpolation of `a` along `dim` at fractional positions."""
    n = a.shape[dim]
    lo = torch.floor(pos)
    w = pos - lo
    i0 = lo.long()
    i1 = i0 + 1
    i0, i1 = (i0 % n, i1 % n) if wrap else (i0.clamp(0, n - 1), i1.clamp(0, n - 1))
    sh = [1] * a.dim()
    sh[dim] = -1
    w = w.reshape(sh)
    return a.index_select(dim, i0) * (1.0 - w) + a.index_select(dim, i1) * w


def _noise(seed, nx, ny, nz, coarse=4):
    """Three components of a smooth solenoidal random field on a coarse grid,
    periodic in z, unit rms, resampled to the staggered arrays' shapes
    [k][j][i]; the same field to rounding on the periodic planes k and k+nz-2."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    cz, cy, cx = max(6, (nz - 2) // coarse), max(8, (ny + 1) // coarse), max(8, nx // coarse)
    psi = torch.randn((3, 1, cz, cy, cx), generator=g, device=DEV, dtype=torch.float64)
    for _ in range(2):  # binomial smoothing
        for dim in (2, 3, 4):
            n = psi.shape[dim]
            if dim == 2:
                up, dn = torch.roll(psi, 1, 2), torch.roll(psi, -1, 2)
            else:
                up = torch.cat([psi.narrow(dim, 0, 1), psi.narrow(dim, 0, n - 1)], dim)
                dn = torch.cat([psi.narrow(dim, 1, n - 1), psi.narrow(dim, n - 1, 1)], dim)
            psi = 0.5 * psi + 0.25 * (up + dn)
    p = psi[:, 0]
    dx = lambda a: torch.gradient(a, dim=2)[0]
    dy = lambda a: torch.gradient(a, dim=1)[0]
    dz = lambda a: 0.5 * (torch.roll(a, -1, 0) - torch.roll(a, 1, 0))
    c = [dy(p[2]) - dz(p[1]), dz(p[0]) - dx(p[2]), dx(p[1]) - dy(p[0])]
    rms = torch.sqrt(sum((q * q).mean() for q in c) / 3.0)
    out = []
    for q, (n1, n2, n3) in zip(c, ((nx, ny + 1, nz + 1), (nx + 1, ny, nz + 1), (nx + 1, ny + 1, nz))):
        ar = lambda n: torch.arange(n, device=DEV, dtype=torch.float64)
        q = _lerp(q / rms, 2, ar(n1) * (cx - 1) / (n1 - 1))
        q = _lerp(q, 1, ar(n2) * (cy - 1) / (n2 - 1))
        out.append(_lerp(q, 0, ar(n3) * cz / (nz - 2), wrap=True))
    return out


@functools.lru_cache(None)
def _blasius():
    eta, f, df, _ = bl.blasius_table()
    return eta, f, df


@functools.lru_cache(None)
def _profile(retheta, loglaw):
    kw = dict(kappa=bl.KAPPA_WM, C=bl.reichardt_c(bl.KAPPA_WM, bl.B_WM)) if loglaw else {}
    nu, utau, _ = bl.turbulent_inflow_profile(retheta, **kw)
    return nu, utau, kw


def _box(kind, nx, ny, nz, seed, retheta=None):
    """Grid, boundary vectors, start field and run parameters of one box."""
    b = {"nx": nx, "ny": ny, "nz": nz}
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=DEV)
    if kind in ("plate", "modes"):
        # Blasius plate in displacement-thickness units (Re 500; 1000 for the forced one)
        re, lx, ly, lz, alpha = (500.0, 60.0, 6.0, 6.0, 1.5) if kind == "plate" else (1000.0, 400.0, 20.0, 40.0, 1.5)
        lx, lz = (lx * nx / 128, lz * nz / 32) if kind == "plate" else (lx * nx / 1024, lz * nz / 128)
        nu = 1.0 / re
        x0 = (1.0 / 1.7208) ** 2 / nu
        x, y, z = bl.uniform_faces(nx, lx, x0), bl.tanh_faces(ny, ly, alpha), bl.periodic_faces(nz, lz)
        eta, f, df = _blasius()
        bc = bl.blasius_boundary(x, y, nu, (eta, f, df))
        xg, yg = bl.centres_ghost(x), bl.centres_ghost(y)
        e = yg[:, None] * np.sqrt(1.0 / (2.0 * nu * x[None, :]))
        U2 = np.where(e < 0, -1.0, 1.0) * np.interp(np.abs(e), eta, df, right=1.0)
        e = y[:, None] * np.sqrt(1.0 / (2.0 * nu * xg[None, :]))
        V2 = np.interp(e, eta, eta * df - f) / np.sqrt(2.0 * xg[None, :] / nu)
        amp, dt = 2e-3, 0.2 * lx / nx
        u, v, w = _noise(seed, nx, ny, nz)
        env_c, env_f = t(np.tanh(yg / 0.5) * np.exp(-(yg / 3.0) ** 2)), t(np.tanh(y / 0.5) * np.exp(-(y / 3.0) ** 2))
        if kind == "modes":
            dt = min(dt, 2.0 * np.pi / 0.1 / 400)
            b["modes"] = _modes(y, lz)
    else:
        lnx = kind == "wmles"
        re = retheta or (2000.0 if lnx else 1100.0)
        nu, utau, kw = _profile(re, lnx)
        lx, ly, lz, alpha = ((nx * 0.125, 2.0, nz * 0.0625, 0.05) if lnx else
                             (nx * 100.0 / 814.0, 4.0, nz * 8.0 / 193.0, 2.0))
        x0 = (re / 0.036) ** 1.25 * nu
        x, y, z = bl.uniform_faces(nx, lx, x0), bl.tanh_faces(ny, ly, alpha), bl.periodic_faces(nz, lz)
        xg, yg = bl.centres_ghost(x), bl.centres_ghost(y)
        prof = bl.composite_profile(yg, 1.0, utau, nu, **kw)
        top = bl.turbulent_top(x, nu)
        if lnx:
            top = (top[0], np.zeros_like(top[1]), top[2])
        bc = (prof, np.zeros(ny), np.zeros(ny + 1)) + top
        U2 = np.repeat(prof[:, None], nx, axis=1)
        V2 = np.zeros((ny, nx + 1))
        amp = 0.05 if lnx else 0.10
        u, v, w = _noise(seed, nx, ny, nz)
        m = lambda yy: np.clip((1.5 - yy) / 0.3, 0.0, 1.0) * np.tanh(yy / 0.05)
        env_c, env_f = t(m(yg)), t(m(y))
        dt = 0.03 * min(1.0, 96.0 / ny) if lnx else 0.03
    dt = min(dt, 0.4 * min(np.diff(bl.centres_ghost(a)).min() for a in (x, y, z)) ** 2 / nu)
    U = t(U2)[None] + amp * env_c[None, :, None] * u
    V = t(V2)[None] + amp * env_f[None, :, None] * v
    W = amp * env_c[None, :, None] * w
    # the planes a saved state has on its boundaries: no-slip wall, top vectors
    U[:, 0], W[:, 0], V[:, 0] = -U[:, 1], -W[:, 1], 0.0
    U[:, -1], V[:, -1], W[:, -1] = t(bc[3]), t(bc[4]), t(bc[5])
    b.update(x=x, y=y, z=z, bc=bc, nu=nu, U=U, V=V, W=W, dt=dt)
    return b


def _modes(y, lz):
    """Temporal inflow modes as a mode file gives them: a two-dimensional wave
    and an oblique pair of frequency 0.1, shapes confined to the layer."""
    yg = bl.centres_ghost(y)
    s = lambda yy: np.tanh(np.maximum(yy, 0.0)) * np.exp(-(yy / 2.0) ** 2)
    amp = np.array([1e-3, 1e-4 * np.exp(0.7j), 1e-4 * np.exp(2.1j)])
    qu = (s(yg) * (1.0 + 0.5j * np.cos(yg)))[:, None, None] * amp[None, :, None]
    qv = (0.3j * s(y) * np.tanh(y))[:, None, None] * amp[None, :, None]
    qw = (s(yg))[:, None, None] * (np.array([0.0, 1.0, -1.0]) * amp)[None, :, None]
    return np.array([0.0, 1.0, -1.0]) * 2.0 * np.pi / lz, np.array([0.1]), qu, qv, qw


def _run_params(case, b):
    """The CFL entry of the run: a positive number (dt from compute_dt, held
    by the viscous limit) for the turbulent boxes, a fixed step elsewhere."""
    if case["kind"] in ("turbulent", "ensemble"):
        dmin = min(np.diff(bl.centres_ghost(b[a])).min() for a in "xyz")
        return min(0.5, b["dt"] * b["nu"] / dmin ** 2)
    return -2e-4 if case.get("les", 0) >= 2 else -b["dt"]


def _pinned(t):
    h = torch.empty(t.shape, dtype=torch.float64, pin_memory=True)
    h.copy_(t)
    return h.numpy().T  # Fortran order (i, j, k)


def _wall_row(b):
    yg = bl.centres_ghost(b["y"])
    return int(np.argmin(np.abs(yg[1:-1] - 0.1))) + 2


def _lund(case, b):
    return (case["lund"], max(2, case["nx"] // 10), 1.0, 10.0)


def _boxes(case, seed):
    if case["kind"] != "ensemble":
        return [_box(case["kind"], case["nx"], case["ny"], case["nz"], seed)]
    r = np.random.default_rng(17)  # the shapes belong to the case, the fields to the seed
    out = []
    for q in range(case["boxes"]):
        nx, nz, re = int(r.choice([128, 192, 256])), int(r.choice([64, 96])), float(r.choice([800.0, 1100.0, 1500.0]))
        out.append(_box("turbulent", nx, case["ny"], nz, seed * 131 + q, retheta=re))
    return out


def _net_data(case, seed):
    """Wall samples: (u, w, ln(h|u|/nu)/10, 100 h dp/dx) -> 1000 tau."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    n = case["rows"]
    r = torch.randn((n, 5), generator=g, device=DEV, dtype=torch.float64)
    u = 0.62 + 0.1 * r[:, 0]
    X = torch.stack([u, 0.06 * r[:, 1], torch.log((1400.0 * u.abs()).clamp_min(1.0)) / 10.0, 0.2 * r[:, 2]], 1)
    T = torch.stack([1.6 * u * u.abs() / 0.38 + 0.1 * r[:, 2] + 0.7 * r[:, 3], 0.06 * r[:, 1] * 2.0 + 0.3 * r[:, 4]], 1)
    return X.float().cpu().numpy(), T.float().cpu().numpy()


def prepare(case, seed):
    if case["kind"] == "net":
        net = blgpu.WallNet(seed=11)
        X, T = _net_data(case, seed)
        net.add_data(X, T)
        return {"case": case, "net": net, "params": net.params}
    prec = blgpu.FP64 if case["precision"] == "fp64" else blgpu.MIXED
    boxes = []
    for b in _boxes(case, seed):
        s = blgpu.Solver(b["nx"], b["ny"], b["nz"], b["nu"], _run_params(case, b), rk_scheme=case.get("rk", 3),
                         les_model=case.get("les", 0), precision=prec)
        s.set_grid(b["x"], b["y"], b["z"])
        s.set_boundary(*b["bc"])
        if "modes" in b:
            s.set_inflow_modes(*b["modes"])
        if s.cfg.cfl < 0:
            s.set_dt(-s.cfg.cfl)
        if case["kind"] == "wmles":
            s.set_wall_model(1, _wall_row(b))
        boxes.append({"s": s, "in": [_pinned(b[q]) for q in "UVW"],
                      "out": [_pinned(torch.zeros_like(b[q])) for q in "UVW"],
                      "lund": _lund(case, b) if case.get("lund") else None})
    st = {"case": case, "boxes": boxes}
    if case["kind"] == "ensemble":
        st["ens"] = blgpu.Ensemble([q["s"] for q in boxes])
    return st


# the z-means a run writes out, without those that a spanwise-symmetric flow
# leaves at zero, and in the mixed form without the pressure's (a laminar
# plate's pressure is a small residue of the box-scale one there: its mean
# differs by 6e-2 between FP32 and FP64 transforms)
def _stats(case):
    return ("Umean", "U2mean", "V2mean", "W2mean", "UVmean", "Cf") + (
        ("Pmean", "P2mean") if case["precision"] == "fp64" else ())



def run(state):
    case = state["case"]
    if case["kind"] == "net":
        net = state["net"]
        net.params = state["params"]
        loss = net.train(case["steps"], batch=case["batch"], lr=2e-3)
        return {"params": net.params, "loss": loss}
    for q in state["boxes"]:
        q["s"].upload_state_async(*q["in"])
        if q["lund"]:
            q["s"].set_rescaling(*q["lund"])
    if case["kind"] == "ensemble":
        state["ens"].advance(case["steps"])
        state["ens"].sync()
    else:
        state["boxes"][0]["s"].advance(case["steps"])
    for q in state["boxes"]:
        q["s"].download_state_async(*q["out"])
    out = {"fields": [q["out"] for q in state["boxes"]]}
    if case.get("stats"):
        s = state["boxes"][0]["s"].compute_statistics()
        out["stats"] = {k: s[k] for k in _stats(case)}
    for q in state["boxes"]:
        q["s"].sync()
    return out


# ---------------------------------------------------------------------------
# work and tolerances
# ---------------------------------------------------------------------------
def _shapes(case):
    if case["kind"] != "ensemble":
        return [(case["nx"], case["ny"], case["nz"])]
    r = np.random.default_rng(17)
    out = []
    for _ in range(case["boxes"]):
        nx, nz, _re = int(r.choice([128, 192, 256])), int(r.choice([64, 96])), float(r.choice([800.0, 1100.0, 1500.0]))
        out.append((nx, case["ny"], nz))
    return out


def work(case):
    """Element passes of the step: per substep RHS and RK update 9 (first) or
    12, projection 13 (divergence into the transforms 4, spectral solve 2,
    velocity correction 7), one pressure save a step; an eddy viscosity adds
    its evaluation (4) and its read by the RHS (1) a substep; the state goes
    up and comes down once in FP64."""
    if case["kind"] == "net":
        n = case["steps"] * min(case["batch"], case["rows"])
        return {"bytes": 28.0 * n + 4.0 * 8770 * 6 * case["steps"], "flops": 6.0 * 8640 * n}
    e = 8 if case["precision"] == "fp64" else 4
    subs = case.get("rk", 3)
    per = {3: 33, 2: 18}[subs] + 13 * subs + 1 + (5 * subs if case.get("les") else 0)
    bytes_, flops = 0.0, 0.0
    for nx, ny, nz in _shapes(case):
        c = float(nx) * ny * nz
        bytes_ += c * (per * e * case["steps"] + 6 * 8.0)
        point = 220.0 + 10.0 * math.log2(nx) + 10.0 * math.log2(nz) + 24.0 + (1200.0 if case.get("les", 0) >= 2 else 80.0 if case.get("les") else 0.0)
        flops += c * subs * case["steps"] * point
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """About four times the distance of the solver's forms from 64 bits after
    these steps.  FP64: 6e-11 (30 steps of the largest box, whose sums run in
    another order than the restatement's).  Mixed: u 3e-7, v 2e-6, w 1e-6 in
    the turbulent and LES boxes; v and w of the laminar plates, 1e-3 of u and
    carried by pressure differences, 1e-4.  The network trains with BF16
    operands: weights 1e-2 from FP64 ones after 400 steps."""
    if case["kind"] == "net":
        return {"rel": 1e-2, "max": 0.3}
    if case["precision"] == "fp64":
        return {"rel": 1e-9, "max": 1e-6}
    if case["kind"] in ("plate", "modes"):
        return {"rel": 5e-4, "max": 2e-2}
    return {"rel": 1e-5, "max": 2e-3}


# ---------------------------------------------------------------------------
# the same in 64 bits, by plain torch operations
# ---------------------------------------------------------------------------
class _Ref:
    """One box in FP64: arrays [k][j][i], index 0 = the Fortran index 1."""

    def __init__(self, b, cfl, rk, les, lund, wall_row):
        self.b, self.cfl, self.rk, self.les, self.jh = b, cfl, rk, les, wall_row
        self.nx, self.ny, self.nz = nx, ny, nz = b["nx"], b["ny"], b["nz"]
        self.nxg, self.nyg, self.nzg = nx + 1, ny + 1, nz + 1
        self.nu = b["nu"]
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=DEV)
        self.h = {a: b[a] for a in "xyz"}
        self.h.update({a + "g": bl.centres_ghost(b[a]) for a in "xyz"})
        self.c = {a: t(v) for a, v in self.h.items()}
        h = self.h
        self.F = {a: t(np.diff(h[a])) for a in "xyz"}         # F[n] = f(n+2) - f(n+1)
        self.C = {a: t(np.diff(h[a + "g"])) for a in "xyz"}   # C[n] = fg(n+2) - fg(n+1)
        w0 = (h["yg"][1:] - h["y"]) / np.diff(h["yg"])
        self.w0, self.w1 = t(w0), t(1.0 - w0)
        self.dmin = {a: np.diff(h[a + "g"]).min() for a in "xyz"}
        self.U, self.V, self.W = b["U"].clone(), b["V"].clone(), b["W"].clone()
        self.P = torch.zeros((self.nzg, self.nyg, self.nxg), device=DEV, dtype=torch.float64)
        self.nut = torch.zeros_like(self.P) if les else None
        self.bc = [t(a) for a in b["bc"]]
        self.t, self.dt = 0.0, abs(cfl)
        self._poisson_setup()
        self.lund = lund
        if lund:
            self.means = self._station_means()
        if wall_row:
            self.utau = t(np.sqrt(0.5 * 0.027 * (b["x"] / self.nu) ** (-1.0 / 7.0)))
        self.ax = None

    # -- metric helpers: values at the Fortran indices lo..hi of an axis -------
    def _v(self, a, lo, hi, dim):
        sh = [1, 1, 1]
        sh[2 - dim] = -1
        return a[lo:hi + 1].reshape(sh)

    def f(self, ax, lo, hi, d=0):  # face spacing f(n) - f(n-1)
        return self._v(self.F[ax], lo + d - 2, hi + d - 2, "xyz".index(ax))

    def g(self, ax, lo, hi, d=0):  # centre spacing fg(n+1) - fg(n)
        return self._v(self.C[ax], lo + d - 1, hi + d - 1, "xyz".index(ax))

    def w(self, q, lo, hi, d=0):
        return self._v(self.w1 if q else self.w0, lo + d - 1, hi + d - 1, 1)

    # -- right-hand sides -------------------------------------------------------
    def rhs(self):
        nx, ny, nz, nxg, nyg, nzg, nu = self.nx, self.ny, self.nz, self.nxg, self.nyg, self.nzg, self.nu

        def at(a, R):
            return lambda i=0, j=0, k=0: a[R[4] - 1 + k:R[5] + k, R[2] - 1 + j:R[3] + j, R[0] - 1 + i:R[1] + i]

        out = []
        # u on i = 2..nx-1, j = 2..nyg-1, k = 2..nzg-1
        R = (2, nx - 1, 2, nyg - 1, 2, nzg - 1)
        X, Y, Z = R[0:2], R[2:4], R[4:6]
        u, v, w = at(self.U, R), at(self.V, R), at(self.W, R)
        w0, w1, w0m, w1m = self.w(0, *Y), self.w(1, *Y), self.w(0, *Y, -1), self.w(1, *Y, -1)
        r = -((0.5 * (u() + u(1))) ** 2 - (0.5 * (u(-1) + u())) ** 2) / self.g("x", *X)
        r -= ((w0 * u() + w1 * u(0, 1)) * 0.5 * (v() + v(1)) -
              (w0m * u(0, -1) + w1m * u()) * 0.5 * (v(0, -1) + v(1, -1))) / self.f("y", *Y)
        r -= 0.25 * ((u() + u(0, 0, 1)) * (w() + w(1)) - (u(0, 0, -1) + u()) * (w(0, 0, -1) + w(1, 0, -1))) / self.f("z", *Z)
        if self.les:
            n = at(self.nut, R)
            nx1, nx2 = nu + n(), nu + n(1)
            ny1 = nu + 0.5 * (w0m * (n(0, -1) + n(1, -1)) + w1m * (n() + n(1)))
            ny2 = nu + 0.5 * (w0 * (n() + n(1)) + w1 * (n(0, 1) + n(1, 1)))
            nz1 = nu + 0.25 * (n() + n(0, 0, -1) + n(1) + n(1, 0, -1))
            nz2 = nu + 0.25 * (n() + n(0, 0, 1) + n(1) + n(1, 0, 1))
        else:
            nx1 = nx2 = ny1 = ny2 = nz1 = nz2 = nu
        r += (nx2 * (u(1) - u()) / self.f("x", *X, 1) - nx1 * (u() - u(-1)) / self.f("x", *X)) / self.g("x", *X)
        r += (ny2 * (u(0, 1) - u()) / self.g("y", *Y) - ny1 * (u() - u(0, -1)) / self.g("y", *Y, -1)) / self.f("y", *Y)
        r += (nz2 * (u(0, 0, 1) - u()) / self.g("z", *Z) - nz1 * (u() - u(0, 0, -1)) / self.g("z", *Z, -1)) / self.f("z", *Z)
        r[:, :, -1] = 0.0
        out.append(r)
        # v on i = 2..nxg-1, j = 2..ny-1, k = 2..nzg-1
        R = (2, nxg - 1, 2, ny - 1, 2, nzg - 1)
        X, Y, Z = R[0:2], R[2:4], R[4:6]
        u, v, w = at(self.U, R), at(self.V, R), at(self.W, R)
        w0, w1 = self.w(0, *Y), self.w(1, *Y)
        r = -((0.5 * (v() + v(0, 1))) ** 2 - (0.5 * (v(0, -1) + v())) ** 2) / self.g("y", *Y)
        r -= ((w0 * u() + w1 * u(0, 1)) * 0.5 * (v() + v(1)) -
              (w0 * u(-1) + w1 * u(-1, 1)) * 0.5 * (v(-1) + v())) / self.f("x", *X)
        r -= (0.5 * (v() + v(0, 0, 1)) * (w0 * w() + w1 * w(0, 1)) -
              0.5 * (v(0, 0, -1) + v()) * (w0 * w(0, 0, -1) + w1 * w(0, 1, -1))) / self.f("z", *Z)
        if self.les:
            n = at(self.nut, R)
            e = lambda i=0, k=0: w0 * n(i, 0, k) + w1 * n(i, 1, k)
            nx1, nx2 = nu + 0.5 * (e(-1) + e()), nu + 0.5 * (e() + e(1))
            ny1, ny2 = nu + n(), nu + n(0, 1)
            nz1, nz2 = nu + 0.5 * (e(0, -1) + e()), nu + 0.5 * (e() + e(0, 1))
        else:
            nx1 = nx2 = ny1 = ny2 = nz1 = nz2 = nu
        r += (nx2 * (v(1) - v()) / self.g("x", *X) - nx1 * (v() - v(-1)) / self.g("x", *X, -1)) / self.f("x", *X)
        r += (ny2 * (v(0, 1) - v()) / self.f("y", *Y, 1) - ny1 * (v() - v(0, -1)) / self.f("y", *Y)) / self.g("y", *Y)
        r += (nz2 * (v(0, 0, 1) - v()) / self.g("z", *Z) - nz1 * (v() - v(0, 0, -1)) / self.g("z", *Z, -1)) / self.f("z", *Z)
        r[:, :, -1] = 0.0
        out.append(r)
        # w on i = 2..nxg-1, j = 2..nyg-1, k = 2..nz-1
        R = (2, nxg - 1, 2, nyg - 1, 2, nz - 1)
        X, Y, Z = R[0:2], R[2:4], R[4:6]
        u, v, w = at(self.U, R), at(self.V, R), at(self.W, R)
        w0, w1, w0m, w1m = self.w(0, *Y), self.w(1, *Y), self.w(0, *Y, -1), self.w(1, *Y, -1)
        r = -((0.5 * (w() + w(0, 0, 1))) ** 2 - (0.5 * (w(0, 0, -1) + w())) ** 2) / self.g("z", *Z)
        r -= 0.25 * ((u() + u(0, 0, 1)) * (w() + w(1)) - (u(-1) + u(-1, 0, 1)) * (w(-1) + w())) / self.f("x", *X)
        r -= 0.5 * ((v() + v(0, 0, 1)) * (w0 * w() + w1 * w(0, 1)) -
                    (v(0, -1) + v(0, -1, 1)) * (w0m * w(0, -1) + w1m * w())) / self.f("y", *Y)
        if self.les:
            n = at(self.nut, R)
            m = lambda i=0, j=0: n(i, j) + n(i, j, 1)
            nx1, nx2 = nu + 0.25 * (m() + m(-1)), nu + 0.25 * (m() + m(1))
            ny1, ny2 = nu + 0.5 * (w0m * m(0, -1) + w1m * m()), nu + 0.5 * (w0 * m() + w1 * m(0, 1))
            nz1, nz2 = nu + n(), nu + n(0, 0, 1)
        else:
            nx1 = nx2 = ny1 = ny2 = nz1 = nz2 = nu
        r += (nx2 * (w(1) - w()) / self.g("x", *X) - nx1 * (w() - w(-1)) / self.g("x", *X, -1)) / self.f("x", *X)
        r += (ny2 * (w(0, 1) - w()) / self.g("y", *Y) - ny1 * (w() - w(0, -1)) / self.g("y", *Y, -1)) / self.f("y", *Y)
        r += (nz2 * (w(0, 0, 1) - w()) / self.f("z", *Z, 1) - nz1 * (w() - w(0, 0, -1)) / self.f("z", *Z)) / self.g("z", *Z)
        r[:, :, -1] = 0.0
        out.append(r)
        return out

    # -- boundary pass ----------------------------------------------------------
    def boundary(self, o, rkt):
        U, V, W = self.U, self.V, self.W
        Uo, Vo, Wo = o
        Ui, Vi, Wi, Ut, Vt, Wt = self.bc
        if self.lund and self.lund[0] == 3:
            U[:, :, 0], V[:, :, 0], W[:, :, 0] = self.lp
        elif self.lund:
            lu, lv, lw = self.lp
            U[:, :, 0], V[:, :, 0] = Ui + lu, Vi + lv
            ks = (torch.arange(1, self.nz + 1, device=DEV) + 16) % self.nz
            W[:, :, 0] = Wi + lw[ks]
        else:
            U[:, :, 0], V[:, :, 0], W[:, :, 0] = Ui, Vi, Wi
            if "modes" in self.b:
                zm, tm, qu, qv, qw = self.b["modes"]
                for q, a, z in ((qu, U, "zg"), (qv, V, "zg"), (qw, W, "z")):
                    for n, kz in enumerate(zm):
                        for m, om in enumerate(tm):
                            th = kz * self.c[z] - om * self.t
                            c = torch.as_tensor(q[:, n, m], device=DEV)
                            a[:, :, 0] += c.real * torch.cos(th)[:, None] - c.imag * torch.sin(th)[:, None]
        c = rkt * self.dt * float(Ut[-1])
        x, xg = self.h["x"], self.h["xg"]
        U[:, :, -2] = Uo[:, :, -2] - c * (Uo[:, :, -2] - Uo[:, :, -3]) / (x[-2] - x[-3])
        V[:, :, -2] = Vo[:, :, -2] - c * (Vo[:, :, -2] - Vo[:, :, -3]) / (xg[-2] - xg[-3])
        W[:, :, -2] = Wo[:, :, -2] - c * (Wo[:, :, -2] - Wo[:, :, -3]) / (xg[-2] - xg[-3])
        for a in (U, V, W):
            a[:, :, -1] = a[:, :, -2]
        for a in (U, V):
            a[0], a[-2], a[-1] = a[-3].clone(), a[1].clone(), a[2].clone()
        W[0], W[-1] = W[-2].clone(), W[1].clone()
        U[:, -1], V[:, -1], W[:, -1] = Ut, Vt, Wt
        if self.ax is None:
            U[:, 0] = -U[:, 1]
        else:
            k = torch.arange(1, self.nzg + 1, device=DEV)
            k = torch.where(k == 1, self.nzg - 2, torch.where(k == self.nzg - 1, 2, torch.where(k == self.nzg, 3, k)))
            i = torch.arange(1, self.nx + 1, device=DEV).clamp(2, self.nx - 1)
            U[:, 0] = U[:, 1] - self.ax[k - 2][:, i - 2] * (self.h["yg"][1] - self.h["yg"][0])
        W[:, 0], V[:, 0] = -W[:, 1], 0.0
        ks = slice(1, self.nzg - 2)
        Q = ((U[ks, 1:-1, 0] - U[ks, 1:-1, -2]) * self.F["y"]).sum()
        Q = Q + ((V[ks, 0, 1:-2] - V[ks, -1, 1:-2]) * self.F["x"][:self.nxg - 3]).sum()
        U[:, :, -2] += Q / float(self.F["y"].sum()) / (self.nzg - 3)
        U[:, :, -1] = U[:, :, -2]

    # -- projection -------------------------------------------------------------
    def _poisson_setup(self):
        N, M, NM = self.nx - 2, self.nz - 2, self.ny - 1
        ar = lambda n: torch.arange(n, device=DEV, dtype=torch.float64)
        kx = 2.0 * (torch.cos(math.pi * ar(N) / N) - 1.0) / self.dmin["x"] ** 2
        kz = 2.0 * (torch.cos(2.0 * math.pi * ar(M // 2 + 1) / M) - 1.0) / self.dmin["z"] ** 2
        y, yg = self.h["y"], self.h["yg"]
        dy = np.diff(y)
        up, lo = 1.0 / dy / (yg[2:] - yg[1:-1]), 1.0 / dy / (yg[1:-1] - yg[:-2])
        d = 1.0 / dy * (-1.0 / (yg[2:] - yg[1:-1]) - 1.0 / (yg[1:-1] - yg[:-2]))
        d[0] += lo[0]
        d[-1] += up[-1]
        self.up, self.lo = up, lo
        piv = torch.empty((NM, M // 2 + 1, N), device=DEV, dtype=torch.float64)
        p = d[0] + kx[None] + kz[:, None]
        p[0, 0] *= 1.5
        piv[0] = 1.0 / p
        for b in range(1, NM):
            piv[b] = 1.0 / (d[b] + kx[None] + kz[:, None] - lo[b] * up[b - 1] * piv[b - 1])
        self.piv = piv
        self.tw = torch.exp(-1j * math.pi * ar(N) / (2.0 * N))

    def project(self, save_p):
        N, M, NM = self.nx - 2, self.nz - 2, self.ny - 1
        U, V, W = self.U, self.V, self.W
        K = slice(1, M + 1)
        d = (U[K, 1:-1, 1:N + 1] - U[K, 1:-1, 0:N]) / self.F["x"][:N]
        d += (V[K, 1:, 1:N + 1] - V[K, :-1, 1:N + 1]) / self.F["y"][:, None]
        d += (W[1:M + 1, 1:-1, 1:N + 1] - W[0:M, 1:-1, 1:N + 1]) / self.F["z"][:M, None, None]
        e = torch.fft.rfft(torch.cat([d, d.flip(2)], 2), dim=2)[:, :, :N]
        e = (e * self.tw).real.contiguous()
        q = torch.fft.rfft(e, dim=0).permute(1, 0, 2).contiguous()  # [b][kz][kx]
        del d, e
        for b in range(1, NM):
            q[b] -= self.lo[b] * self.piv[b - 1] * q[b - 1]
        q[NM - 1] *= self.piv[NM - 1]
        for b in range(NM - 2, -1, -1):
            q[b] = (q[b] - self.up[b] * q[b + 1]) * self.piv[b]
        e = torch.fft.irfft(q.permute(1, 0, 2), n=M, dim=0)
        del q
        e = torch.cat([e * self.tw.conj(), torch.zeros((M, NM, 1), device=DEV, dtype=torch.complex128)], 2)
        p = torch.fft.irfft(e, n=2 * N, dim=2)[:, :, :N]
        del e
        p = torch.cat([p, p[:, :, -1:]], 2)   # i = 2..nxg-1
        p = torch.cat([p, p[:1]], 0)          # k = 2..nzg-1
        if save_p:
            self.P[1:-1, 1:-1, 1:-1] = p / (0.5 * self.dt)
            P = self.P
            P[:, :, 0], P[:, :, -1] = P[:, :, 1].clone(), P[:, :, -2].clone()
            P[:, 0], P[:, -1] = P[:, 1].clone(), P[:, -2].clone()
            P[0], P[-1] = P[1].clone(), P[-2].clone()
        U[1:-1, 1:-1, 1:-1] -= (p[:, :, 1:] - p[:, :, :-1]) / self.C["x"][1:-1]
        V[1:-1, 1:-1, 1:-1] -= (p[:, 1:] - p[:, :-1]) / self.C["y"][1:-1, None]
        W[1:-1, 1:-1, 1:-1] -= (p[1:] - p[:-1]) / self.C["z"][1:-1, None, None]

    # -- eddy viscosity ----------------------------------------------------------
    def _sij(self, U, V, W):
        nxg, nyg, nzg = self.nxg, self.nyg, self.nzg
        X, Y, Z = (2, nxg - 1), (2, nyg - 1), (2, nzg - 1)
        s = [(U[1:-1, 1:-1, 1:] - U[1:-1, 1:-1, :-1]) / self.f("x", *X),
             (V[1:-1, 1:, 1:-1] - V[1:-1, :-1, 1:-1]) / self.f("y", *Y),
             (W[1:, 1:-1, 1:-1] - W[:-1, 1:-1, 1:-1]) / self.f("z", *Z)]
        cx, cy, cz = self.C["x"], self.C["y"][:, None], self.C["z"][:, None, None]
        e = 0.5 * ((U[:, 1:] - U[:, :-1]) / cy + (V[:, :, 1:] - V[:, :, :-1]) / cx)[1:-1]
        s.append(0.25 * (e[:, :-1, :-1] + e[:, :-1, 1:] + e[:, 1:, :-1] + e[:, 1:, 1:]))
        e = 0.5 * ((U[1:] - U[:-1]) / cz + (W[:, :, 1:] - W[:, :, :-1]) / cx)[:, 1:-1]
        s.append(0.25 * (e[:-1, :, :-1] + e[:-1, :, 1:] + e[1:, :, :-1] + e[1:, :, 1:]))
        e = 0.5 * ((V[1:] - V[:-1]) / cz + (W[:, 1:] - W[:, :-1]) / cy)[:, :, 1:-1]
        s.append(0.25 * (e[:-1, :-1] + e[:-1, 1:] + e[1:, :-1] + e[1:, 1:]))
        S = torch.sqrt(sum((2.0 if c < 3 else 4.0) * q * q for c, q in enumerate(s)))
        return s, S

    def smagorinsky(self):
        dy = self.F["y"]
        cs2 = (0.11 * (self.dmin["x"] * self.dmin["z"] * dy) ** (1.0 / 3.0)) ** 2
        self.nut[1:-1, 1:-1, 1:-1] = cs2[:, None] * self._sij(self.U, self.V, self.W)[1]

    def dynamic(self):
        per, nzg = self.les == 3, self.nzg

        def ghosts(a, face=None, x=True, z=True):
            if x:
                if per and face != "x":
                    a[:, :, 0], a[:, :, -2], a[:, :, -1] = a[:, :, -3].clone(), a[:, :, 1].clone(), a[:, :, 2].clone()
                elif per:
                    a[:, :, 0], a[:, :, -1] = a[:, :, -2].clone(), a[:, :, 1].clone()
                else:
                    a[:, :, 0], a[:, :, -1] = a[:, :, 1].clone(), a[:, :, -2].clone()
            if z:
                if face == "z":
                    a[0], a[-1] = a[-2].clone(), a[1].clone()
                else:
                    a[0], a[-2], a[-1] = a[-3].clone(), a[1].clone(), a[2].clone()
            return a

        def filt(a):  # rows a[:, j] are the whole y section; x, z interior
            y = torch.empty_like(a)
            y[:, 1:-1] = a[:, :-2] / 6.0 + a[:, 1:-1] * (2.0 / 3.0) + a[:, 2:] / 6.0
            y[:, 0] = 2.0 / 3.0 * a[:, 0] + 1.0 / 3.0 * a[:, 1]
            y[:, -1] = 1.0 / 3.0 * a[:, -2] + 2.0 / 3.0 * a[:, -1]
            y = y[:-2] / 6.0 + y[1:-1] * (2.0 / 3.0) + y[2:] / 6.0
            return y[:, :, :-2] / 6.0 + y[:, :, 1:-1] * (2.0 / 3.0) + y[:, :, 2:] / 6.0

        U, V, W = self.U, self.V, self.W
        z3 = lambda: torch.zeros((self.nzg, self.nyg - 2, self.nxg), device=DEV, dtype=torch.float64)
        uc, vc, wc = z3(), z3(), z3()
        uc[:, :, 1:-1] = 0.5 * (U[:, 1:-1, :-1] + U[:, 1:-1, 1:])
        vc[:] = 0.5 * (V[:, :-1] + V[:, 1:])
        wc[1:-1] = 0.5 * (W[:-1, 1:-1] + W[1:, 1:-1])
        ghosts(uc, z=False)
        ghosts(wc, x=False)
        cen = (uc, vc, wc)
        pair = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))
        hat = [filt(q) for q in cen]
        L = []
        for p, q in pair:
            L.append(filt(ghosts(cen[p] * cen[q])) - hat[p] * hat[q])
        del hat, cen, uc, vc, wc
        full = []
        for a, face in ((U, "x"), (V, "y"), (W, "z")):
            q = torch.zeros_like(a)
            q[1:-1, :, 1:-1] = filt(a)
            full.append(ghosts(q, face))
        s, S = self._sij(*full)
        M = [4.0 * S * q for q in s]
        del full
        s, S = self._sij(U, V, W)
        for c in range(6):
            a = z3()
            a[1:-1, :, 1:-1] = S * s[c]
            M[c] -= filt(ghosts(a))
        ml = sum((1.0 if c < 3 else 2.0) * M[c] * L[c] for c in range(6))
        mm = sum((1.0 if c < 3 else 2.0) * M[c] * M[c] for c in range(6))
        n = z3()
        if self.les == 2:
            n[1:-1, :, 1:-1] = -0.5 * (ml[:nzg - 3].mean(0) / mm[:nzg - 3].mean(0)) * S
        else:
            n[1:-1, :, 1:-1] = -0.5 * (ml / mm) * S
            ghosts(n)
        self.nut[:, 1:-1] = torch.where(n > 0.0, n, torch.zeros_like(n))
        self.nut[:, 0], self.nut[:, -1] = self.nut[:, 1], self.nut[:, -2]

    # -- wall model, Lund inflow, dt ----------------------------------------------
    def wall_stress(self):
        kap, B, yr = 0.38, 5.2, float(self.h["yg"][self.jh - 1])
        um = self.U[1:-1, self.jh - 1, 1:-1].mean(0)
        q = self.utau[1:-1].clone()
        live = torch.ones_like(q, dtype=torch.bool)
        for _ in range(30):
            lg = torch.log(yr * q / self.nu)
            fx = q / kap * lg + B * q - um
            live &= fx.abs() >= 1e-10
            q = torch.where(live, q - fx / (lg / kap + 1.0 / kap + B), q)
        q = torch.where(torch.isnan(q), torch.zeros_like(q), q)
        self.utau[1:-1] = q
        n = self.nut[1:self.nzg - 2]
        e = float(self.w0[0]) * n[:, 0] + float(self.w1[0]) * n[:, 1]
        nuw = self.nu + 0.5 * (e[:, 1:self.nx - 1] + e[:, 2:self.nx])
        self.ax = q[None] ** 2 / nuw

    def _station_means(self):
        ir = self.lund[1] - 1
        return [self.U[1:-1, :, ir].mean(0), self.U[1:-1, :, 0].mean(0),
                self.V[1:-1, :, ir].mean(0), self.V[1:-1, :, 0].mean(0)]

    def rescale(self):
        mode, ir, delta, T = self.lund
        ir -= 1
        nu, yg, y = self.nu, self.c["yg"], self.c["y"]
        inst = self._station_means()
        uinf = float(inst[0][-1])
        a = self.dt / T
        self.means = [a * p + (1.0 - a) * q for p, q in zip(inst, self.means)]
        mu, mui, mv, _ = self.means

        def d99(m):
            m, h = m.cpu().numpy(), self.h["yg"]
            hit = np.nonzero(m >= 0.99 * uinf)[0]
            j = int(hit[0]) if hit.size and hit[0] >= 1 else self.nyg // 2 - 1
            c = (0.99 * uinf - m[j - 1]) / (m[j] - m[j - 1])
            return abs(c * h[j] + (1.0 - c) * h[j - 1])

        def theta(m):
            e = m / uinf * (1.0 - m / uinf)
            return abs(float((0.5 * (e[1:] + e[:-1]) * (yg[1:] - yg[:-1])).sum()))

        dr, tr, ti = d99(mu), theta(mu), theta(mui)
        uv = float((0.5 * (self.U[1:-1, 0, ir] + self.U[1:-1, 1, ir]) * self.V[1:-1, 0, ir]).mean())
        ur = math.sqrt(abs(nu * float(mu[1] - mu[0]) / float(yg[1] - yg[0]) - uv))
        ui = ur * (tr / ti) ** 0.125
        gam = ui / ur

        def interp(src, ys, yi):  # src [..., n]
            n = ys.numel()
            j = torch.searchsorted(ys.contiguous(), yi.contiguous(), right=True)
            jc = j.clamp(1, n - 1)
            c = (ys[jc] - yi) / (ys[jc] - ys[jc - 1])
            r = c * src[..., jc - 1] + (1.0 - c) * src[..., jc]
            r = torch.where(j >= n, src[..., -1:].expand_as(r), r)
            r[..., 0] = 0.0
            return r

        def weight(h):
            e, bb, al = h / delta, 0.2, 4.0
            return 0.5 * (1.0 + torch.tanh(al * (e - bb) / ((1.0 - 2.0 * bb) * e + bb)) / math.tanh(al))

        Wg, Wf = weight(yg), weight(y)
        um_i = gam * interp(mu, ur * yg / nu, ui * yg / nu)
        um_o = gam * interp(mu, yg / dr, yg / delta) + (1.0 - gam) * uinf
        vm_i, vm_o = interp(mv, ur * y / nu, ui * y / nu), interp(mv, y / dr, y / delta)
        if mode == 5:
            um_i, um_o, vm_i, vm_o = (0.0 * q for q in (um_i, um_o, vm_i, vm_o))
        fu, fv, fw = self.U[:, :, ir] - mu, self.V[:, :, ir] - mv, self.W[:, :, ir]
        both = lambda q, h: (gam * interp(q, ur * h / nu, ui * h / nu), gam * interp(q, h / dr, h / delta))
        i_, o_ = both(fu, yg)
        lu = (um_i + i_) * (1.0 - Wg) + (um_o + o_) * Wg
        i_, o_ = both(fv, y)
        lv = (vm_i + i_) * (1.0 - Wf) + (vm_o + o_) * Wf
        i_, o_ = both(fw, yg)
        self.lp = (lu, lv, i_ * (1.0 - Wg) + o_ * Wg)

    def compute_dt(self):
        if self.cfl < 0:
            self.dt = -self.cfl
            return
        lim = []
        for a, ax in ((self.U[1:-1, 1:-1, 1:], "x"), (self.V[1:-1, 1:, 1:-1], "y"), (self.W[1:, 1:-1, 1:-1], "z")):
            dim = 2 - "xyz".index(ax)
            m = a.abs().amin(dim=[q for q in range(3) if q != dim])
            lim.append(self.cfl * float((self.C[ax][1:] / m).max()))
        vis = min(self.cfl * self.dmin[a] ** 2 / self.nu for a in "xyz")
        self.dt = min(min(lim), vis)

    def step(self):
        self.compute_dt()
        o = [self.U.clone(), self.V.clone(), self.W.clone()]
        to, dt = self.t, self.dt
        if self.lund:
            self.rescale()
        coef = {3: ((8.0 / 15.0, 0.0), (0.25, 5.0 / 12.0), (0.25, 0.75)), 2: ((0.5, 0.0), (0.0, 1.0))}[self.rk]
        tt = {3: (8.0 / 15.0, 2.0 / 3.0, 1.0), 2: (0.5, 1.0)}[self.rk]
        rkt = (8.0 / 15.0, 2.0 / 3.0, 1.0)
        first = None
        for s, (c1, c2) in enumerate(coef):
            if self.les == 1:
                self.smagorinsky()
            elif self.les:
                self.dynamic()
            if self.jh:
                self.wall_stress()
            r = self.rhs()
            if s == 0:
                first = r
            for a, b, q1, q2 in zip((self.U, self.V, self.W), o, first, r):
                inc = dt * c1 * q1 if s == 0 else dt * (c1 * q1 + c2 * q2)
                a[1:-1, 1:-1, 1:-1] = b[1:-1, 1:-1, 1:-1] + inc
            del r
            self.t = to + tt[s] * dt
            self.boundary(o, rkt[s])
            self.project(s == 0)
            self.boundary(o, rkt[s])

    def statistics(self):
        nx, ny = self.nx, self.ny
        K, w0, w1 = slice(1, self.nzg - 1), self.w0[:, None], self.w1[:, None]
        t1 = w0 * self.U[K, :-1] + w1 * self.U[K, 1:]
        t2 = 0.5 * (self.V[K, :, :-1] + self.V[K, :, 1:])
        wi = 0.5 * (self.W[:self.nz - 2, :, :-1] + self.W[:self.nz - 2, :, 1:])
        t3 = w0 * wi[:, :-1] + w1 * wi[:, 1:]
        P = self.P[K, :ny, :nx]
        out = {"Umean": t1.mean(0), "U2mean": (t1 * t1).mean(0), "V2mean": (t2 * t2).mean(0),
               "W2mean": (t3 * t3).mean(0), "UVmean": (t1 * t2).mean(0), "Pmean": P.mean(0), "P2mean": (P * P).mean(0)}
        du = (self.U[K, 1].mean(0) - self.U[K, 0].mean(0)) / float(self.C["y"][0])
        tau = 0.0
        if self.les:
            n = torch.zeros((self.nyg, self.nxg), device=DEV, dtype=torch.float64)
            n[:ny, :nx] = self.nut[K, :ny, :nx].mean(0)
            tau = 0.25 * (n[0, :-1] + n[1, :-1] + n[0, 1:] + n[1, 1:]) * du
        out["Cf"] = 2.0 * (-out["UVmean"][0] + self.nu * du + tau)
        return {k: v.cpu().numpy().T for k, v in out.items()}


def _exact_net(case, seed):
    X, T = (torch.as_tensor(a, device=DEV, dtype=torch.float64) for a in _net_data(case, seed))
    net = blgpu.WallNet(seed=11)  # the initial weights
    p = torch.as_tensor(net.params, device=DEV, dtype=torch.float64)
    net.close()
    # the training order: a Fisher-Yates shuffle driven by the splitmix64 generator
    n, mask = case["rows"], (1 << 64) - 1
    s = 11 ^ 0xA5A5A5A5
    order = list(range(n))
    for r in range(n - 1, 0, -1):
        s = (s + 0x9E3779B97F4A7C15) & mask
        z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        q = (z ^ (z >> 31)) % (r + 1)
        order[r], order[q] = order[q], order[r]
    order = torch.as_tensor(order, device=DEV)
    B = min(case["batch"], n)
    p.requires_grad_(True)
    m1, m2, loss = torch.zeros_like(p), torch.zeros_like(p), None
    for t in range(1, case["steps"] + 1):
        at = order[(torch.arange(B, device=DEV) + (t - 1) * B) % n]
        h, o = X[at], 0
        for a, b in ((4, 64), (64, 64), (64, 64), (64, 2)):
            w, o = p[o:o + a * b].reshape(b, a), o + a * b
            h = h @ w.T + p[o:o + b]
            o += b
            if b == 64:
                h = torch.nn.functional.gelu(h)
        loss = ((h - T[at]) ** 2).sum() / B
        g, = torch.autograd.grad(loss, p)
        with torch.no_grad():
            m1 = 0.9 * m1 + 0.1 * g
            m2 = 0.999 * m2 + 0.001 * g * g
            p -= 2e-3 * (m1 / (1.0 - 0.9 ** t)) / (torch.sqrt(m2 / (1.0 - 0.999 ** t)) + 1e-8)
    return {"params": p.detach().cpu().numpy(), "loss": float(loss)}


def exact(case, seed):
    if case["kind"] == "net":
        return _exact_net(case, seed)
    fields, stats = [], None
    for b in _boxes(case, seed):
        r = _Ref(b, _run_params(case, b), case.get("rk", 3), case.get("les", 0), _lund(case, b) if case.get("lund") else None,
                 _wall_row(b) if case["kind"] == "wmles" else 0)
        for _ in range(case["steps"]):
            r.step()
        fields.append([a.cpu().numpy().T for a in (r.U, r.V, r.W)])
        if case.get("stats"):
            stats = {k: v for k, v in r.statistics().items() if k in _stats(case)}
        del r
    return {"fields": fields, "stats": stats} if case.get("stats") else {"fields": fields}
