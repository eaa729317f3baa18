"""Timed cases of the timestep library: what a user's program has it do, through its entry points.

A case is one of three kinds of pass:

* ``run``: a solver that holds a flow advances ``steps`` timesteps and hands the fields back to the
  program's (pinned) host arrays, as a time loop does between two field dumps.  ``calls`` says
  whether the program calls the library once per step (a host that looks at the CFL number of
  every step, as the reference's time loop does) or once per interval.  With ``upload`` each pass
  starts from the program's own initial fields (a sweep over short runs).
* ``ensemble``: many independent boxes advanced together, then every box's fields come back.
* ``analysis``: the diagnostics, the energy spectrum and the droplet statistics of a flow.

Sizes are the library's grid sizes (16 to 1024 points per axis, 192 among them; boxes need not be
cubes).  The flows are the usual ones of this code: a seeded solenoidal velocity of unit rms with
large-scale ABC forcing, drops of radius 0.3 at seeded centres with the interface one cell wide,
tracers at seeded uniform positions.
"""
import ctypes
import math

import numpy as np
import torch

from mhit36_mixedp_b200 import Ensemble, Params, Solver
from mhit36_mixedp_b200 import api

LX = 8.0 * math.atan(1.0)
TINY = 1.0e-16
AXES = (16, 32, 64, 128, 192, 256, 512, 1024)
ENSEMBLE_32 = "64x16,128x10,192x6"


def _case(name=None, kind="run", nx=64, ny=0, nz=0, steps=1, calls="each", upload=False, phi=False, drops=0, tracers=0,
          interp="linear1d", poisson="fp64", laplacian="exact", dt=2e-4, nu=0.003, boxes=""):
    c = dict(kind=kind, nx=nx, ny=ny or nx, nz=nz or nx, steps=steps, calls=calls, upload=upload, phi=phi, drops=drops,
             tracers=tracers, interp=interp, poisson=poisson, laplacian=laplacian, dt=dt, nu=nu, boxes=boxes)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest configuration: 64^3 single-phase, the host looks at every step
        _case("ns_64_fp64", nx=64, steps=100, dt=5e-4, nu=0.006),
        # the reference's validation size, single phase, one call per output interval
        _case("ns_128_fp64", nx=128, steps=100, calls="bulk", dt=2e-4, nu=6.25e-4),
        # a sweep of short multiphase runs, each from its own initial fields
        _case("sweep_128_fp32", nx=128, steps=20, upload=True, phi=True, drops=64, poisson="fp32"),
        # a box that is no cube, with drops and tracers
        _case("slab_192x64x128", nx=192, ny=64, nz=128, steps=50, phi=True, drops=16, tracers=100_000),
        # the multiphase production size of a study, FP64 and FP32 pressure solves of the reference
        _case("acdi_256_fp64", nx=256, steps=60, phi=True, drops=64),
        _case("acdi_256_fp32", nx=256, steps=60, calls="bulk", phi=True, drops=64, poisson="fp32"),
        # the headline pair: 512^3 multiphase at matched divergence, FP64 and mixed precision
        _case("acdi_512_fp64", nx=512, steps=40, phi=True, drops=256, dt=1e-4, laplacian="modified"),
        _case("acdi_512_mixed", nx=512, steps=40, phi=True, drops=256, dt=1e-4, laplacian="modified",
              poisson="fp32_incremental"),
        # 512^3 multiphase with a million tracers, the reference's FP32 solve
        _case("tracers_512_fp32", nx=512, steps=40, phi=True, drops=256, tracers=1_000_000, interp="trilinear",
              dt=1e-4, poisson="fp32"),
        # single phase at 1024 points along x, the large-grid transforms
        _case("ns_1024x512x256", nx=1024, ny=512, nz=256, steps=40, calls="bulk", poisson="fp32", dt=5e-5, nu=8e-4),
        # 32 boxes of uneven sizes advanced together
        _case("ensemble_32", kind="ensemble", steps=40, calls="bulk", phi=True, drops=64, poisson="fp32",
              boxes=ENSEMBLE_32),
        # what is looked at when a field is dumped
        _case("analysis_512", kind="analysis", nx=512, steps=2, dt=1e-4, phi=True, drops=256),
    ]


def _stable_dt(nx):
    """The explicit diffusion of the phase field (gamma = max|u|, about 5) bounds dt by dx / (12 gamma)."""
    return 2e-4 * min(1.0, 256 / nx)


def draw(rng):
    kind = rng.choice(["run"] * 6 + ["ensemble", "analysis"])
    poisson = rng.choice(["fp64", "fp64", "fp32", "fp32", "fp32_incremental", "fp32_refined"])
    lap = "modified" if poisson in ("fp32_incremental", "fp32_refined") else rng.choice(["exact", "modified"])
    nu = rng.choice([8e-4, 0.003, 0.006])
    if kind == "ensemble":
        groups = [(n, rng.randint(1, 8)) for n in rng.sample([32, 64, 128, 192], rng.randint(2, 3))]
        return _case(kind=kind, steps=rng.randint(10, 40), calls="bulk", phi=True, drops=rng.randint(8, 64), nu=nu,
                     poisson=rng.choice(["fp32", "fp64"]), boxes=",".join("%dx%d" % g for g in groups))
    while True:
        # cubes as often as boxes; the cell count is what spreads the cost
        n = rng.choice(AXES)
        dims = (n, n, n) if rng.random() < 0.4 else (n, rng.choice(AXES), rng.choice(AXES))
        cells = dims[0] * dims[1] * dims[2]
        if cells <= 1 << 27 and max(dims) <= 16 * min(dims):
            break
    nx, ny, nz = dims
    dt = _stable_dt(nx)
    phi = kind == "analysis" or rng.random() < 0.6
    drops = rng.randint(1, 64) if phi else 0
    if kind == "analysis":
        # the exact divide's divergence is a value (of order dx^2); the discrete one's is round-off
        return _case(kind=kind, nx=nx, ny=ny, nz=nz, steps=rng.randint(1, 4), phi=True, drops=drops, nu=nu, dt=dt)
    tracers = rng.choice([0, 0, int(10 ** rng.uniform(3, 6))])
    most = max(5, min(100, (30 << 27) // cells))
    return _case(nx=nx, ny=ny, nz=nz, steps=rng.randint(max(4, most // 3), most), calls=rng.choice(["each", "bulk"]),
                 upload=cells <= 1 << 21 and rng.random() < 0.25, phi=phi, drops=drops, tracers=tracers,
                 interp=rng.choice(["linear1d", "trilinear"]), poisson=poisson, laplacian=lap, dt=dt, nu=nu)


def _boxes(case):
    """The grids of a case: one for a run, those of "SIZExCOUNT,..." for an ensemble."""
    if case["kind"] != "ensemble":
        return [(case["nx"], case["ny"], case["nz"])]
    return [(int(n),) * 3 for g in case["boxes"].split(",") for n, k in [g.split("x")] for _ in range(int(k))]


def work(case):
    """Bytes: every step reads and writes the state it advances once (velocity and its right-hand
    side, phase field and its own, the tracers' positions and histories).  Operations: the stencils
    and the two transforms of the pressure solve."""
    cells = sum(a * b * c for a, b, c in _boxes(case))
    if case["kind"] == "analysis":
        return {"bytes": 4 * 8 * cells, "flops": cells * (3 * 2.5 * math.log2(cells) + 60)}
    per = 96 + (32 if case["phi"] else 0)
    out = 8 * (5 if case["phi"] else 4)
    flops = 5.0 * math.log2(cells) + 150 + (170 if case["phi"] else 0)
    return {"bytes": case["steps"] * (per * cells + 15 * 8 * case["tracers"]) + out * cells,
            "flops": case["steps"] * (flops * cells + 100 * case["tracers"])}


# ------------------------------------------------------------------------------------ inputs
def _velocity(shape, seed):
    """Seeded solenoidal velocity: Gaussian Fourier modes 0 < |m| <= 4, unit rms per component, on
    the staggered faces of a box of cubic cells."""
    nx, ny, nz = shape
    rng = np.random.default_rng(seed)
    m = np.arange(-4, 5)
    mz, my, mx = np.meshgrid(m, m, m, indexing="ij")
    m2 = mx ** 2 + my ** 2 + mz ** 2
    on = (m2 > 0) & (m2 <= 16)
    amp = (rng.standard_normal((3,) + on.shape) + 1j * rng.standard_normal((3,) + on.shape)) * on
    kv = np.stack([mx * 1.0, my * (nx / ny), mz * (nx / nz)])
    amp = amp - kv * ((kv * amp).sum(0) / np.where(on, (kv * kv).sum(0), 1.0))
    out = []
    for comp in range(3):
        e = []
        for axis, n in enumerate(shape):
            x = (np.arange(n) + (axis > 0) - 0.5 * (axis == comp)) * (2.0 * math.pi / n)
            e.append(torch.from_numpy(np.exp(1j * np.outer(x, m))).cuda())
        a = torch.from_numpy(amp[comp]).cuda() @ e[0].T             # (mz, my, x)
        b = torch.einsum("jq,zqi->zji", e[1], a).reshape(9, ny * nx)
        f = e[2].real @ b.real - e[2].imag @ b.imag
        out.append(f.mul_(1.0 / f.square().mean().sqrt()).reshape(nz, ny, nx))
    return out


def _radius(shape):
    """0.3 in the cube, at most 12 cells (what the interface of one cell resolves), less in a thin box."""
    return 0.3 * min(min(shape), 256) / shape[0]


def _drops(shape, count, seed):
    """Phase field of `count` drops at seeded centres that keep clear of each other: sites of a lattice,
    moved by up to a quarter of the gap (nearest centre by minimum image)."""
    nx, ny, nz = shape
    dx = LX / nx
    rng = np.random.default_rng(seed)
    per = [n * dx for n in shape]
    radius = _radius(shape)
    m = math.ceil(round(count ** (1 / 3), 9))
    sites = np.stack(np.unravel_index(rng.permutation(m ** 3)[:count], (m, m, m)), axis=1)
    gap = np.maximum(np.array(per) / m - 2.0 * radius, 0.0)
    centres = sites * (np.array(per) / m) + rng.uniform(-0.25, 0.25, size=(count, 3)) * gap
    near = torch.full((nz, ny, nx), 1e30, dtype=torch.float64, device="cuda")
    for c in centres:
        d2 = []
        for axis, n in enumerate(shape):
            d = (np.arange(n) + (axis > 0)) * dx - c[axis]
            d2.append(torch.from_numpy((d - per[axis] * np.round(d / per[axis])) ** 2).cuda())
        torch.minimum(near, (d2[2][:, None, None] + d2[1][None, :, None]) + d2[0][None, None, :], out=near)
    near = near.sqrt_().sub_(radius).div_(2.0 * dx).clamp_(max=20.0)
    return near.tanh_().mul_(-0.5).add_(0.5), radius


def _tracers(shape, count, seed):
    """Tracer table (count, 12): tags and uniform positions, no velocity or history yet."""
    rng = np.random.default_rng(seed)
    part = np.zeros((count, 12), order="F")
    part[:, 0] = np.arange(1, count + 1)
    part[:, 1:4] = rng.uniform(0.0, 1.0, size=(count, 3)) * [n * (LX / shape[0]) for n in shape]
    return part


def _inputs(case, shape, seed):
    u, v, w = _velocity(shape, seed)
    phi, radius = _drops(shape, case["drops"], seed + 1) if case["phi"] else (None, 0.3)
    part = _tracers(shape, case["tracers"], seed + 2) if case["tracers"] else None
    return u, v, w, phi, part, radius


def _params(case, shape, radius):
    # Weber number 1: sigma = rho u_rms^2 2R
    return Params(nx=shape[0], ny=shape[1], nz=shape[2], dt=case["dt"], mu=case["nu"], rho=1.0, radius=radius,
                  sigma=2.0 * radius, phiflag=int(case["phi"]), partflag=int(case["tracers"] > 0), npart=case["tracers"],
                  poisson=case["poisson"], laplacian=case["laplacian"], interp=case["interp"], acdi_clamp=1)


def _pinned(n):
    return torch.empty(n, dtype=torch.float64, pin_memory=True).numpy()


def _names(case):
    return ("u", "v", "w", "p", "phi") if case["phi"] else ("u", "v", "w", "p")


def prepare(case, seed):
    """The solver (or ensemble) holding the seeded flow, and the host arrays the fields come back to."""
    shapes = _boxes(case)
    cells = [a * b * c for a, b, c in shapes]
    whole = {f: _pinned(sum(cells)) for f in _names(case)}
    outs, at = [], 0
    for (nx, ny, nz), n in zip(shapes, cells):
        outs.append({f: a[at:at + n].reshape(nz, ny, nx) for f, a in whole.items()})
        at += n
    radii = [_radius(s) for s in shapes]
    params = [_params(case, s, r) for s, r in zip(shapes, radii)]
    state = {"case": case, "whole": whole, "outs": outs}
    if case["kind"] == "ensemble":
        state["ens"] = Ensemble(params)
        state["ens"].autotune()
        state["solvers"] = state["ens"].boxes
    else:
        state["solvers"] = [Solver(params[0])]
    for b, (shape, s, out) in enumerate(zip(shapes, state["solvers"], outs)):
        u, v, w, phi, part, _ = _inputs(case, shape, 1000 * seed + 7 * b)
        fields = [u, v, w] + ([phi] if case["phi"] else [])
        host = [out[f] for f in ("u", "v", "w", "phi") if f in out]
        if case["upload"]:
            host = [_pinned(u.numel()).reshape(u.shape) for _ in fields]
            state["start"] = host
        for h, d in zip(host, fields):
            torch.from_numpy(h).copy_(d)
        s.upload(*host)
        if part is not None:
            s.upload_particles(part)
            state["start_part"] = part
    if case["kind"] == "analysis":
        state["solvers"][0].step(case["steps"])
    return state


def _download(s, out):
    ptr = [api._dptr(out[f]) if f in out else None for f in ("u", "v", "w", "p", "phi")]
    api._check(s._lib.mhit_download_fields(s._ctx, *ptr))


def run(state):
    case = state["case"]
    s = state["solvers"][0]
    if case["kind"] == "analysis":
        d = s.diagnostics()
        e = s.energy_spectrum()
        found = s.label_drops(0.5, 6)
        # the program's own drop table has a row for each drop that there may be
        table = np.zeros((2 * case["drops"], 7))
        cells = np.zeros(2 * case["drops"], dtype=np.int64)
        n = min(len(found["cells"]), len(cells))
        cells[:n] = found["cells"][:n]
        for q, f in enumerate(("volume", "x", "y", "z", "u", "v", "w")):
            table[:n, q] = found[f][:n]
        return {"gumax": d["gumax"], "cfl": d["cfl"], "maxdiv": d["maxdiv"], "ke": d["ke"],
                "dissipation": d["dissipation"], "spectrum": e, "cells": cells, "drops": table}
    if case["upload"]:
        s.upload(*state["start"])
        if case["tracers"]:
            s.upload_particles(state["start_part"])
    mover = state.get("ens", s)
    if case["calls"] == "each":
        for _ in range(case["steps"]):
            mover.step(1)
    else:
        mover.step(case["steps"])
    for box, out in zip(state["solvers"], state["outs"]):
        _download(box, out)
    got = dict(state["whole"])
    if case["tracers"]:
        got["part"] = s.download_particles()
    return got


# ------------------------------------------------------------------------------------ 64-bit values
def _xp(a): return torch.roll(a, -1, 2)
def _xm(a): return torch.roll(a, 1, 2)
def _yp(a): return torch.roll(a, -1, 1)
def _ym(a): return torch.roll(a, 1, 1)
def _zp(a): return torch.roll(a, -1, 0)
def _zm(a): return torch.roll(a, 1, 0)


def _col(values, axis):
    t = torch.tensor(values, dtype=torch.float64, device="cuda")
    return t.reshape([-1 if axis == d else 1 for d in (2, 1, 0)])


def _solve(rhs, shape, laplacian):
    """Pressure of lap(p) = rhs by FFT, exact or 7-point symbol, zero mean."""
    nx, ny, nz = shape
    ddxi = (nx / LX) ** 2
    k2 = 0.0
    for axis, n in enumerate(shape):
        k = np.fft.fftfreq(n, 1.0 / n) if axis else np.arange(n // 2 + 1, dtype=np.float64)
        k2 = k2 + _col((2.0 - 2.0 * np.cos(k * (LX / n))) * ddxi if laplacian == "modified" else (k * nx / n) ** 2, axis)
    hat = torch.fft.rfftn(rhs)
    k2[0, 0, 0] = 1.0
    hat.div_(k2).neg_()
    hat[0, 0, 0] = 0.0
    return torch.fft.irfftn(hat, s=rhs.shape)


def _interpolate(f, pos, offsets, shape, dx, axes):
    """f at pos by linear interpolation along `axes` (the left node along the others)."""
    idx, frac = [], []
    for a in range(3):
        q = pos[a] / dx - offsets[a]
        fl = torch.floor(q)
        idx.append((fl.long(), shape[a]))
        frac.append(q - fl)
    total = 0.0
    for corner in range(8):
        up = [(corner >> a) & 1 for a in range(3)]
        if any(up[a] and a not in axes for a in range(3)):
            continue
        i, j, k = [torch.remainder(idx[a][0] + up[a], idx[a][1]) for a in range(3)]
        wgt = 1.0
        for a in axes:
            wgt = wgt * (frac[a] if up[a] else 1.0 - frac[a])
        total = total + wgt * f[k, j, i]
    return total


def _advance(case, shape, seed, steps):
    """The fields after `steps` timesteps from the seeded flow, in 64 bits throughout."""
    u, v, w, phi, part, radius = _inputs(case, shape, seed)
    nx, ny, nz = shape
    dx = LX / nx
    dxi, ddxi, eps, sigma, mu, dt = 1.0 / dx, 1.0 / dx / dx, dx, 2.0 * radius, case["nu"], case["dt"]
    tab = []
    for axis, n in enumerate(shape):
        x = np.arange(n) * dx + (dx if axis else 0.0)
        tab += [_col(np.sin(2.0 * x + dx / 2), axis), _col(np.cos(2.0 * x + dx / 2), axis)]
    sx, cx, sy, cy, sz, cz = tab
    ro = [None, None, None]
    rphi = None
    if part is not None:
        part = torch.from_numpy(np.ascontiguousarray(part.T)).cuda()
    gumax, al, be, p = 1.0, 1.0, 0.0, None
    for _ in range(steps):
        if part is not None:
            pos = [part[1], part[2], part[3]]
            if case["interp"] == "trilinear":
                vel = [_interpolate(f, pos, [(a > 0) - 0.5 * (a == c) for a in range(3)], shape, dx, (0, 1, 2))
                       for c, f in enumerate((u, v, w))]
            else:
                vel = [_interpolate(f, pos, (0, 1, 1), shape, dx, (c,)) for c, f in enumerate((u, v, w))]
            for c in range(3):
                q = part[1 + c] + dt * (al * vel[c] - be * part[8 + c])
                part[1 + c] = q - LX * torch.floor(q / LX)
                part[4 + c] = vel[c]
                part[8 + c] = vel[c]
        if phi is not None:
            c = phi.clamp(0.0, 1.0)
            psi = eps * torch.log((c + TINY) / (1.0 - c + TINY))
            t = torch.tanh(0.5 * psi / eps)
            n = [_xp(psi) - _xm(psi), _yp(psi) - _ym(psi), _zp(psi) - _zm(psi)]
            del psi
            g = 0.25 * (1.0 - t * t) / (torch.sqrt(n[0] ** 2 + n[1] ** 2 + n[2] ** 2) + TINY)
            sharp = 0.0
            for f, (plus, minus) in zip(n, ((_xp, _xm), (_yp, _ym), (_zp, _zm))):
                f.mul_(g)
                sharp = sharp + (plus(f) - minus(f))
            del n, g, t
            rhs = gumax * (eps * ddxi * (_xp(phi) + _xm(phi) + _yp(phi) + _ym(phi) + _zp(phi) + _zm(phi) - 6.0 * phi)
                           - 0.5 * dxi * sharp)
            for vel, plus, minus in ((u, _xp, _xm), (v, _yp, _ym), (w, _zp, _zm)):
                rhs -= 0.5 * dxi * (plus(vel) * (plus(phi) + phi) - vel * (phi + minus(phi)))
            phi = phi + dt * (al * rhs - (be * rphi if rphi is not None else 0.0))
            rphi = rhs
            chem = (phi * (1.0 - phi) * (1.0 - 2.0 * phi) / eps
                    - eps * ddxi * (_xp(phi) + _xm(phi) + _yp(phi) + _ym(phi) + _zp(phi) + _zm(phi) - 6.0 * phi))
        new = []
        forcing = (sz + cy, sx + cz, sy + cx)
        for c, (f, plus, minus) in enumerate(((u, _xp, _xm), (v, _yp, _ym), (w, _zp, _zm))):
            lap = _xp(f) + _xm(f) + _yp(f) + _ym(f) + _zp(f) + _zm(f) - 6.0 * f
            rhs = mu * ddxi * lap + forcing[c]
            del lap
            for d, (g, up, dn) in enumerate(((u, _xp, _xm), (v, _yp, _ym), (w, _zp, _zm))):
                flux = (f + dn(f)) * (g + minus(g))     # at the low face along d
                if d == c:                              # the cell-centred flux of the own axis
                    flux = (f + up(f)) ** 2
                    rhs -= 0.25 * dxi * (flux - dn(flux))
                else:
                    rhs -= 0.25 * dxi * (up(flux) - flux)
            if phi is not None:
                st = 3.0 * sigma * dxi * chem * (plus(phi) - minus(phi))
                rhs += 0.5 * (minus(st) + st)
            new.append(f + dt * (al * rhs - (be * ro[c] if ro[c] is not None else 0.0)))
            ro[c] = rhs
        u, v, w = new
        del new, rhs, flux
        al, be = 1.5, 0.5
        p = _solve((dxi / dt) * ((_xp(u) - u) + (_yp(v) - v) + (_zp(w) - w)), shape, case["laplacian"])
        u = u - dt * dxi * (p - _xm(p))
        v = v - dt * dxi * (p - _ym(p))
        w = w - dt * dxi * (p - _zm(p))
        u, v, w = u - u.mean(), v - v.mean(), w - w.mean()
        gumax = max(float(u.max()), float(v.max()), float(w.max()))
    return u, v, w, p, phi, part, gumax


def exact(case, seed):
    shapes = _boxes(case)
    got = {f: [] for f in _names(case)}
    for b, shape in enumerate(shapes):
        u, v, w, p, phi, part, gumax = _advance(case, shape, 1000 * seed + 7 * b, case["steps"])
        if case["kind"] == "analysis":
            return _looked_at(case, shape, u, v, w, gumax)
        for f, a in zip(("u", "v", "w", "p", "phi"), (u, v, w, p, phi)):
            if f in got:
                got[f].append(a.cpu().reshape(-1))
    got = {f: torch.cat(a) for f, a in got.items()}
    if case["tracers"]:
        got["part"] = part.cpu().T.contiguous()
    return got


def _looked_at(case, shape, u, v, w, gumax):
    nx, ny, nz = shape
    dx = LX / nx
    div = ((_xp(u) - u) + (_yp(v) - v) + (_zp(w) - w)) / dx
    n = nx * ny * nz
    bins = int(math.ceil(math.sqrt(3.0) * max(shape) / 2)) + 2
    shell = sum(_col(((np.fft.fftfreq(m, 1.0 / m) if a else np.arange(m // 2 + 1.0)) * nx / m) ** 2, a)
                for a, m in enumerate(shape))
    shell = torch.floor(torch.sqrt(shell) + 0.5).long().expand(nz, ny, nx // 2 + 1)
    weight = _col([1.0] + [2.0] * (nx // 2 - 1) + [1.0], 0)
    e = torch.zeros(bins, dtype=torch.float64, device="cuda")
    for f in (u, v, w):
        h = torch.fft.rfftn(f) / n
        power = 0.5 * weight * (h.real ** 2 + h.imag ** 2)
        e += torch.bincount(shell.reshape(-1), power.reshape(-1), minlength=bins)[:bins]
    # the drops' sums and the dissipation's stencil are the library's own definitions
    ke = float(0.5 * (u * u + v * v + w * w).mean())
    return {"gumax": gumax, "cfl": gumax * case["dt"] / dx, "maxdiv": float(div.abs().max()), "ke": ke, "dissipation": None,
            "spectrum": e.cpu(), "cells": None, "drops": None}
