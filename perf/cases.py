"""The work this framework does for its users, as cases to time and check.

A case is a dict of plain values with a "kind":

  step      a resident simulation advanced by `steps` timesteps through
            Solver.step, then read on the device (sync_state, device_state):
            the time loop of a run whose state stays on the GPU
  job       a whole short run on host arrays: set_fields, step, get_fields
  poisson   one stand-alone pressure solve on device arrays, through a handle
            or (n <= 128) through the allocation-free entry point
  analysis  the diagnostics of a resident state: Solver.stats, Solver.drops
  serve     a batch of independent requests through the served Ensemble

Initial fields: a random-phase velocity, E(k) ~ k^4 exp(-2 (k/4)^2) with rms 1
on the staggered grid, and non-overlapping drops with the tanh profile, the
recipes of mhit36_b200/fields.py drawn on the GPU.  dt, mu, sigma and the
linear forcing are those of the benchmark workload.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from mhit36_b200 import Solver, capi
from mhit36_b200.config import InputParams
from mhit36_b200.ensemble import Ensemble

SIZES = (32, 64, 96, 128, 192, 256, 384, 512)
# drops, smallest and largest radius (tests, benchmark configurations)
DROPS = {32: (2, 0.6, 0.8), 64: (4, 0.4, 0.6), 512: (64, 0.2, 0.35)}


def _step(name, n, precision, phase, steps, forcing="linear", k2=0, grid=0):
    if precision == "fp32":
        k2 = 1  # the refinement form solves with the FD-modified k^2
    return {"name": name, "kind": "step", "n": n, "precision": precision, "phase": phase, "steps": steps,
            "forcing": forcing, "k2": k2, "grid": grid}


def listed():
    return [
        # the driver's loop on the smallest grid: one step per call, its diagnostics read back each time
        _step("step_ns_fp64_32", 32, "fp64", False, 1),
        # small drop simulations (tests' and the served stream's sizes), several steps per call
        _step("step_acdi_fp64_64", 64, "fp64", True, 10),
        # the 128^3 configuration with 8 drops
        _step("step_acdi_fp64_128", 128, "fp64", True, 5),
        # a size with a factor 3, the reference's ABC forcing
        _step("step_acdi_abc_fp64_192", 192, "fp64", True, 3, forcing="abc"),
        # the 256^3 configuration
        _step("step_acdi_fp64_256", 256, "fp64", True, 2),
        # the headline workload: 512^3 NS+ACDI with 64 drops, and its FP32 refinement form
        _step("step_acdi_fp64_512", 512, "fp64", True, 2),
        _step("step_acdi_fp32_512", 512, "fp32", True, 2),
        # a short run from host arrays to host arrays in the FP32 form
        {"name": "job_acdi_fp32_192", "kind": "job", "n": 192, "precision": "fp32", "phase": True, "steps": 10,
         "forcing": "linear", "k2": 1, "grid": 0},
        # the pressure solver alone, for a caller with its own time loop: a large grid, and a
        # latency-bound caller that owns all device memory
        {"name": "poisson_384", "kind": "poisson", "n": 384, "noalloc": False, "k2": 0, "grid": 0},
        {"name": "poisson_noalloc_64", "kind": "poisson", "n": 64, "noalloc": True, "k2": 1, "grid": 1},
        # energy, dissipation, divergence, drop count and sizes of a resident state, as a run logs them
        {"name": "analysis_fp64_256", "kind": "analysis", "n": 256, "precision": "fp64"},
        # a served batch: drop and single-phase requests of two grid sizes
        {"name": "serve_fp64_64_96", "kind": "serve", "n": 64, "n2": 96, "precision": "fp64", "requests": 6,
         "steps": 25},
    ]


def draw(rng: random.Random):
    kind = rng.choices(("step", "poisson", "analysis", "job", "serve"), (10, 4, 2, 2, 1))[0]
    if kind == "step":
        n = rng.choice(SIZES)
        most = max(2, min(16, int(2 * (512 / n) ** 3)))  # no more than the largest listed case
        precision = rng.choice(("fp64", "fp64", "fp32"))
        c = _step("", n, precision, rng.random() < 0.7, rng.randint(1, most), rng.choice(("linear", "linear", "abc", "none")),
                  rng.randint(0, 1), rng.randint(0, 1))
        del c["name"]
        return c
    if kind == "poisson":
        n = rng.choice(SIZES)
        return {"kind": "poisson", "n": n, "noalloc": n <= 128 and rng.random() < 0.5, "k2": rng.randint(0, 1),
                "grid": rng.randint(0, 1)}
    if kind == "analysis":
        precision = rng.choice(("fp64", "fp32"))
        return {"kind": "analysis", "n": rng.choice(SIZES), "precision": precision, "k2": 1 if precision == "fp32" else 0}
    if kind == "job":
        precision = rng.choice(("fp64", "fp32"))
        return {"kind": "job", "n": rng.choice((32, 64, 96, 128, 192)), "precision": precision,
                "phase": rng.random() < 0.7, "steps": rng.randint(1, 20), "forcing": rng.choice(("linear", "abc")),
                "k2": 1 if precision == "fp32" else rng.randint(0, 1), "grid": 0}
    return {"kind": "serve", "n": rng.choice((64, 96)), "n2": rng.choice((32, 64, 96, 128)), "precision": "fp64",
            "requests": rng.randint(2, 8), "steps": rng.randint(5, 40)}


# ---------------------------------------------------------------- inputs
def _params(c):
    p = dict(dt=2e-4, mu=6e-3, rho=1.0, sigma=0.5, epsr=1.0, k2_mode=c.get("k2", 0), grid_mode=c.get("grid", 0))
    forcing = c.get("forcing", "linear")
    if forcing == "linear":
        p["lin_force"] = 0.1
    elif forcing == "abc":
        p.update(f1=0.3, f2=0.2, f3=0.1, k0=2.0)
    return InputParams(**p)


def _dx(n, grid):
    return 2 * math.pi / (n if grid else n - 1)


def _velocity(n, gen):
    """u, v, w as (z, y, x) float64 tensors on the GPU."""
    dev = gen.device
    k = torch.fft.fftfreq(n, 1.0 / n, dtype=torch.float64, device=dev)
    kh = torch.arange(n // 2 + 1, dtype=torch.float64, device=dev)
    K = (kh[None, None, :], k[None, :, None], k[:, None, None])  # x, y, z
    k2 = K[0] ** 2 + K[1] ** 2 + K[2] ** 2
    amp = k2 * torch.exp(-(k2 / 16.0))  # sqrt(E/k^2) up to a factor
    k2[0, 0, 0] = 1.0
    F = []
    for _ in range(3):
        f = torch.fft.rfftn(torch.randn(n, n, n, dtype=torch.float64, device=dev, generator=gen))
        F.append(f * (amp / k2.sqrt()))
    div = (K[0] * F[0] + K[1] * F[1] + K[2] * F[2]) / k2
    out = []
    for c in range(3):
        f = F[c] - K[c] * div
        f = f * torch.polar(torch.ones_like(K[c]), -math.pi / n * K[c])  # half a cell back along its own axis
        f[0, 0, 0] = 0
        F[c] = None
        out.append(torch.fft.irfftn(f, s=(n, n, n)))
        del f
    rms = math.sqrt(sum(float((a * a).mean()) for a in out) / 3.0)
    for a in out:
        a /= rms
    return out


def _drops(n, grid, rng, dev, most=None):
    count, rmin, rmax = DROPS.get(n, (8, 0.4, 0.6))
    count = count if most is None else min(count, most)
    dx = _dx(n, grid)
    period = n * dx
    drops = []
    while len(drops) < count:
        c, r = [rng.uniform(0.0, period) for _ in range(3)], rng.uniform(rmin, rmax)
        if all(math.dist([0, 0, 0], [(a - b) - period * round((a - b) / period) for a, b in zip(c, c2)])
               > r + r2 + 4 * dx for c2, r2 in drops):
            drops.append((c, r))
    x = torch.arange(n, dtype=torch.float64, device=dev) * dx
    d = torch.full((n, n, n), 1e9, dtype=torch.float64, device=dev)
    for c, r in drops:
        q = [((x - a) - period * torch.round((x - a) / period)) ** 2 for a in c]
        d = torch.minimum(d, (q[0][None, None, :] + q[1][None, :, None] + q[2][:, None, None]).sqrt_().sub_(r))
    return 0.5 * (1.0 - torch.tanh(d / (2 * dx)))


def _fields(c, seed, n=None, phase=None):
    n = c["n"] if n is None else n
    phase = c.get("phase", True) if phase is None else phase
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    f = _velocity(n, gen)
    f.append(_drops(n, c.get("grid", 0), random.Random(int(seed) + 1), gen.device) if phase else None)
    if c.get("precision") == "fp32":  # inputs the form can hold
        f = [None if a is None else a.float().double() for a in f]
    return f


_staging = {}


def _upload(solver, f, n):
    """Host arrays from one pinned buffer that every solver of this process uploads from."""
    count = sum(a is not None for a in f)
    if _staging.get("size", 0) < count * n ** 3:
        _staging["buf"] = torch.empty(count * n ** 3, dtype=torch.float64, pin_memory=True)
        _staging["size"] = count * n ** 3
    ptrs = []
    for q in range(4):
        if f[q] is None:
            ptrs.append(None)
            continue
        h = _staging["buf"][q * n ** 3:(q + 1) * n ** 3]
        h.copy_(f[q].reshape(-1))
        ptrs.append(h.data_ptr())
    solver.set_fields_ptr(*ptrs)


class _Array:
    """A resident device field as torch reads it, without a copy; a tensor on it keeps the solver alive."""

    def __init__(self, ptr, n, dtype, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n, n, n), "typestr": dtype, "data": (ptr, False), "version": 3}


def _view(solver, ptr, n, precision):
    return torch.as_tensor(_Array(ptr, n, "<f4" if precision == "fp32" else "<f8", solver), device="cuda")


def _raw(a):
    return None if a is None else a.reshape(-1).cpu().numpy()


def _requests(c):
    """(n, phase, steps, seed offset) of each request of a served batch."""
    return [(c["n"] if q % 3 else c["n2"], q % 4 != 1, c["steps"] + 5 * (q % 3), 100 * q) for q in range(c["requests"])]


def prepare(case, seed):
    c = dict(case)
    if c["kind"] in ("step", "analysis"):
        f = _fields(c, seed)
        s = Solver(c["n"], _params(c), precision=c["precision"], phase_field=c.get("phase", True))
        _upload(s, f, c["n"])
        c["solver"] = s
    elif c["kind"] == "job":
        c["fields"] = [None if a is None else a.cpu().numpy().T for a in _fields(c, seed)]  # a[i, j, k], file order
        c["solver"] = Solver(c["n"], _params(c), precision=c["precision"], phase_field=c["phase"])
    elif c["kind"] == "poisson":
        n = c["n"]
        c["rhs"] = _rhs(n, seed)
        c["p"] = torch.empty_like(c["rhs"])
        if c["noalloc"]:
            c["lib"] = capi.load_library()
        else:
            c["solver"] = Solver(n, _params(c), phase_field=False)
    else:
        c["ensemble"] = Ensemble(budget_bytes=8 << 30, slots_per_class=8)
        c["list"] = []
        for n, phase, steps, off in _requests(c):
            c["list"].append((n, steps, [_raw(a) for a in _fields(c, seed + off, n, phase)]))
    torch.cuda.synchronize()
    return c


def _rhs(n, seed):
    """A zero-mean source with energy at all scales, as the divergence of a predicted velocity has."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    r = torch.randn(n, n, n, dtype=torch.float64, device="cuda", generator=gen)
    return r - r.mean()


def run(c):
    kind, n = c["kind"], c["n"]
    if kind == "step":
        s = c["solver"]
        d = s.step(c["steps"])
        s.sync_state()
        ptrs = s.device_state()
        return {"fields": [_view(s, p, n, c["precision"]) for p in ptrs if p], "umax": d["umax"], "cfl": d["cfl"]}
    if kind == "job":
        s = c["solver"]
        s.set_fields(*c["fields"])
        d = s.step(c["steps"])
        return {"fields": [a for a in s.get_fields() if a is not None], "umax": d["umax"], "cfl": d["cfl"]}
    if kind == "poisson":
        if c["noalloc"]:
            rc = c["lib"].mhit_poisson_noalloc(c["rhs"].data_ptr(), c["p"].data_ptr(), n, c["k2"], c["grid"],
                                               torch.cuda.current_stream().cuda_stream)
            if rc:
                raise capi.MhitError(rc, "mhit_poisson_noalloc")
        else:
            c["solver"].poisson_device(c["rhs"].data_ptr(), c["p"].data_ptr())
        return c["p"]
    if kind == "analysis":
        st = c["solver"].stats()
        cells, deq = c["solver"].drops()
        return {"stats": [st[k] for k in ("ke", "dissipation", "max_div", "phi_sum", "phi_max")], "cells": cells,
                "deq": deq}
    e, p, out = c["ensemble"], _params(c), []
    ids = [e.submit(n_, p, *f, nsteps=steps, precision=c["precision"], borrow=True) for n_, steps, f in c["list"]]
    e.run()
    for i in ids:
        q = e.query(i)
        if q["state"] != "done":
            raise RuntimeError("request %d: %s, status %d" % (i, q["state"], q["status"]))
        out.append([a for a in e.result(i) if a is not None])
        e.release(i)
    return out


# ---------------------------------------------------------------- work
def _step_bytes(n, precision, phase):
    """Bytes of one step that no schedule saves on grids beyond the cache: the
    state (u, v, w, their AB2 history, phi) in and out, the predicted velocity
    out and back in (the projection needs all of it first), and the half
    spectrum out and in between the x, y, z, y and x transforms."""
    e = 4 if precision == "fp32" else 8
    passes = (14 if phase else 12) + 6 + 8
    if precision == "fp32":
        passes += 2 + 3 + 1 + 8  # p0 out and in, the residual's read of ustar and p0's spectrum in, second solve
    return passes * e * n ** 3


def _step_flops(n, phase):
    return (260 if phase else 130) * n ** 3 + 15 * n ** 3 * math.log2(n)


def work(c):
    kind, n = c["kind"], c["n"]
    if kind == "step":
        return {"bytes": c["steps"] * _step_bytes(n, c["precision"], c["phase"]),
                "flops": c["steps"] * _step_flops(n, c["phase"])}
    if kind == "job":
        host = 2 * (4 if c["phase"] else 3) * 8 * n ** 3
        return {"bytes": host + c["steps"] * _step_bytes(n, c["precision"], c["phase"]),
                "flops": c["steps"] * _step_flops(n, c["phase"])}
    if kind == "poisson":
        return {"bytes": 10 * 8 * n ** 3, "flops": 15 * n ** 3 * math.log2(n)}  # rhs, p, four spectrum exchanges
    if kind == "analysis":
        return {"bytes": 4 * (4 if c["precision"] == "fp32" else 8) * n ** 3, "flops": 60 * n ** 3}
    total = {"bytes": 0, "flops": 0}
    for n_, phase, steps, _ in _requests(c):
        total["bytes"] += steps * _step_bytes(n_, c["precision"], phase) + 2 * (4 if phase else 3) * 8 * n_ ** 3
        total["flops"] += steps * _step_flops(n_, phase)
    return total


def tolerance(c):
    """About four times the largest difference from exact() seen over the ranges: 4e-16 (fields), 8e-16 (pressure
    solves) and 4e-15 (largest) in 64 bits, 8e-7 and 5e-6 in the FP32 form.  The diagnostics are 64-bit sums in both."""
    if c.get("precision") == "fp32" and c["kind"] != "analysis":
        return {"rel": 3e-6, "max": 2e-5}
    return {"rel": 3e-15, "max": 2e-14}


# ---------------------------------------------------------------- 64-bit values in plain torch
def _k2(n, k2, grid, dev):
    m = torch.arange(n, dtype=torch.float64, device=dev)
    if k2:
        return 4.0 / _dx(n, grid) ** 2 * torch.sin(math.pi * m / n) ** 2
    return torch.where(m < n // 2, m, m - n) ** 2


def _solve(rhs, k2, grid):
    """p with lap p = rhs on the periodic grid, zero mean."""
    n = rhs.shape[0]
    q = _k2(n, k2, grid, rhs.device)
    f = torch.fft.rfftn(rhs)
    d = q[:, None, None] + q[None, :, None] + q[None, None, :n // 2 + 1]
    d[0, 0, 0] = 1.0
    f.div_(d).neg_()
    f[0, 0, 0] = 0
    del d
    return torch.fft.irfftn(f, s=(n, n, n))


def _p(a, ax):
    return torch.roll(a, -1, 2 - ax)  # value at +1 along x (0), y (1), z (2)


def _m(a, ax):
    return torch.roll(a, 1, 2 - ax)


def _lap(a):
    return sum(_p(a, ax) + _m(a, ax) for ax in range(3)) - 6.0 * a


def _phase(phi, vel, p, n, gumax):
    dx = _dx(n, p.grid_mode)
    dxi, eps, enum = 1.0 / dx, p.epsr * dx, float(np.float32(1e-16))
    val = phi.clamp(0.0, 1.0)
    psi = eps * torch.log((val + enum) / (1.0 - val + enum))
    g = [_p(psi, ax) - _m(psi, ax) for ax in range(3)]
    del psi
    norm = (g[0] ** 2 + g[1] ** 2 + g[2] ** 2).sqrt_().add_(enum)
    t = (2.0 * val - 1.0) / (1.0 + 2.0 * enum)
    amp = 0.25 * (1.0 - t * t) / norm
    del val, norm, t
    rhs = gumax * eps * dxi * dxi * _lap(phi)
    for ax in range(3):
        f = amp * g[ax]
        g[ax] = None
        rhs -= gumax * (_p(f, ax) - _m(f, ax)) * 0.5 * dxi
        u = vel[ax]
        rhs -= (_p(u, ax) * (_p(phi, ax) + phi) - u * (phi + _m(phi, ax))) * 0.5 * dxi
    return phi + p.dt * rhs


def _momentum(vel, phi, p, n):
    dx = _dx(n, p.grid_mode)
    dxi, eps = 1.0 / dx, p.epsr * dx
    out = []
    force = None
    if phi is not None:
        chem = phi * (1.0 - phi) * (1.0 - 2.0 * phi) / eps - eps * _lap(phi) * dxi * dxi
        force = [6.0 * p.sigma * chem * 0.5 * (_p(phi, ax) - _m(phi, ax)) * dxi for ax in range(3)]
        del chem
    x = torch.arange(n, dtype=torch.float64, device=vel[0].device) * dx
    sn, cs = torch.sin(p.k0 * x), torch.cos(p.k0 * x)
    X, Y, Z = (lambda a: a[None, None, :]), (lambda a: a[None, :, None]), (lambda a: a[:, None, None])
    for a in range(3):
        r = p.mu * _lap(vel[a]) * dxi * dxi / p.rho
        for b in range(3):
            if a == b:  # flux through cell centres
                f = (_p(vel[a], a) + vel[a]) ** 2
                r -= 0.25 * dxi * (f - _m(f, a))
            else:  # flux through the edge between faces a and b
                f = (vel[a] + _m(vel[a], b)) * (vel[b] + _m(vel[b], a))
                r -= 0.25 * dxi * (_p(f, b) - f)
        if a == 0:
            r += p.f3 * Z(sn) + p.f2 * Y(cs)
        elif a == 1:
            r += p.f1 * X(sn) + p.f3 * Z(cs)
        else:
            r += p.f2 * Y(sn) + p.f1 * X(cs)
        if p.lin_force:
            r += p.lin_force * vel[a]
        if force is not None:
            r += 0.5 * (force[a] + _m(force[a], a)) / p.rho
        out.append(r)
    return out


def _advance(f, p, n, steps):
    """`steps` timesteps of u, v, w, phi in 64 bits: (fields, umax, cfl)."""
    vel, phi = list(f[:3]), f[3]
    dxi = 1.0 / _dx(n, p.grid_mode)
    old, gumax = None, 1.0
    for _ in range(steps):
        if phi is not None:
            phi = _phase(phi, vel, p, n, gumax)
        rhs = _momentum(vel, phi, p, n)
        for a in range(3):
            vel[a] = vel[a] + p.dt * (rhs[a] if old is None else 1.5 * rhs[a] - 0.5 * old[a])
        old = rhs
        div = sum(_p(vel[a], a) - vel[a] for a in range(3)) * (p.rho * dxi / p.dt)
        pr = _solve(div, p.k2_mode, p.grid_mode)
        for a in range(3):
            vel[a] = vel[a] - p.dt / p.rho * (pr - _m(pr, a)) * dxi
            vel[a] -= vel[a].mean()
        gumax = max(float(v.max()) for v in vel)
    return vel + ([] if phi is None else [phi]), gumax, gumax * p.dt * dxi


def _components(mask):
    """Cell counts of the 26-connected periodic components, by their first cell in scan order."""
    n = mask.shape[0]
    far = n ** 3
    lab = torch.where(mask, torch.arange(far, device=mask.device).reshape(n, n, n), far)
    while True:
        new = lab
        for ax in range(3):
            new = torch.minimum(new, torch.minimum(_p(new, ax), _m(new, ax)))
        new = torch.where(mask, new, far)
        if torch.equal(new, lab):
            break
        lab = new
    return torch.unique(lab[mask], return_counts=True)[1]


def exact(case, seed):
    c = dict(case)
    kind, n = c["kind"], c["n"]
    if kind in ("step", "job"):
        f, umax, cfl = _advance(_fields(c, seed), _params(c), n, c["steps"])
        if kind == "job":
            f = [a.cpu().numpy().T for a in f]
        return {"fields": f, "umax": umax, "cfl": cfl}
    if kind == "poisson":
        return _solve(_rhs(n, seed), c["k2"], c["grid"])
    if kind == "analysis":
        u, v, w, phi = _fields(c, seed)
        p, dx = _params(c), _dx(n, 0)
        h = 0.5 * (n - 1) / (2 * float(np.float32(3.14159265358979)))  # the post-processor's float32 pi
        d = [[(_p(a, ax) - _m(a, ax)) * h for ax in range(3)] for a in (u, v, w)]
        ss = sum(d[a][a] ** 2 for a in range(3)) + sum(
            2.0 * (0.5 * (d[a][b] + d[b][a])) ** 2 for a, b in ((0, 1), (0, 2), (1, 2)))
        div = sum(_p(a, ax) - a for ax, a in enumerate((u, v, w))) / dx
        cells = _components(phi >= 0.5).cpu().numpy()
        return {"stats": [0.5 * float((u * u + v * v + w * w).mean()), 2.0 * p.mu / p.rho * float(ss.mean()),
                          float(div.abs().max()), float(phi.sum()), float(phi.max())],
                "cells": cells, "deq": dx * (6.0 / math.pi * cells.astype(np.float64)) ** (1.0 / 3.0)}
    out = []
    for n_, phase, steps, off in _requests(c):
        out.append([a.cpu().numpy().T for a in
                    _advance(_fields(c, seed + off, n_, phase), _params(c), n_, steps)[0]])
    return out
