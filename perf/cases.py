"""Timed workloads of the library, each through its public entry points.

A case is one pass of what a user's program repeats:

* ``frame``: a save frame of the time loop on the state API: `steps`
  predictor-force-corrector steps (the potential in the last one), the
  conservation sums and the snapshot's positions and velocities in pinned
  host memory.  `form` "one-sided" is a context as created; "pair" selects the
  symmetric kernel as the driver's ``--kernel pair`` does.  `systems` > 1 is
  the batched ensemble of independent galaxies.
* ``loop``: the reference's own time loop with its launches replaced call by
  call: predictor, force and corrector on the caller's device arrays.
* ``fp64``: steps with the direct sum in the reference's precision; the
  accelerations and potentials come back too.
* ``bin``: convert_particles_to_grid on the caller's device arrays: the
  zeroing, the binning with the mass deposit, and the prefix sums.
* ``cic``: cloud-in-cell deposit of the masses and interpolation of a field
  back to the bodies, device arrays.
* ``wave``: one step of the Wave mode (deposit, stencil iterations,
  gradient, gather, corrector).

Bodies come from the seeded galaxy generator (disk of stars + Plummer dark
matter, one to two).  A frame returns what the driver saves there (snapshot
and conservation row).
"""
from __future__ import annotations

import math
import pathlib
import sys

import numpy as np
import torch

_PKG = str(pathlib.Path(__file__).resolve().parents[1] / "khrr-nbody_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import khrr  # noqa: E402
from khrr.galaxy import ensemble_sizes, make_galaxy, two_galaxy_encounter  # noqa: E402

DT = 0.002
C_WAVE = 4574.337022617616
LIE_KEYS = ("Lx", "Ly", "Lz", "Ix", "Iy", "Iz", "Ek", "Ep", "E", "R_max", "Z_max", "Vr_max", "Vfi_max", "Vz_max")
HALO = {"Mh": 1.0, "a": 0.3333, "Rh": 1.0}


def listed():
    return [
        # The smallest galaxy in use (the tests' and the smoke run's size), a
        # context as created: launches and latency count.
        {"name": "frame_3072", "kind": "frame", "n": 3072, "systems": 1, "form": "one-sided", "eps_dm": 0.004, "steps": 5},
        # A ragged body count with softenings of its own for each component.
        {"name": "frame_10007_ragged", "kind": "frame", "n": 10007, "systems": 1, "form": "pair", "eps_dm": 0.008, "steps": 5},
        # The small benchmark galaxy (16,384 stars + 32,768 dark matter).
        {"name": "frame_49152", "kind": "frame", "n": 49152, "systems": 1, "form": "pair", "eps_dm": 0.004, "steps": 5},
        # A program that keeps its own device arrays, ragged count, two softenings.
        {"name": "loop_100003", "kind": "loop", "n": 100003, "form": "pair", "eps_dm": 0.008},
        # The headline galaxy (262,144 stars + 524,288 dark matter).
        {"name": "frame_786432", "kind": "frame", "n": 786432, "systems": 1, "form": "pair", "eps_dm": 0.004, "steps": 2},
        # Uneven independent galaxies advanced together.
        {"name": "ensemble_24", "kind": "frame", "n": 24, "systems": 24, "form": "pair", "eps_dm": 0.004, "steps": 2},
        # The reference's own precision on the small benchmark galaxy.
        {"name": "fp64_49152", "kind": "fp64", "n": 49152, "eps_dm": 0.004, "steps": 2},
        # Save-time binning of the large system on its 256^3 mesh.
        {"name": "bin_2097152_256", "kind": "bin", "n": 2097152, "nx": 256, "half": 4.0},
        # Cloud-in-cell on the encounter's mesh, dense galaxy cores.
        {"name": "cic_786432_128", "kind": "cic", "n": 786432, "nx": 128, "half": 4.0},
        # The two-galaxy encounter on the mesh path: 128^3, FP32 stencil, CIC, halo on.
        {"name": "wave_128_fp32", "kind": "wave", "n": 786432, "nx": 128, "half": 4.0, "dt": 0.002, "fp64": False, "cic": True, "halo": True},
        # The large mesh with the FP32 stencil.
        {"name": "wave_256_fp32", "kind": "wave", "n": 393216, "nx": 256, "half": 4.0, "dt": 0.0005, "fp64": False, "cic": True, "halo": False},
        # The driver's default Wave mode: 200^3 cells of 0.2, FP64 stencil, nearest grid point.
        {"name": "wave_200_fp64", "kind": "wave", "n": 49152, "nx": 200, "half": 20.0, "dt": 0.002, "fp64": True, "cic": False, "halo": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["frame", "frame", "frame", "loop", "ensemble", "fp64", "bin", "cic", "wave", "wave"])
    eps = rng.choice([0.004, 0.008])
    form = rng.choice(["one-sided", "pair"])
    if kind == "frame":
        n = _log(rng, 2048, 160000)
        if rng.random() < 0.5:
            n = max(2048, n // 1024 * 1024)
        return {"kind": "frame", "n": n, "systems": 1, "form": form, "eps_dm": eps, "steps": rng.randint(1, 6)}
    if kind == "loop":
        return {"kind": "loop", "n": _log(rng, 2048, 200000), "form": form, "eps_dm": eps}
    if kind == "ensemble":
        k = rng.randint(4, 32)
        return {"kind": "frame", "n": k, "systems": k, "form": form, "eps_dm": eps, "steps": rng.randint(1, 3)}
    if kind == "fp64":
        return {"kind": "fp64", "n": _log(rng, 2048, 90000), "eps_dm": eps, "steps": rng.randint(1, 3)}
    if kind in ("bin", "cic"):
        return {"kind": kind, "n": _log(rng, 20000, 2000000), "nx": _log(rng, 32, 256), "half": rng.choice([2.0, 4.0])}
    nx, fp64 = rng.choice([48, 64, 96, 100, 120, 128, 144, 160, 200, 201, 240, 256]), rng.random() < 0.5
    half = 20.0 if rng.random() < 0.4 else 4.0
    return {"kind": "wave", "n": _log(rng, 4096, 400000), "nx": nx, "half": half, "dt": 0.002 if half > 10 else 0.0005,
            "fp64": fp64, "cic": rng.random() < 0.5, "halo": rng.random() < 0.5}


# ---- bodies -------------------------------------------------------------------
def _bodies(case, seed):
    """(pos, vel, mass, eps2, offsets) of a case, float64 arrays."""
    n = case["n"]
    if case.get("systems", 1) > 1:
        # The sizes belong to the case; the bodies to the seed.
        parts = [make_galaxy(ns, nd, 100 * seed + k, eps_dm=case["eps_dm"]).arrays()
                 for k, (ns, nd) in enumerate(_system_sizes(case))]
        pos, vel, mass, eps = (np.concatenate([p[q] for p in parts]) for q in range(4))
        return pos, vel, mass, eps * eps, np.cumsum([0] + [len(p[2]) for p in parts])
    if case["kind"] in ("cic", "wave") and n % 6 == 0:
        return (*two_galaxy_encounter(n // 6, n // 2 - n // 6, seed), None)
    ns = n // 3 // 512 * 512 if n % 1024 == 0 else n // 3
    pos, vel, mass, eps = make_galaxy(ns, n - ns, seed, eps_dm=case.get("eps_dm", 0.004)).arrays()
    return pos, vel, mass, eps * eps, None


def _system_sizes(case):
    return ensemble_sizes(case["systems"], seed=77, lo=4096, hi=32768)


def _gpu(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()


def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()


def _wave_params(case):
    dx = 2.0 * case["half"] / case["nx"]
    return khrr.WaveParams.make(case["nx"], dx, c=C_WAVE)


def _iterations(case):
    return int(case["dt"] / _wave_params(case).dt)


SETUP_ITERS = 300


# ---- what a program has before the call ----------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    pos, vel, mass, eps2, off = _bodies(case, seed)
    n = len(mass)
    ctx = khrr.Context(0)
    s = {"case": case, "ctx": ctx, "n": n}
    if case.get("form") == "pair":
        ctx.set_tuning(128, 8, 128, 0, 2)
    if kind in ("frame", "fp64", "wave"):
        s["pos"], s["vel"] = _pinned(n, 3), _pinned(n, 3)
        if kind == "wave" and case["halo"]:
            ctx.set_external_field(**HALO)
        ctx.upload(pos, vel, mass, eps2, offsets=off)
        if kind == "frame":
            ctx.forces(khrr.ACC | khrr.PHI)
        elif kind == "fp64":
            s["acc"], s["phi"] = _pinned(n, 3), _pinned(n)
            ctx.forces(khrr.ACC | khrr.PHI | khrr.FP64)
        else:
            s["acc"] = _pinned(n, 3)
            ctx.set_mesh_solver(_wave_params(case), assign=khrr.ASSIGN_CIC if case["cic"] else khrr.ASSIGN_NGP,
                                fp64=case["fp64"], iters_per_step=_iterations(case), setup_iters=SETUP_ITERS)
            ctx.forces(khrr.ACC | khrr.PHI | khrr.MESH)
        ctx.synchronize()
        return s
    s["stream"] = torch.cuda.ExternalStream(ctx.stream)
    s["pos"], s["vel"], s["mass"], s["eps2"] = _gpu(pos), _gpu(vel), _gpu(mass), _gpu(eps2)
    if kind == "loop":
        for k in ("acc", "post", "velt", "acct"):
            s[k] = torch.zeros_like(s["pos"])
        torch.cuda.synchronize()
        p = s["pos"].data_ptr()
        ctx.accel(s["acc"].data_ptr(), p, p, s["mass"].data_ptr(), s["eps2"].data_ptr(), n, khrr.OVERWRITE)
        ctx.synchronize()
        return s
    nx, half = case["nx"], case["half"]
    cells = nx ** 3
    s["mesh"] = khrr.Mesh.make((-half,) * 3, (2 * half / nx,) * 3, (nx,) * 3)
    s["cell_mass"] = torch.zeros(cells, dtype=torch.float64, device="cuda")
    if kind == "bin":
        s["pci"] = torch.zeros((n, 2), dtype=torch.int32, device="cuda")
        s["info"] = torch.zeros((cells, 2), dtype=torch.int32, device="cuda")
        s["count"] = torch.zeros(cells, dtype=torch.int32, device="cuda")
        s["max_pbc"] = torch.zeros((cells + 511) // 512, dtype=torch.int32, device="cuda")
    else:
        g = torch.Generator(device="cuda").manual_seed(seed)
        s["cell_acc"] = torch.randn((cells, 3), dtype=torch.float64, device="cuda", generator=g)
        s["cell_phi"] = torch.randn(cells, dtype=torch.float64, device="cuda", generator=g)
        s["acc"], s["phi"] = torch.zeros_like(s["pos"]), torch.zeros_like(s["mass"])
    torch.cuda.synchronize()
    return s


# ---- one pass -------------------------------------------------------------------
def run(s):
    case, ctx, n = s["case"], s["ctx"], s["n"]
    kind = case["kind"]
    if kind == "frame":
        ctx.step(DT, case["steps"], khrr.PHI)
        lie = ctx.conservation()
        ctx.download_into(pos=s["pos"], vel=s["vel"])
        return {"pos": s["pos"], "vel": s["vel"], "lie": np.array([lie[k] for k in LIE_KEYS])}
    if kind == "fp64":
        ctx.step(DT, case["steps"], khrr.PHI | khrr.FP64)
        ctx.download_into(pos=s["pos"], vel=s["vel"], acc=s["acc"], phi=s["phi"])
        return {k: s[k] for k in ("pos", "vel", "acc", "phi")}
    if kind == "wave":
        ctx.step(case["dt"], 1, khrr.MESH)
        ctx.download_into(pos=s["pos"], vel=s["vel"], acc=s["acc"])
        return {k: s[k] for k in ("pos", "vel", "acc")}
    if kind == "loop":
        pos, vel, acc, post, velt, acct = (s[k].data_ptr() for k in ("pos", "vel", "acc", "post", "velt", "acct"))
        mass, eps2 = s["mass"].data_ptr(), s["eps2"].data_ptr()
        ctx.integ_time(acc, post, velt, pos, vel, DT, 0, 0.0, acc, n)
        ctx.accel(acct, post, post, mass, eps2, n, khrr.OVERWRITE)
        ctx.integ_time(acct, pos, vel, post, velt, DT, 1, 0.0, acc, n)
        return {"pos": s["pos"], "vel": s["vel"]}
    if kind == "bin":
        with torch.cuda.stream(s["stream"]):
            for k in ("info", "count", "cell_mass"):
                s[k].zero_()
        ctx.assign_particles_to_cells(s["pos"].data_ptr(), n, s["mesh"], s["pci"].data_ptr(), s["info"].data_ptr(),
                                      s["count"].data_ptr(), s["mass"].data_ptr(), s["cell_mass"].data_ptr())
        ctx.compute_prefix_sums(s["info"].data_ptr(), s["max_pbc"].data_ptr(), case["nx"] ** 3, khrr.SCAN_EXCLUSIVE)
        # the slot of a body inside its cell is the arrival order of atomics
        return {"cell_id": s["pci"][:, 0], "info": s["info"], "max_pbc": s["max_pbc"], "cell_mass": s["cell_mass"]}
    with torch.cuda.stream(s["stream"]):
        s["cell_mass"].zero_()
    pos = s["pos"].data_ptr()
    ctx.cic_deposit(pos, s["mass"].data_ptr(), n, s["mesh"], s["cell_mass"].data_ptr())
    ctx.cic_gather(pos, n, s["mesh"], s["cell_acc"].data_ptr(), s["cell_phi"].data_ptr(), s["acc"].data_ptr(),
                   s["phi"].data_ptr())
    return {"cell_mass": s["cell_mass"], "acc": s["acc"], "phi": s["phi"]}


# ---- the work a pass cannot do without ------------------------------------------
def work(case):
    """Direct sum: 23 flops per unordered pair (an FMA counts 2) and the state
    read and written once per step.  Stencil: each field value read and
    written once per iteration (phi, phi_old and mass in, phi out)."""
    kind = case["kind"]
    if kind in ("frame", "loop", "fp64"):
        sizes = [sum(p) for p in _system_sizes(case)] if case.get("systems", 1) > 1 else [case["n"]]
        steps = case.get("steps", 1)
        return {"bytes": float(steps * 152 * sum(sizes)), "flops": float(steps * sum(23.0 * m * m / 2 for m in sizes))}
    n, cells = case["n"], case["nx"] ** 3
    if kind == "bin":
        return {"bytes": 40.0 * n + 20.0 * cells, "flops": 12.0 * n}
    if kind == "cic":
        return {"bytes": (24.0 + 8.0 + 32.0) * n + (8.0 + 32.0) * cells, "flops": 8.0 * 14 * n}
    it, word = _iterations(case), 8.0 if case["fp64"] else 4.0
    return {"bytes": it * 4.0 * word * cells + 152.0 * n, "flops": it * 15.0 * cells + 200.0 * n}


# ---- the same in 64 bits ----------------------------------------------------------
def _direct(pos, mass, eps2, off):
    """FP64 direct sum per system: (acc, phi)."""
    acc, phi = torch.zeros_like(pos), torch.zeros_like(mass)
    for a, b in zip(off[:-1], off[1:]):
        x, m, e = pos[a:b], mass[a:b], eps2[a:b]
        rows = max(1, (1 << 25) // (b - a))
        for i in range(0, b - a, rows):
            j = min(i + rows, b - a)
            d = [x[None, :, k] - x[i:j, None, k] for k in range(3)]
            r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2] + 0.5 * (e[None, :] + e[i:j, None])
            inv = torch.rsqrt(r2)
            w = m[None, :] * inv
            phi[a + i:a + j] = -w.sum(1)
            w = w * inv * inv
            for k in range(3):
                acc[a + i:a + j, k] = (w * d[k]).sum(1)
    return acc, phi


def _field(p, on):
    """The analytic halo of HALO (no bulge)."""
    if not on:
        return torch.zeros_like(p)
    a, mh, r2 = HALO["a"], HALO["Mh"], 3.0 * HALO["Rh"]
    core = HALO["Rh"] / a - math.atan(HALO["Rh"] / a)
    r = p.norm(dim=1)
    inside = -mh / core * (r / a - torch.atan(r / a)) / r ** 3
    outside = -mh * (r2 / a - math.atan(r2 / a)) / core / r ** 3
    return torch.where(r < r2, inside, outside)[:, None] * p


def _lie(pos, vel, mass, phi):
    c = torch.linalg.cross(pos, vel)
    r = (pos[:, 0] ** 2 + pos[:, 1] ** 2).sqrt()
    vr = (vel[:, 0] * pos[:, 0] + vel[:, 1] * pos[:, 1]) / r
    vf = c[:, 2] / r
    ek, ep = (mass * (vel * vel).sum(1)).sum(), (mass * phi).sum()
    return torch.stack([*(mass[:, None] * c).sum(0), *(mass[:, None] * vel).sum(0), ek, ep, 0.5 * (ek + ep), r.max(),
                        pos[:, 2].abs().max(), vr.abs().max(), vf.max().clamp(min=0.0), vel[:, 2].abs().max()])


def _corners(pos, nx, half, cic):
    """(cell, weight, inside) of each corner of each body's cloud; NGP has one."""
    dx = 2 * half / nx
    u = (pos + half) / dx
    if not cic:
        c = u.trunc().clamp(0, nx - 1).long()
        return [((c[:, 2] * nx + c[:, 1]) * nx + c[:, 0], torch.ones_like(u[:, 0]))]
    u = u - 0.5
    f0 = u.floor()
    f = u - f0
    out = []
    for q in range(8):
        b = torch.tensor([q & 1, q >> 1 & 1, q >> 2], device=pos.device)
        c = f0 + b
        w = torch.where(b.bool(), f, 1.0 - f).prod(1)
        inside = ((c >= 0) & (c < nx)).all(1)
        c = c.clamp(0, nx - 1).long()
        out.append(((c[:, 2] * nx + c[:, 1]) * nx + c[:, 0], torch.where(inside, w, torch.zeros_like(w))))
    return out


def _deposit(corners, mass, cells):
    out = torch.zeros(cells, dtype=torch.float64, device=mass.device)
    for c, w in corners:
        out.index_add_(0, c, mass * w)
    return out


def _stencil(phi, old, mass, case, iters):
    """Damped-wave iterations on z, y, x arrays."""
    P, nx = _wave_params(case), case["nx"]
    x = torch.arange(nx, dtype=torch.float64, device=phi.device) * P.dx
    L = P.sim_l - P.bc_l
    hi = torch.where(x > L, P.diss_extra * (x - L) ** 2, torch.zeros_like(x))  # x >= 0 here
    sx = P.diss_extra * (x - L) ** 2
    Q = (P.diss_base + sx[None, None, :] + hi[None, :, None] + hi[:, None, None]) * (P.c * P.dt * 0.5)
    w, K = 1.0 / (1.0 + Q), (P.c * P.dt / P.dx) ** 2
    i = slice(1, -1)
    wi, kold = w[i, i, i], ((Q - 1.0) * w)[i, i, i]
    src = (-(P.c * P.dt) ** 2 * 4.0 * math.pi / P.dx ** 3) * (mass.view(nx, nx, nx) * w)[i, i, i]
    for _ in range(iters):
        nb = phi[:-2, i, i] + phi[2:, i, i] + phi[i, :-2, i] + phi[i, 2:, i] + phi[i, i, :-2] + phi[i, i, 2:]
        new = torch.zeros_like(phi)
        new[i, i, i] = (K * nb + 2.0 * (1.0 - 3.0 * K) * phi[i, i, i]) * wi + old[i, i, i] * kold + src
        phi, old = new, phi
    return phi, old


def _gradient(phi, dx):
    """-grad(phi) as (cells, 3), one-sided differences (not halved) on faces."""
    out = []
    for axis in (2, 1, 0):
        p = phi.movedim(axis, 0)
        d = torch.empty_like(p)
        d[1:-1] = 0.5 * (p[2:] - p[:-2])
        d[0], d[-1] = p[1] - p[0], p[-1] - p[-2]
        out.append(d.movedim(0, axis).reshape(-1) * (-1.0 / dx))
    return torch.stack(out, 1)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("frame", "loop") and case["n"] > 170000:
        return None  # the 64-bit direct sum takes too long
    pos, vel, mass, eps2, off = _bodies(case, seed)
    off = [0, len(mass)] if off is None else [int(o) for o in off]
    pos, vel, mass, eps2 = _gpu(pos), _gpu(vel), _gpu(mass), _gpu(eps2)
    if kind in ("frame", "loop", "fp64"):
        acc, phi = _direct(pos, mass, eps2, off)
        for _ in range(case.get("steps", 1)):
            velt = vel + DT * acc
            pos = pos + 0.5 * DT * (vel + velt)
            acc, phi = _direct(pos, mass, eps2, off)
            vel = 0.5 * (vel + velt + DT * acc)
        if kind == "loop":
            return {"pos": pos, "vel": vel}
        if kind == "fp64":
            return {"pos": pos, "vel": vel, "acc": acc, "phi": phi}
        return {"pos": pos, "vel": vel, "lie": _lie(pos, vel, mass, phi)}
    nx, half = case["nx"], case["half"]
    cells, dx = nx ** 3, 2 * half / nx
    if kind == "bin":
        return {"cell_id": None, "info": None, "max_pbc": None,
                "cell_mass": _deposit(_corners(pos, nx, half, False), mass, cells)}
    if kind == "cic":
        g = torch.Generator(device="cuda").manual_seed(seed)
        field = torch.randn((cells, 3), dtype=torch.float64, device="cuda", generator=g)
        value = torch.randn(cells, dtype=torch.float64, device="cuda", generator=g)
        corners = _corners(pos, nx, half, True)
        return {"cell_mass": _deposit(corners, mass, cells), "acc": sum(w[:, None] * field[c] for c, w in corners),
                "phi": sum(w * value[c] for c, w in corners)}
    phi = torch.zeros((nx, nx, nx), dtype=torch.float64, device="cuda")
    old = torch.zeros_like(phi)

    def force(p, iters):
        nonlocal phi, old
        corners = _corners(p, nx, half, case["cic"])
        phi, old = _stencil(phi, old, _deposit(corners, mass, cells), case, iters)
        field = _gradient(phi, dx)
        return sum(w[:, None] * field[c] for c, w in corners)

    dt = case["dt"]
    acc = force(pos, SETUP_ITERS)
    f = acc + _field(pos, case["halo"])
    velt = vel + dt * f
    pos = pos + 0.5 * dt * (vel + velt)
    acc = force(pos, _iterations(case))
    vel = 0.5 * (vel + velt + dt * (acc + _field(pos, case["halo"])))
    return {"pos": pos, "vel": vel, "acc": acc}
