"""The work whose speed is measured: calls a user of this library makes, each through
its public entry points, from the smallest (where launches and latency count) to the
largest.

A case is a dict of plain values with a "kind":

  run        a stretch of a simulation on one box between two host snapshots:
             upload, `steps` PM steps, download (nyxpm_box_upload, nyxpm_step,
             nyxpm_box_download), in the FP64 or the mixed form
  solve      Gravity::solve_for_phi alone: right-hand side, V-cycles, phi to the host
  particles  the particle container under a caller's own gravity field: time-step
             estimate, moveKickDrift, RedistributeLocal, moveKick, AssignDensity
  noalloc    the allocation-free deposit on the caller's device arrays
  ensemble   a batch of boxes of uneven sizes: upload, `steps` ensemble steps, download
  amr        a multilevel run without subcycling: upload, `steps` steps, download

`stage` says which part of a run's life the particles are in: "early" is a lattice
displaced by a fifth of a cell (a = 0.02), "late" one displaced by a cell and a half
with a tenth of the particles in a few dense clumps (a = 0.3), so that cells hold
from none to hundreds of particles.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from nyx_gb300 import _lib
from nyx_gb300.amr import AmrHierarchy
from nyx_gb300.ensemble import Ensemble, ensemble_workload
from nyx_gb300.pm import Box, Context, DarkMatterParticleContainer

# Nyx code units: Mpc, M_sun, km/s (Einstein-de Sitter, h = 0.675, the library's defaults)
G = 6.67408e-8 * 1.98848e33 * (3.0856776e24 / 1e5) ** 2 / 3.0856776e24 ** 3
H0 = 67.5
EARLY = {"a": 0.02, "disp": 0.2, "clumps": 0.0}
LATE = {"a": 0.3, "disp": 1.5, "clumps": 0.1}
DA = 0.0096           # the 256^3 workload's step in a: 0.02 -> 0.5 in 50 steps


def listed():
    return [
        # The smallest call: a 32^3 density on a host code's own device arrays.
        {"name": "noalloc_32", "kind": "noalloc", "n": 32, "np": 32768, "stage": "early"},
        # A small FP64 run, the 32^3 grid of the reference's inputs_nohydro.rt.
        {"name": "run_fp64_32", "kind": "run", "form": "fp64", "n": 32, "np": 32768, "stage": "early",
         "steps": 10, "reuse": False, "masses": False},
        # The plain PM configuration: 64^3 particles on 64^3, ten steps.
        {"name": "run_fp64_64", "kind": "run", "form": "fp64", "n": 64, "np": 262144, "stage": "early",
         "steps": 10, "reuse": False, "masses": False},
        # The FP64 drop-in at scale, clustered, the reference's schedule (two solves per step).
        {"name": "run_fp64_256", "kind": "run", "form": "fp64", "n": 256, "np": 16777216, "stage": "late",
         "steps": 3, "reuse": False, "masses": False},
        # A mid-sized mixed run on the one-solve schedule a server uses.
        {"name": "run_mixed_64", "kind": "run", "form": "mixed", "n": 64, "np": 262144, "stage": "early",
         "steps": 20, "reuse": True, "masses": False},
        # An odd grid (5 * 2^5), half filled, unequal masses, clustered.
        {"name": "run_mixed_160", "kind": "run", "form": "mixed", "n": 160, "np": 2048001, "stage": "late",
         "steps": 4, "reuse": False, "masses": True},
        # The mixed form at scale on the reference's schedule.
        {"name": "run_mixed_256", "kind": "run", "form": "mixed", "n": 256, "np": 16777216, "stage": "early",
         "steps": 5, "reuse": False, "masses": False},
        # The Poisson solve alone, for a caller that keeps its own particles moving.
        {"name": "solve_fp64_128", "kind": "solve", "form": "fp64", "n": 128, "np": 2097152, "stage": "late"},
        # The particle container alone, under a host code's own gravity solver.
        {"name": "particles_fp64_128", "kind": "particles", "form": "fp64", "n": 128, "np": 2097153,
         "stage": "late", "masses": True},
        # A batch of sixteen boxes of 32^3 to 128^3, half of them half filled.
        {"name": "ensemble_16", "kind": "ensemble", "boxes": 16, "mix": 4, "steps": 10},
        # The reference's multilevel particle test grids (fixed_grids.mass), small.
        {"name": "amr_16", "kind": "amr", "layout": "fixed_grids", "n": 16, "np": 5596, "steps": 3},
        # The zoom-shaped multilevel workload: base 128^3 and two nested levels of 128^3.
        {"name": "amr_128", "kind": "amr", "layout": "zoom", "n": 128, "np": 2359296, "steps": 2},
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _grid(rng, lo, hi):
    """A grid the multigrid takes (m * 2^k with m in 4, 5, 6, 7), log-uniform in [lo, hi]."""
    grids = [m << k for k in range(1, 8) for m in (4, 5, 6, 7) if lo <= m << k <= hi]
    t = _log_uniform(rng, lo, hi)
    return min(sorted(grids), key=lambda g: abs(math.log(g / t)))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "solve", "particles", "noalloc", "ensemble", "amr"])
    form = rng.choice(["fp64", "mixed"])
    stage = rng.choice(["early", "late"])
    if kind == "run":
        n = _grid(rng, 16, 224)
        return {"kind": kind, "form": form, "n": n, "np": max(64, int(n ** 3 * rng.uniform(0.4, 1.0))),
                "stage": stage, "steps": rng.randint(2, 5 if n > 128 else 12),
                "reuse": rng.random() < 0.5, "masses": rng.random() < 0.3}
    if kind == "solve":
        n = _grid(rng, 16, 192)
        return {"kind": kind, "form": form, "n": n, "np": int(n ** 3 * rng.uniform(0.4, 1.0)), "stage": stage}
    if kind == "particles":
        n = _grid(rng, 16, 192)
        return {"kind": kind, "form": form, "n": n, "np": int(n ** 3 * rng.uniform(0.4, 1.0)), "stage": stage,
                "masses": rng.random() < 0.5}
    if kind == "noalloc":
        n = _grid(rng, 8, 64)
        return {"kind": kind, "n": n, "np": int(_log_uniform(rng, 64, n ** 3)), "stage": stage}
    if kind == "ensemble":
        case = {"kind": kind, "boxes": rng.randint(2, 20), "mix": rng.randint(1, 10 ** 6),
                "steps": rng.randint(2, 10)}
        while case["boxes"] > 2 and work(case)["flops"] > 7e10:   # within the listed batch's work
            case["boxes"] -= 1
        return case
    n = rng.choice([16, 24, 32, 48, 64, 80, 96])
    return {"kind": kind, "layout": "zoom", "n": n, "np": n ** 3 + int(n ** 3 * rng.uniform(0.02, 0.125)),
            "steps": rng.randint(1, 3)}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((seed * 1000003 + salt) & 0x7fffffff)
    return g


def _displacement(n, slope, gen):
    """A unit-rms Zel'dovich displacement field, shape (3, n, n, n) over (z, y, x)."""
    f64 = torch.float64
    white = torch.randn((n, n, n), generator=gen, device="cuda", dtype=f64)
    k = torch.fft.fftfreq(n, d=1.0 / n, dtype=f64, device="cuda")
    kx = torch.fft.rfftfreq(n, d=1.0 / n, dtype=f64, device="cuda")
    ks = (kx[None, None, :], k[None, :, None], k[:, None, None])
    k2 = ks[0] ** 2 + ks[1] ** 2 + ks[2] ** 2
    k2[0, 0, 0] = 1.0
    dk = torch.fft.rfftn(white) * k2 ** (0.25 * slope)
    dk[0, 0, 0] = 0.0
    psi = torch.stack([torch.fft.irfftn(1j * kd / k2 * dk, s=(n, n, n)) for kd in ks])
    return psi / psi.pow(2).sum(0).mean().sqrt()


def _particles(n, np_, stage, seed, salt=0, slope=-2.0):
    """(pos, vel, particle mass) on the GPU in a unit box: np_ of the n^3 lattice sites
    (all of them and more in clumps where np_ asks for that), displaced."""
    st = EARLY if stage == "early" else LATE
    gen = _generator(seed, salt)
    psi = _displacement(n, slope, gen).reshape(3, -1).t() * (st["disp"] / n)
    x = (torch.arange(n, device="cuda", dtype=torch.float64) + 0.5) / n
    z, y, x = torch.meshgrid(x, x, x, indexing="ij")
    pos = torch.stack([x, y, z], dim=-1).reshape(-1, 3)
    keep = min(np_, n ** 3)
    if keep < n ** 3:
        at = torch.randperm(n ** 3, generator=gen, device="cuda")[:keep].sort().values
        pos, psi = pos[at], psi[at]
    pos = pos + psi
    vel = psi * (st["a"] * H0 * st["a"] ** -1.5)
    extra = np_ - keep
    if st["clumps"]:
        m = int(st["clumps"] * keep)
        at = torch.randperm(keep, generator=gen, device="cuda")[:m]
        centre = torch.rand((6, 3), generator=gen, device="cuda", dtype=torch.float64)
        which = torch.randint(0, 6, (m,), generator=gen, device="cuda")
        pos[at] = centre[which] + 0.02 * torch.randn((m, 3), generator=gen, device="cuda", dtype=torch.float64)
    if extra:
        pos = torch.cat([pos, 0.5 + 0.1 * torch.randn((extra, 3), generator=gen, device="cuda", dtype=torch.float64)])
        sig = vel.std()
        v = sig * torch.randn((extra, 3), generator=gen, device="cuda", dtype=torch.float64)
        vel = torch.cat([vel, v.clamp(-2.5 * sig, 2.5 * sig)])
    pos = torch.remainder(pos, 1.0)
    pos[pos >= 1.0] = 0.0
    return pos.contiguous(), vel.contiguous(), 3.0 * H0 * H0 / (8.0 * math.pi * G) / np_


def _masses(np_, mass, seed):
    return mass * (0.5 + torch.rand(np_, generator=_generator(seed, 77), device="cuda", dtype=torch.float64))


def _pinned(t):
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)


def _pinned_like(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def _steps(case):
    """a_old and the step in a of the case's first step."""
    if case["kind"] == "ensemble":
        return 0.02, 0.009
    if case["kind"] == "amr":
        return 0.02, 0.0005
    a = EARLY["a"] if case["stage"] == "early" else LATE["a"]
    return a, (0.003 if case.get("n", 0) <= 64 else DA)


def _schedule(ctx, case):
    a, da = _steps(case)
    k = case.get("steps", 1)
    return ctx.step_schedule(a, a + da * k, k)


def _acceleration(case, seed, scale):
    """A host code's gravity field on the case's grid: smooth, (3, n^3) component-major."""
    n = case["n"]
    psi = _displacement(n, -3.0, _generator(seed, 31))
    return (psi.reshape(3, -1) * scale).contiguous()


# boxes of the reference's fixed_grids.mass in their own levels' index spaces
FIXED_GRIDS = [[((12, 6, 12), (25, 19, 27)), ((0, 0, 12), (7, 7, 19)), ((26, 26, 12), (31, 31, 19))],
               [((28, 20, 28), (41, 33, 37))]]


def _amr_boxes(case):
    if case["layout"] == "fixed_grids":
        return FIXED_GRIDS
    n = case["n"]
    return [[((n // 2,) * 3, (3 * n // 2 - 1,) * 3)], [((3 * n // 2,) * 3, (5 * n // 2 - 1,) * 3)]]


def _ensemble_boxes(case):
    return ensemble_workload(case["boxes"], seed=case["mix"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "noalloc":
        pos, _, mass = _particles(case["n"], case["np"], case["stage"], seed)
        x, y, z = (pos[:, d].contiguous() for d in range(3))
        return {"kind": kind, "case": case, "lib": _lib.load(), "xyz": (x, y, z), "mass": mass,
                "rho": torch.empty(case["n"] ** 3, device="cuda", dtype=torch.float64),
                "err": C.create_string_buffer(256)}
    ctx = Context(device=0)
    s = {"kind": kind, "case": case, "ctx": ctx, "sched": _schedule(ctx, case)}
    if kind == "ensemble":
        specs = _ensemble_boxes(case)
        s["ens"] = Ensemble(ctx, int(sum(1.05 * Ensemble.box_bytes(b.n, b.np) for b in specs)) + (64 << 20))
        s["boxes"] = []
        for k, b in enumerate(specs):
            pos, vel, mass = _particles(b.n, b.np, "early", seed, salt=k + 1, slope=b.slope)
            s["boxes"].append((s["ens"].add(b.n, 1.0, b.np), pos.cpu().numpy(), vel.cpu().numpy(), mass))
        return s
    pos, vel, mass = _particles(case["n"], case["np"], case.get("stage", "early"), seed)
    s["pos"], s["vel"] = _pinned(pos), _pinned(vel)
    s["mass"] = _pinned(_masses(case["np"], mass, seed)).numpy() if case.get("masses") else mass
    if kind == "amr":
        s["amr"] = AmrHierarchy(ctx, case["n"], 1.0, _amr_boxes(case), case["np"])
        s["out"] = _pinned_like((case["np"], 3)), _pinned_like((case["np"], 3))
        return s
    s["box"] = Box(ctx, case["n"], 1.0, case["np"], precision=case["form"])
    if kind == "run":
        s["out"] = _pinned_like((case["np"], 3)), _pinned_like((case["np"], 3))
    elif kind == "solve":
        s["box"].upload(s["pos"].numpy(), s["vel"].numpy(), s["mass"])
        s["box"].deposit(read_back=False)
        s["phi"] = _pinned_like(case["n"] ** 3)
    else:
        a, _, dt = s["sched"][0]
        # an acceleration that moves a particle by about half a cell in the step
        s["acc"] = _acceleration(case, seed, a * a / (dt * dt) * 0.5 / case["n"])
        s["dm"] = DarkMatterParticleContainer(s["box"])
        s["out"] = _pinned_like((case["np"], 3)), _pinned_like((case["np"], 3))
        s["rho"] = _pinned_like(case["n"] ** 3)
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    return globals()["_run_" + s["kind"]](s)


def _run_noalloc(s):
    c = s["case"]
    x, y, z = s["xyz"]
    st = s["lib"].nyxpm_deposit_noalloc(C.c_void_p(x.data_ptr()), C.c_void_p(y.data_ptr()), C.c_void_p(z.data_ptr()),
                                        c["np"], s["mass"], c["n"], 1.0, C.c_void_p(s["rho"].data_ptr()),
                                        C.c_void_p(torch.cuda.current_stream().cuda_stream), s["err"], 256)
    if st != 0:
        raise RuntimeError(s["err"].value.decode())
    return {"rho": s["rho"]}


def _run_run(s):
    box, (pos, vel) = s["box"], s["out"]
    box.upload(s["pos"].numpy(), s["vel"].numpy(), s["mass"])
    if s["case"]["reuse"]:
        box.init_field(s["sched"][0][0])
    for a_old, a_new, dt in s["sched"]:
        box.step(a_old, a_new, dt, reuse_field=s["case"]["reuse"])
    box.download_ptr(pos.data_ptr(), vel.data_ptr())
    return {"pos": pos, "vel": vel}


def _run_solve(s):
    box = s["box"]
    box.solve_phi(s["sched"][0][0], zero_guess=True)
    box.ctx.check(box.ctx.lib.nyxpm_get_phi(box.ctx.handle, box.handle, C.c_void_p(s["phi"].data_ptr())), "get_phi")
    return {"phi": s["phi"]}


def _run_particles(s):
    box, dm, (pos, vel) = s["box"], s["dm"], s["out"]
    a_old, a_new, dt = s["sched"][0]
    a_half = 0.5 * (a_old + a_new)
    dm.InitFromArrays(s["pos"].numpy(), s["vel"].numpy(), s["mass"])
    limit = dm.estTimestep(s["acc"], a_old)
    dm.moveKickDrift(None, 0, dt, a_old, a_half)
    dm.RedistributeLocal()
    dm.moveKick(s["acc"], 0, dt, a_new, a_half)
    box.ctx.check(box.ctx.lib.nyxpm_deposit(box.ctx.handle, box.handle, C.c_void_p(s["rho"].data_ptr())), "deposit")
    box.download_ptr(pos.data_ptr(), vel.data_ptr())
    return {"pos": pos, "vel": vel, "rho": s["rho"], "dt": limit}


def _run_ensemble(s):
    ens = s["ens"]
    for slot, pos, vel, mass in s["boxes"]:
        ens.upload(slot, pos, vel, mass)
    for a_old, a_new, dt in s["sched"]:
        ens.step({b[0]: a_old for b in s["boxes"]}, {b[0]: a_new for b in s["boxes"]}, {b[0]: dt for b in s["boxes"]})
    return [ens.download(b[0]) for b in s["boxes"]]


def _run_amr(s):
    amr, (pos, vel) = s["amr"], s["out"]
    amr.upload(s["pos"].numpy(), s["vel"].numpy(), s["mass"])
    for a_old, a_new, dt in s["sched"]:
        amr.step(a_old, a_new, dt)
    s["ctx"].check(amr.lib.nyxpm_amr_download(s["ctx"].handle, amr.handle, C.c_void_p(pos.data_ptr()),
                                              C.c_void_p(vel.data_ptr())), "amr_download")
    return {"pos": pos, "vel": vel}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
V_CYCLES = 8          # V(2,2) cycles to a residual of 1e-10
CYCLE_FLOPS = 60      # per cell: 4 sweeps of 7, residual, transfers, and the coarser levels
PARTICLE_FLOPS = 60   # CIC weights with either the deposit's sums or the kick's


def _step_flops(cells, np_, solves):
    return solves * V_CYCLES * CYCLE_FLOPS * cells + (solves + 2) * PARTICLE_FLOPS * np_


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        specs = _ensemble_boxes(case)
        np_ = sum(b.np for b in specs)
        cells = sum(b.n ** 3 for b in specs)
        return {"bytes": 96 * np_, "flops": _step_flops(cells, np_, 1) * case["steps"]}
    n, np_ = case["n"], case["np"]
    if kind == "noalloc":
        return {"bytes": 24 * np_ + 8 * n ** 3, "flops": PARTICLE_FLOPS * np_}
    if kind == "solve":
        width = 8 if case["form"] == "fp64" else 4
        return {"bytes": (width + 8) * n ** 3, "flops": V_CYCLES * CYCLE_FLOPS * n ** 3}
    extra = 8 * np_ if case.get("masses") else 0
    if kind == "particles":
        return {"bytes": 96 * np_ + extra + 32 * n ** 3, "flops": 3.5 * PARTICLE_FLOPS * np_}
    cells = n ** 3
    if kind == "amr":
        cells += sum(math.prod(hi[d] - lo[d] + 1 for d in range(3)) for lv in _amr_boxes(case) for lo, hi in lv)
        return {"bytes": 96 * np_, "flops": _step_flops(cells, np_, 2) * case["steps"]}
    solves = case["steps"] + 1 if case["reuse"] else 2 * case["steps"]
    return {"bytes": 96 * np_ + extra, "flops": solves * V_CYCLES * CYCLE_FLOPS * cells
            + (solves + 2 * case["steps"]) * PARTICLE_FLOPS * np_}


# ---------------------------------------------------------------------------
# the same in 64 bits, by plain torch
# ---------------------------------------------------------------------------
def _clouds(pos, n):
    """Cells (np, 8) and weights (np, 8) of the CIC clouds of positions in a unit box."""
    l = pos * n + 0.5
    i = torch.floor(l)
    f = l - i
    i = i.to(torch.int64)
    cells, weights = [], []
    for kk in (0, 1):
        for jj in (0, 1):
            for ii in (0, 1):
                at = [torch.remainder(i[:, d] - o, n) for d, o in enumerate((ii, jj, kk))]
                cells.append(at[0] + n * (at[1] + n * at[2]))
                w = [f[:, d] if o == 0 else 1.0 - f[:, d] for d, o in enumerate((ii, jj, kk))]
                weights.append(w[0] * w[1] * w[2])
    return cells, weights


def _density(pos, mass, n):
    rho = torch.zeros(n ** 3, dtype=torch.float64, device="cuda")
    for c, w in zip(*_clouds(pos, n)):
        rho.index_add_(0, c, w * mass)
    return rho * float(n) ** 3


def _potential(rho, n, a):
    """The 7-point Laplacian's solution for -4 pi G (rho - mean) / a, zero mean."""
    k = torch.arange(n, dtype=torch.float64, device="cuda") * (2.0 * math.pi / n)
    lam = (2.0 * torch.cos(k) - 2.0) * float(n) ** 2
    lam = lam[:, None, None] + lam[None, :, None] + lam[None, None, : n // 2 + 1]
    lam[0, 0, 0] = 1.0
    rk = torch.fft.rfftn((rho - rho.mean()).reshape(n, n, n) * (-4.0 * math.pi * G / a))
    rk[0, 0, 0] = 0.0
    return torch.fft.irfftn(rk / lam, s=(n, n, n))


def _gravity(phi, n):
    return torch.stack([(torch.roll(phi, -1, d) - torch.roll(phi, 1, d)).reshape(-1) * (0.5 * n) for d in (2, 1, 0)])


def _kick(pos, vel, g, n, dt, a_prev, a_cur):
    acc = torch.zeros_like(vel)
    for c, w in zip(*_clouds(pos, n)):
        for d in range(3):
            acc[:, d] += w * g[d][c]
    return (a_prev * vel + 0.5 * dt * acc) / a_cur


def _wrap(pos):
    pos = torch.remainder(pos, 1.0)
    pos[pos >= 1.0] = 0.0
    return pos


def _field(pos, mass, n, a):
    return _gravity(_potential(_density(pos, mass, n), n, a), n)


def _exact_run(pos, vel, mass, n, sched, reuse):
    g = None
    for a_old, a_new, dt in sched:
        a_half = 0.5 * (a_old + a_new)
        if g is None or not reuse:
            g = _field(pos, mass, n, a_old)
        vel = _kick(pos, vel, g, n, dt, a_old, a_half)
        pos = pos + dt / a_half * vel
        g = _field(pos, mass, n, a_new)
        vel = _kick(pos, vel, g, n, dt, a_half, a_new)
        pos = _wrap(pos)
    return pos, vel


def exact(case, seed):
    kind = case["kind"]
    if kind == "amr":
        return None   # the composite solution has no short closed form
    if kind == "noalloc":
        pos, _, mass = _particles(case["n"], case["np"], case["stage"], seed)
        return {"rho": _density(pos, mass, case["n"])}
    sched = _schedule(Context(device=0), case)
    if kind == "ensemble":
        out = []
        for k, b in enumerate(_ensemble_boxes(case)):
            pos, vel, mass = _particles(b.n, b.np, "early", seed, salt=k + 1, slope=b.slope)
            out.append(_exact_run(pos, vel, mass, b.n, sched, True))
        return out
    n = case["n"]
    pos, vel, mass = _particles(n, case["np"], case["stage"], seed)
    m = _masses(case["np"], mass, seed) if case.get("masses") else mass
    if kind == "solve":
        return {"phi": _potential(_density(pos, m, n), n, sched[0][0]).reshape(-1)}
    if kind == "run":
        pos, vel = _exact_run(pos, vel, m, n, sched, case["reuse"])
        return {"pos": pos, "vel": vel}
    a_old, a_new, dt = sched[0]
    a_half = 0.5 * (a_old + a_new)
    g = _acceleration(case, seed, a_old * a_old / (dt * dt) * 0.5 / n)
    speed = vel.abs().max(dim=1).values * (n / a_old)
    cell = torch.floor(pos * n).to(torch.int64).remainder(n)
    at = cell[:, 0] + n * (cell[:, 1] + n * cell[:, 2])
    limit = torch.minimum(0.5 / speed, 1.0 / torch.sqrt(g[:, at].pow(2).sum(0).sqrt() * n)).min()
    vel = _kick(pos, vel, g, n, dt, a_old, a_half)
    pos = _wrap(pos + dt / a_half * vel)
    vel = _kick(pos, vel, g, n, dt, a_half, a_new)
    return {"pos": pos, "vel": vel, "rho": _density(pos, m, n), "dt": float(limit)}
