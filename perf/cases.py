"""The work that users of the framework have it do, through its public entry points.

Kinds of a case (each case is a dict of plain values):
  nbody       a Context in the direct N-body strategy: the steps up to the next save, and the save
  pm          a Context in the wave (particle-mesh) strategy: the same
  relax       the setup relaxation of the wave potential before a particle-mesh run
  ensemble    independent galaxies stepped together
  adjoint     N-body leapfrog and the gradient of a loss on its final positions (torch)
  pm_adjoint  the same through the particle-mesh step

A save is what the solver's run does at one: the save-time sync, the conservation sums and the
state read back to the host. The host arrays are FP64 in every precision; run() hands them on in
the type that the context computes in.
"""
import math

import numpy as np
import torch

import rrgsim_b200 as rg
from rrgsim_b200.adjoint import LeapfrogEngine, PMEngine, nbody_leapfrog, pm_leapfrog

DISK_HALF = 8.0        # a mesh spans +-8 disk scale lengths
DT_NBODY, DT_PM = 1e-3, 2e-3
SETUP = 300            # setup substeps of a particle-mesh run (relax: its own count)
PI = 3.14159265358979  # the solver's constant


def listed():
    return [
        # a small galaxy with a snapshot every ten steps: latency and launches count
        {"name": "nbody_4096_fp32", "kind": "nbody", "n": 4096, "precision": "fp32", "steps": 10,
         "two": False},
        # a bulge and a disk of equal particles, the direct sum at its ordinary size
        {"name": "nbody_65536_fp32", "kind": "nbody", "n": 65536, "precision": "fp32", "steps": 4,
         "two": False},
        # star and dark components (two masses, two softenings), a size that divides nothing,
        # double-float positions
        {"name": "nbody_30011_mixed", "kind": "nbody", "n": 30011, "precision": "mixed",
         "steps": 4, "two": True},
        # the same in the reference's own precision
        {"name": "nbody_20011_fp64", "kind": "nbody", "n": 20011, "precision": "fp64", "steps": 4,
         "two": True},
        # the benchmark's disk: 2^20 particles on 128^3, 20 wave substeps a step
        {"name": "pm_1m_128_fp32", "kind": "pm", "n": 1048576, "nx": 128, "precision": "fp32",
         "steps": 48, "substeps": 20},
        # a mesh that is no power of two, a ragged particle count
        {"name": "pm_300k_96_fp32", "kind": "pm", "n": 300007, "nx": 96, "precision": "fp32",
         "steps": 32, "substeps": 20},
        # the reference's own precision on a small mesh
        {"name": "pm_262144_64_fp64", "kind": "pm", "n": 262144, "nx": 64, "precision": "fp64",
         "steps": 32, "substeps": 20},
        # the largest mesh in use: more than L2 holds
        {"name": "pm_4m_256_fp32", "kind": "pm", "n": 4194304, "nx": 256, "precision": "fp32",
         "steps": 16, "substeps": 20},
        # the setup relaxation of the benchmark's mesh (thousands of substeps before each run)
        {"name": "relax_128_fp32", "kind": "relax", "n": 262144, "nx": 128, "precision": "fp32",
         "iterations": 1500},
        # galaxies of 1,024 to 16,384 particles stepped together
        {"name": "ensemble_24_fp32", "kind": "ensemble", "galaxies": 24, "nmin": 1024,
         "nmax": 16384, "steps": 10},
        # fitting initial conditions by gradient: forward and backward through 20 steps
        {"name": "adjoint_16384_fp32", "kind": "adjoint", "n": 16384, "precision": "fp32",
         "steps": 20, "every": 10},
        {"name": "pm_adjoint_262144_64_fp32", "kind": "pm_adjoint", "n": 262144, "nx": 64,
         "precision": "fp32", "steps": 10, "every": 5, "substeps": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["nbody", "nbody", "nbody", "pm", "pm", "pm", "pm", "relax", "ensemble",
                       "adjoint", "pm_adjoint"])
    if kind == "nbody":
        precision = rng.choice(["fp32", "fp32", "mixed", "fp64"])
        n = _log(rng, 512, {"fp32": 65536, "mixed": 49152, "fp64": 20000}[precision])
        return {"kind": kind, "n": n, "precision": precision, "steps": rng.randint(2, 4),
                "two": rng.random() < 0.5}
    if kind == "pm":
        precision = rng.choice(["fp32", "fp32", "fp32", "mixed", "fp64"])
        # meshes of any width, as often a multiple of eight
        nx = _log(rng, 24, 128 if precision == "fp64" else 224)
        if rng.random() < 0.5:
            nx = 8 * max(3, round(nx / 8))
        n = max(2048, min(int(nx ** 3 * rng.uniform(0.1, 1.0)), 2097152))
        return {"kind": kind, "n": n, "nx": nx, "precision": precision,
                "steps": rng.randint(4, 12), "substeps": rng.choice([7, 10, 20, 20])}
    if kind == "relax":
        nx = _log(rng, 32, 128)
        if rng.random() < 0.5:
            nx = 8 * round(nx / 8)
        return {"kind": kind, "n": _log(rng, 4096, 262144), "nx": nx,
                "precision": rng.choice(["fp32", "fp32", "fp64"]),
                "iterations": rng.randint(200, 800)}
    if kind == "ensemble":
        return {"kind": kind, "galaxies": rng.randint(4, 24), "nmin": 512,
                "nmax": rng.choice([4096, 8192, 16384]), "steps": rng.randint(4, 10)}
    precision = rng.choice(["fp32", "fp32", "fp64"])
    if kind == "adjoint":
        steps = rng.randint(5, 20)
        return {"kind": kind, "n": _log(rng, 1000, 8000 if precision == "fp64" else 16384),
                "precision": precision, "steps": steps, "every": rng.randint(2, steps)}
    nx = _log(rng, 24, 64)
    steps = rng.randint(3, 10)
    return {"kind": kind, "n": _log(rng, 10000, 262144), "nx": nx, "precision": precision,
            "steps": steps, "every": rng.randint(2, steps), "substeps": rng.choice([10, 20])}


# ------------------------------------------------------------------------------------------------
# initial conditions, FP64, from the seed alone
# ------------------------------------------------------------------------------------------------
def _uniform(gen, *shape):
    return torch.rand(*shape, generator=gen, device="cuda", dtype=torch.float64)


def _generator(seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) + 12345)
    return gen


def _isotropic(gen, n):
    z = 2.0 * _uniform(gen, n) - 1.0
    phi = 2.0 * math.pi * _uniform(gen, n)
    s = torch.sqrt(1.0 - z * z)
    return torch.stack([s * torch.cos(phi), s * torch.sin(phi), z], 1)


def _plummer(gen, n, mass=1.0, scale=1.0):
    u = _uniform(gen, n) * 0.99 + 1e-6
    r = 1.0 / torch.sqrt(u.pow(-2.0 / 3.0) - 1.0)
    pos = scale * r[:, None] * _isotropic(gen, n)
    sigma = torch.sqrt(mass / (6.0 * scale * torch.sqrt(1.0 + r * r)))
    vel = sigma[:, None] * torch.randn(n, 3, generator=gen, device="cuda", dtype=torch.float64)
    return pos, vel


def _disk(gen, n, mass=1.0):
    r = -torch.log(_uniform(gen, n).clamp_min(1e-12) * _uniform(gen, n).clamp_min(1e-12))
    r = torch.where(r > 7.5, 7.5 * _uniform(gen, n), r).clamp_min(1e-3)
    phi = 2.0 * math.pi * _uniform(gen, n)
    z = (0.1 * torch.atanh((2.0 * _uniform(gen, n) - 1.0).clamp(-1 + 1e-9, 1 - 1e-9)))
    z = z.clamp(-7.5, 7.5)
    vc = torch.sqrt(mass * (1.0 - (1.0 + r) * torch.exp(-r)) / r)
    c, s = torch.cos(phi), torch.sin(phi)
    pos = torch.stack([r * c, r * s, z], 1)
    vel = torch.stack([-vc * s, vc * c, torch.zeros_like(r)], 1)
    vel += 0.1 * vc[:, None] * torch.randn(n, 3, generator=gen, device="cuda",
                                           dtype=torch.float64)
    return pos, vel


def _nbody_ic(case, seed):
    """pos, vel, mass, soft2: a bulge and a disk; two: with their own masses and softenings."""
    gen, n = _generator(seed), case["n"]
    nb = n // 5
    pb, vb = _plummer(gen, nb, 0.2, 0.2)
    pd, vd = _disk(gen, n - nb)
    mass = torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")
    soft2 = torch.full((n,), 1e-4, dtype=torch.float64, device="cuda")
    if case["two"]:
        mass[:nb] = 0.3 / nb
        mass[nb:] = 0.7 / (n - nb)
        soft2[:nb] = 4e-4
    return torch.cat([pb, pd]), torch.cat([vb, vd]), mass, soft2


def _pm_ic(case, seed):
    gen, n = _generator(seed), case["n"]
    pos, vel = _disk(gen, n)
    return pos, vel, torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda")


def _ensemble_ic(case, seed):
    """counts, then pos, vel, mass of all galaxies and soft2 of each."""
    gen = _generator(seed)
    lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
    u = torch.linspace(0.0, 1.0, case["galaxies"], dtype=torch.float64)
    counts = torch.exp(lo + (hi - lo) * u).round().long().tolist()
    pos, vel, mass, soft2 = [], [], [], []
    for g, n in enumerate(counts):
        p, v = _plummer(gen, n) if g % 2 else _disk(gen, n)
        pos.append(p)
        vel.append(v)
        mass.append(torch.full((n,), 1.0 / n, dtype=torch.float64, device="cuda"))
        soft2.append((0.005 * (1 + g % 4)) ** 2)
    return counts, torch.cat(pos), torch.cat(vel), torch.cat(mass), np.array(soft2)


def _speed(vel):
    return 10.0 * float(torch.linalg.vector_norm(vel, dim=1).max())


def _wave(case, vel):
    """The mesh over +-8 and its wave parameters, as the benchmark sets them."""
    grid = rg.GridInfo.from_values(case["nx"], 2.0 * DISK_HALF / case["nx"], 0.0)
    wave = rg.WaveParams.make(grid.dx, diss_base=0.25 / grid.dx, wave_speed=_speed(vel),
                              iterations=case.get("substeps", 20),
                              setup_iterations=case.get("iterations", SETUP), tolerance=0.0)
    return grid, wave


def _pinned(*shape):
    return torch.empty(*shape, dtype=torch.float64, pin_memory=True).numpy()


def _f64(t):
    return t.cpu().numpy()


# ------------------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        counts, pos, vel, mass, soft2 = _ensemble_ic(case, seed)
        return {"case": case, "ens": rg.Ensemble(counts, _f64(pos), _f64(vel), _f64(mass), soft2,
                                                 DT_NBODY)}
    real = torch.float64 if case["precision"] == "fp64" else torch.float32
    if kind == "adjoint":
        gen = _generator(seed)
        pos, vel = _plummer(gen, case["n"])
        seen = pos + 0.05 * torch.randn(case["n"], 3, generator=gen, device="cuda",
                                        dtype=torch.float64)
        mass = torch.full((case["n"],), 1.0 / case["n"], dtype=torch.float64, device="cuda")
        engine = LeapfrogEngine(case["n"], DT_NBODY, case["steps"], 4e-4, case["precision"],
                                case["every"])
        x, v, m = (t.to(real).requires_grad_(True) for t in (pos, vel, mass))
        return {"case": case, "engine": engine, "in": (x, v, m), "seen": seen.to(real)}
    if kind == "pm_adjoint":
        gen = _generator(seed)
        pos, vel = _disk(gen, case["n"])
        seen = pos + 0.05 * torch.randn(case["n"], 3, generator=gen, device="cuda",
                                        dtype=torch.float64)
        mass = torch.full((case["n"],), 1.0 / case["n"], dtype=torch.float64, device="cuda")
        grid, wave = _wave(case, vel)
        engine = PMEngine(case["n"], 1.0 / case["n"], grid, wave, DT_PM, case["steps"],
                          case["precision"], case["every"])
        phi = _poisson(case["nx"], pos, mass).to(real)
        x, v, m = (t.to(real).requires_grad_(True) for t in (pos, vel, mass))
        return {"case": case, "engine": engine, "in": (x, v, m), "seen": seen.to(real),
                "phi": phi}
    # a Context
    n = case["n"]
    ctx = rg.Context(0, case["precision"])
    if kind == "nbody":
        pos, vel, mass, soft2 = _nbody_ic(case, seed)
    else:
        pos, vel, mass = _pm_ic(case, seed)
        soft2 = torch.full((n,), 1e-4, dtype=torch.float64)
    ctx.load_particles(_f64(pos), _f64(vel), _f64(mass), _f64(soft2))
    sim = rg.SimParams(time_max=1.0, dt_save=0.01,
                       dt_dynamics=DT_NBODY if kind == "nbody" else DT_PM,
                       saves_without_dump=0, use_wave_model=0 if kind == "nbody" else 1)
    if kind != "nbody":
        grid, wave = _wave(case, vel)
        ctx.init_grid(grid)
        ctx.set_wave_params(wave)
    ctx.solver_init(sim)
    if kind == "relax":
        out = {"acc": _pinned(n, 3), "grav": _pinned(n)}
    else:
        ctx.precalc()
        ctx.sync_particles_and_grid()  # (as the solver's run: the first step's accelerations)
        ctx.prepare_steps(case["steps"])
        out = {"pos": _pinned(n, 3), "vel": _pinned(n, 3)}
        if kind == "nbody":
            out |= {"acc": _pinned(n, 3), "grav": _pinned(n)}
    return {"case": case, "ctx": ctx, "out": out}


def _typed(arrays, precision):
    t = {k: torch.from_numpy(a) for k, a in arrays.items()}
    return t if precision == "fp64" else {k: a.to(torch.float32) for k, a in t.items()}


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "ensemble":
        state["ens"].step(case["steps"])
        return _typed(state["ens"].get(), "fp32")
    if kind in ("adjoint", "pm_adjoint"):
        x, v, m = state["in"]
        if kind == "adjoint":
            xn, vn = nbody_leapfrog(x, v, m, 4e-4, DT_NBODY, case["steps"],
                                    engine=state["engine"])
        else:
            xn, vn = pm_leapfrog(x, v, m, state["phi"], state["phi"], state["engine"])
        loss = ((xn - state["seen"]) ** 2).sum(1).mean()
        gx, gv, gm = torch.autograd.grad(loss, (x, v, m))
        return {"x": xn.detach(), "v": vn.detach(), "loss": loss.detach(), "gx": gx, "gv": gv,
                "gm": gm}
    ctx = state["ctx"]
    if kind == "relax":
        ctx.precalc()
        ctx.sync_particles_and_grid()
        return _typed(ctx.get_particles(out=state["out"]), case["precision"])
    ctx.calc_steps(case["steps"])
    ctx.sync_particles_and_grid()
    cons = ctx.calc_conservation()
    got = _typed(ctx.get_particles(out=state["out"]), case["precision"])
    # (the momentum and angular momentum of a galaxy at rest are rounding noise)
    return got | {"Ek": cons["Ek"], "Ep": cons["Ep"]}


# ------------------------------------------------------------------------------------------------
def work(case):
    """What a pass cannot do without. A pair: 20 operations, as the N-body literature counts; a
    force product of the backward pass: 28. A wave cell and substep: 10. Bytes: a mesh step reads
    and writes the particles and its levels once and writes the field; a relaxation reads and
    writes its levels once; what a save hands over."""
    kind, steps = case["kind"], case.get("steps", 1)
    r = 8 if case.get("precision") == "fp64" else 4
    if kind == "ensemble":
        lo, hi = math.log(case["nmin"]), math.log(case["nmax"])
        k = max(1, case["galaxies"] - 1)
        counts = [math.exp(lo + (hi - lo) * g / k) for g in range(case["galaxies"])]
        return {"bytes": sum(counts) * (48 * 2 * steps + 72),
                "flops": 20.0 * steps * sum(c * c for c in counts)}
    n = case["n"]
    if kind == "nbody":
        return {"bytes": n * (8 * r * 2 * steps + 80.0), "flops": 20.0 * n * n * (steps + 1)}
    if kind == "adjoint":
        return {"bytes": n * r * 8.0 * 4 * steps, "flops": (20.0 + 28.0) * n * n * steps}
    cells = float(case["nx"]) ** 3
    if kind == "relax":
        return {"bytes": cells * (8 + 4 * r + 4 * r) + n * 80.0,
                "flops": 10.0 * cells * case["iterations"] + 200.0 * n}
    step = {"bytes": 2 * 8 * r * n + cells * (8 + 4 * r + 4 * r),
            "flops": 10.0 * cells * case["substeps"] + 200.0 * n}
    back = 3.0 if kind == "pm_adjoint" else 1.0
    return {"bytes": back * steps * step["bytes"] + n * 48.0, "flops": back * steps * step["flops"]}


# ------------------------------------------------------------------------------------------------
# the same in plain torch, FP64
# ------------------------------------------------------------------------------------------------
def _pair_rows(xi, hi, x, m, h):
    d = x[None, :, :] - xi[:, None, :]
    inv = torch.rsqrt((d * d).sum(2) + (hi[:, None] + h[None, :]))
    k = m[None, :] * inv
    return torch.einsum("ij,ijk->ik", k * inv * inv, d), -k.sum(1)


def _direct(x, m, h, potential=False):
    rows = max(1, 1 << 25 >> max(0, (x.shape[0] - 1).bit_length()))
    acc, pot = [], []
    for i in range(0, x.shape[0], rows):
        a, p = _pair_rows(x[i:i + rows], h[i:i + rows], x, m, h)
        acc.append(a)
        pot.append(p)
    return (torch.cat(acc), torch.cat(pot)) if potential else torch.cat(acc)


def _direct_for_grad(x, m, h):
    from torch.utils.checkpoint import checkpoint
    rows = max(1, 1 << 24 >> max(0, (x.shape[0] - 1).bit_length()))
    return torch.cat([checkpoint(lambda a, b, c, d: _pair_rows(a, b, c, d, h)[0], x[i:i + rows],
                                 h[i:i + rows], x, m, use_reentrant=False)
                      for i in range(0, x.shape[0], rows)])


def _leapfrog(x, v, a, dt, force):
    u = 2.0 * v + dt * a
    x = x + 0.5 * dt * u
    a = force(x)
    return x, 0.5 * (u + dt * a), a


def _energies(x, v, m, pot):
    return {"Ek": float(0.5 * (m * (v * v).sum(1)).sum()), "Ep": float(0.5 * (m * pot).sum())}


def _cic(nx, pos, mass):
    """Cell masses; differentiable in pos and mass."""
    dx = 2.0 * DISK_HALF / nx
    u = ((pos + DISK_HALF) / dx - 0.5).clamp(0.0, nx - 1 - 1e-6)
    i0 = torch.floor(u.detach()).long()
    i1 = torch.clamp(i0 + 1, max=nx - 1)
    f = u - i0
    w, idx = (1.0 - f, f), (i0, i1)
    grid = torch.zeros(nx ** 3, dtype=torch.float64, device=pos.device)
    for c in range(8):
        a, b, d = c & 1, (c >> 1) & 1, c >> 2
        cell = idx[a][:, 0] + nx * (idx[b][:, 1] + nx * idx[d][:, 2])
        grid = grid.index_add(0, cell, mass * w[a][:, 0] * w[b][:, 1] * w[d][:, 2])
    return grid.view(nx, nx, nx)


def _poisson(nx, pos, mass):
    """The settled potential of the particles on the mesh (fast Fourier transform, host)."""
    dx = 2.0 * DISK_HALF / nx
    rho = _cic(nx, pos.cpu(), mass.cpu()) / dx ** 3
    k = 2.0 * torch.cos(2.0 * math.pi * torch.arange(nx, dtype=torch.float64) / nx) - 2.0
    lap = (k[:, None, None] + k[None, :, None] + k[None, None, :]) / dx ** 2
    lap[0, 0, 0] = 1.0
    f = torch.fft.fftn(4.0 * PI * (rho - rho.mean())) / lap
    f[0, 0, 0] = 0.0
    return torch.fft.ifftn(f).real.contiguous().reshape(-1).cuda()


def _substeps(nx, phi, old, mgrid, c, count):
    """Damped wave substeps at wave speed c, dissipation 1 / (4 dx), half the Courant step."""
    dx = 2.0 * DISK_HALF / nx
    dt = 0.5 * dx / (c * math.sqrt(3.0))
    q = 0.25 / dx * c * dt * 0.5
    k = c * c * dt * dt / dx ** 2
    f = 4.0 * PI * (mgrid / dx ** 3 - 1.0 / (2.0 * DISK_HALF) ** 3)
    f = -c * c * dt * dt / (1 + q) * f
    for _ in range(count):
        lap = torch.roll(phi, 1, 0) + torch.roll(phi, -1, 0)
        for axis in (1, 2):
            lap = lap + torch.roll(phi, 1, axis) + torch.roll(phi, -1, axis)
        new = k / (1 + q) * lap + 2 * (1 - 3 * k) / (1 + q) * phi + (q - 1) / (1 + q) * old + f
        phi, old = new, phi
    return phi, old


def _field(nx, phi):
    """Cell accelerations: central differences, one-sided at the faces."""
    dx, out = 2.0 * DISK_HALF / nx, []
    for axis in (2, 1, 0):
        p = phi.movedim(axis, 0)
        g = torch.cat([(p[1] - p[0])[None], 0.5 * (p[2:] - p[:-2]), (p[-1] - p[-2])[None]])
        out.append((-g / dx).movedim(0, axis).reshape(-1))
    return torch.stack(out, 1)


def _interp(nx, field, pos):
    f = (pos + DISK_HALF) / (2.0 * DISK_HALF / nx) - 0.5
    a = torch.floor(f.detach().to(torch.float32)).long()
    frac = f - a
    w, idx = (1.0 - frac, frac), (a.clamp(0, nx - 1), (a + 1).clamp(0, nx - 1))
    acc = 0.0
    for c in range(8):
        i, j, k = c & 1, (c >> 1) & 1, c >> 2
        cell = idx[i][:, 0] + nx * (idx[j][:, 1] + nx * idx[k][:, 2])
        acc = acc + (w[i][:, 0] * w[j][:, 1] * w[k][:, 2])[:, None] * field[cell]
    return acc


def _nearest_phi(nx, phi, pos):
    cell = ((pos + DISK_HALF) / (2.0 * DISK_HALF / nx)).long().clamp(0, nx - 1)
    return phi.reshape(-1)[cell[:, 0] + nx * (cell[:, 1] + nx * cell[:, 2])]


def exact(case, seed):
    kind = case["kind"]
    if kind == "nbody":
        x, v, m, soft2 = _nbody_ic(case, seed)
        h = 0.5 * soft2
        a = _direct(x, m, h)
        for _ in range(case["steps"]):
            x, v, a = _leapfrog(x, v, a, DT_NBODY, lambda p: _direct(p, m, h))
        pot = _direct(x, m, h, True)[1]
        return {"pos": x, "vel": v, "acc": a, "grav": pot} | _energies(x, v, m, pot)
    if kind == "ensemble":
        counts, pos, vel, mass, soft2 = _ensemble_ic(case, seed)
        got, at = [], 0
        for g, n in enumerate(counts):
            x, v, m = pos[at:at + n], vel[at:at + n], mass[at:at + n]
            h = torch.full((n,), 0.5 * soft2[g], dtype=torch.float64, device="cuda")
            a = _direct(x, m, h)
            for _ in range(case["steps"]):
                x, v, a = _leapfrog(x, v, a, DT_NBODY, lambda p: _direct(p, m, h))
            got.append((x, v, a))
            at += n
        return {k: torch.cat([t[i] for t in got]) for i, k in enumerate(("pos", "vel", "acc"))}
    if kind == "adjoint":
        gen = _generator(seed)
        pos, vel = _plummer(gen, case["n"])
        seen = pos + 0.05 * torch.randn(case["n"], 3, generator=gen, device="cuda",
                                        dtype=torch.float64)
        h = torch.full((case["n"],), 2e-4, dtype=torch.float64, device="cuda")
        m = torch.full((case["n"],), 1.0 / case["n"], dtype=torch.float64, device="cuda")
        x0, v0, m = (t.requires_grad_(True) for t in (pos, vel, m))
        x, v, a = x0, v0, _direct_for_grad(x0, m, h)
        for _ in range(case["steps"]):
            x, v, a = _leapfrog(x, v, a, DT_NBODY, lambda p: _direct_for_grad(p, m, h))
    else:
        nx = case["nx"]
        if kind == "pm_adjoint":
            gen = _generator(seed)
            pos, vel = _disk(gen, case["n"])
            seen = pos + 0.05 * torch.randn(case["n"], 3, generator=gen, device="cuda",
                                            dtype=torch.float64)
            m = torch.full((case["n"],), 1.0 / case["n"], dtype=torch.float64, device="cuda")
            speed = _speed(vel)
            phi = _poisson(nx, pos, m).view(nx, nx, nx)
            old = phi
            pos, vel, m = (t.requires_grad_(True) for t in (pos, vel, m))
        else:
            pos, vel, m = _pm_ic(case, seed)
            speed = _speed(vel)
            old = torch.zeros(nx, nx, nx, dtype=torch.float64, device="cuda")
            phi, old = _substeps(nx, old, old, _cic(nx, pos, m), speed,
                                 case.get("iterations", SETUP))
        x0, v0 = pos, vel
        x, v, a = x0, v0, _interp(nx, _field(nx, phi), x0)
        if kind == "relax":
            return {"acc": a, "grav": _nearest_phi(nx, phi, x)}
        for _ in range(case["steps"]):
            u = 2.0 * v + DT_PM * a
            x = x + 0.5 * DT_PM * u
            phi, old = _substeps(nx, phi, old, _cic(nx, x, m), speed, case["substeps"])
            a = _interp(nx, _field(nx, phi), x)
            v = 0.5 * (u + DT_PM * a)
        if kind == "pm":
            return {"pos": x, "vel": v} | _energies(x, v, m, _nearest_phi(nx, phi, x))
    loss = ((x - seen) ** 2).sum(1).mean()
    gx, gv, gm = torch.autograd.grad(loss, (x0, v0, m))
    return {"x": x.detach(), "v": v.detach(), "loss": loss.detach(), "gx": gx, "gv": gv, "gm": gm}
