#!/usr/bin/env python
"""Benchmark of the particle-mesh step (the headline workload) on B200.

Workload "pm_disk_1M_128": N = 1,048,576 exponential-disk particles (G = 1, M = 1, Rd = 1,
sech^2 z0 = 0.1, circular speed from the enclosed mass + 10% Gaussian dispersion, seed 1) on a
128^3 periodic wave grid spanning +-8 Rd; CIC deposit, damped wave potential with c = 10 vmax,
gamma = 1 / (4 dx / c), 20 substeps per step, trilinear interpolation, leapfrog dt = 2e-3; FP32.
A step = predict + deposit + 20 wave substeps + gradient + interpolation + correct.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]

Prints one JSON line. Under torchrun (N > 1) every rank runs an independent replica of the
workload (the path has no data-path collective at this size): value = all ranks' particle
steps / max-over-ranks time. `--impl reference` times the CPU restatement of the reference
kernels (FP64, OpenMP on the host cores) on the same workload.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

N_PART = 1 << 20
NX = 128
HALF = 8.0
DT = 2e-3
SUBSTEPS = 20
SEED = 1
METRIC = "PM particle-steps/s"
UNIT = "particle-steps/s"
WORKLOAD = "pm_disk_1M_128"


def peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return d.get("hbm_gbs", 6650.0), "measured", d
    return 6650.0, "fallback", {}


def make_inputs(setup_iterations: int = 20000):
    import rrgsim_b200 as rg
    pos, vel = rg.generate_exp_disk(SEED, N_PART, 1.0, 1.0, 0.1, 7.5, 7.5, 0.1, 0.0, 0.0)
    mass = np.full(N_PART, 1.0 / N_PART)
    soft2 = np.full(N_PART, 1e-4)
    grid = rg.GridInfo.from_values(NX, 2 * HALF / NX, 0.0)
    vmax = float(np.max(np.linalg.norm(vel, axis=1)))
    c = 10.0 * vmax
    wave = rg.WaveParams.make(grid.dx, diss_base=1.0 / (4 * grid.dx), wave_speed=c,
                              iterations=SUBSTEPS, setup_iterations=setup_iterations,
                              tolerance=1e-6,
                              steady_check_step=30, steady_hold_steps=3)
    sim = rg.SimParams(time_max=1e9, dt_save=1e9, dt_dynamics=DT, saves_without_dump=0,
                       use_wave_model=1)
    return pos, vel, mass, soft2, grid, wave, sim


class ClockSampler:
    """nvidia-smi clocks/throttle reasons sampled every 200 ms during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index = index
        self.proc = None
        self.lines: list[str] = []

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except FileNotFoundError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                smax.append(float(f[2]))
            except ValueError:
                continue
            for nm, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def dist_setup(gpus: int):
    if gpus <= 1 or "RANK" not in os.environ:
        return 0, 1, 0
    import datetime

    import torch
    import torch.distributed as dist
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    return dist.get_rank(), dist.get_world_size(), local


def max_over_ranks(x: float, world: int) -> float:
    if world <= 1:
        return x
    import torch
    import torch.distributed as dist
    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([x], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def barrier(world: int):
    if world > 1:
        import torch.distributed as dist
        dist.barrier()


# ------------------------------------------------------------------------------------------------
def pm_step_error(ctx, mass, grid, wave) -> dict:
    """The error of one fused step of the measured workload against the FP64 oracle: the
    context's synced state (positions, velocities, accelerations, both wave levels) is read
    back and stepped once by the oracle and once by the context; the relative error of the new
    accelerations (median and 90th percentile over particles) and of the new positions."""
    import oracle as orc
    part = ctx.get_particles()
    cur, prev = ctx.get_wave_state()
    og = orc.make_grid(grid.nx, grid.dx, bc_frac=0.0, wave_speed=wave.wave_speed,
                       diss_base=wave.diss_base, bc_type=1,
                       rho_mean=1.0 / (grid.nx * grid.dx) ** 3, steady_check_step=10 ** 9)
    st = orc.WaveState(grid.nx)
    st.bufs[0][:] = prev
    st.bufs[1][:] = cur
    orc.set_threads(os.cpu_count() or 1)
    rp, _, ra = orc.pm_steps(part["pos"], part["vel"], part["acc"], mass, og, SUBSTEPS, DT, st, 1)
    ctx.calc_steps(1)
    got = ctx.get_particles()
    ea = np.linalg.norm(got["acc"] - ra, axis=1) / np.maximum(np.linalg.norm(ra, axis=1), 1e-300)
    ep = np.linalg.norm(got["pos"] - rp, axis=1) / np.maximum(np.linalg.norm(rp, axis=1), 1e-300)
    return {"what": "one fused step from the same state vs the FP64 oracle (FP32 compute)",
            "acc_rel_median": float(np.median(ea)), "acc_rel_p90": float(np.percentile(ea, 90)),
            "pos_rel_median": float(np.median(ep)), "pos_rel_max": float(np.max(ep))}


def direct_errors(c3: dict) -> dict:
    """Median and 99th-percentile relative error of the bulge + disk initial accelerations in
    each precision against the FP64 oracle's direct sum of the same inputs."""
    import oracle as orc
    pos, m, s2 = c3.pop("inputs")
    orc.set_threads(os.cpu_count() or 1)
    ref = orc.direct_acc(pos, m, s2)
    out = {}
    for prec, acc in c3.pop("acc0").items():
        e = np.linalg.norm(acc - ref, axis=1) / np.linalg.norm(ref, axis=1)
        out[prec] = {"median": float(np.median(e)), "p99": float(np.percentile(e, 99))}
    return out


def cpu_pm_sample(state, steps: int, threads: int) -> tuple[float, str]:
    """Times `steps` PM steps of the CPU restatement (FP64, OpenMP) at full size from the given
    relaxed state; returns (particle-steps/s, sample description)."""
    import oracle as orc
    pos, vel, acc, mass, phi_prev, phi_curr, grid, wave = state
    orc.set_threads(threads)
    og = orc.make_grid(grid.nx, grid.dx, bc_frac=0.0, wave_speed=wave.wave_speed,
                       diss_base=wave.diss_base, bc_type=1,
                       rho_mean=1.0 / (grid.nx * grid.dx) ** 3, steady_check_step=10 ** 9)
    st = orc.WaveState(grid.nx)
    st.bufs[0][:] = phi_prev
    st.bufs[1][:] = phi_curr
    t0 = time.perf_counter()
    orc.pm_steps(pos, vel, acc, mass, og, SUBSTEPS, DT, st, steps)
    el = time.perf_counter() - t0
    return N_PART * steps / el, f"{steps} PM steps of the full workload (N=2^20, 128^3, 20 substeps)"


def run_reference(args):
    # rank 0 alone times the CPU implementation; it needs no collective, so no process group
    # is formed and the other ranks leave at once
    if int(os.environ.get("RANK", "0")) != 0:
        return
    world = 1
    import oracle as orc
    # the same inputs as the native arm, generated by the oracle's restatement of the disk
    # generator (the same bits), so this arm loads nothing of the product library
    pos, vel = orc.exp_disk(SEED, N_PART, 1.0, 1.0, 0.1, 7.5, 7.5, 0.1)
    mass = np.full(N_PART, 1.0 / N_PART)
    dx = 2 * HALF / NX
    wave_speed = 10.0 * float(np.max(np.linalg.norm(vel, axis=1)))
    threads = os.cpu_count() or 1
    orc.set_threads(threads)
    og = orc.make_grid(NX, dx, bc_frac=0.0, wave_speed=wave_speed, diss_base=1.0 / (4 * dx),
                       bc_type=1, rho_mean=1.0 / (NX * dx) ** 3, tolerance=1e-6,
                       steady_check_step=30, steady_hold_steps=3)
    # precalc as the reference: deposit, relax, gradient, interpolate (not timed). The
    # relaxation is cut to 60 substeps here: a step costs the same whatever the potential holds.
    st = orc.WaveState(NX)
    mg = orc.cic_fp64(pos, mass, og)
    st.solve(og, mg, 60)
    acc = orc.interp(pos, og, orc.gradient(og, st.curr))
    for _ in range(min(args.warmup, 1)):
        pos, vel, acc = orc.pm_steps(pos, vel, acc, mass, og, SUBSTEPS, DT, st, 1)
    # each step is one full PM step; the run stops after ~90 s of steps
    t0 = time.perf_counter()
    done = 0
    while done < args.steps and (done == 0 or time.perf_counter() - t0 < 90.0):
        pos, vel, acc = orc.pm_steps(pos, vel, acc, mass, og, SUBSTEPS, DT, st, 1)
        done += 1
    el = time.perf_counter() - t0
    v = N_PART * done / el
    args.steps = done
    line = {
        "impl": "reference", "metric": METRIC, "value": v, "unit": UNIT, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * el / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic", "config": {"workload": WORKLOAD, "particles": N_PART, "grid": NX,
                                        "substeps": SUBSTEPS, "dt": DT},
        "cpu_baseline": {"value": v, "unit": UNIT, "cores": threads, "kind": "port",
                         "sample": f"{args.steps} full PM steps, FP64 OpenMP restatement of "
                                   f"the reference kernels"},
        "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)
    barrier(world)


# ------------------------------------------------------------------------------------------------
def run_native(args):
    import torch

    import rrgsim_b200 as rg
    rank, world, local = dist_setup(args.gpus)
    dev = local if world > 1 else 0
    torch.cuda.set_device(dev)
    pos, vel, mass, soft2, grid, wave, sim = make_inputs(args.setup_iterations)
    stream = torch.cuda.Stream(device=dev)
    ctx = rg.Context(dev, "fp32")
    ctx.set_stream(stream.cuda_stream)
    ctx.load_particles(pos, vel, mass, soft2)
    ctx.init_grid(grid)
    ctx.set_wave_params(wave)
    if args.sort_interval is not None:
        ctx.set_sort_interval(args.sort_interval)
    ctx.solver_init(sim)
    t0 = time.perf_counter()
    ctx.precalc()
    ctx.sync_particles_and_grid()
    setup_s = time.perf_counter() - t0

    # warm-up steps, then the CUDA graphs of the timed call itself are recorded and
    # instantiated (nothing runs), so the timed region only replays them
    ctx.calc_steps(args.warmup)
    ctx.prepare_steps(args.steps)
    ctx.synchronize()

    # ---- device-timed region: K steps, inputs resident in HBM --------------------------------
    clocks = ClockSampler(dev)
    barrier(world)
    torch.cuda.synchronize()
    clocks.start()
    time.sleep(0.3)
    l0 = rg.kernel_launch_count()
    ev0 = torch.cuda.Event(enable_timing=True)
    ev1 = torch.cuda.Event(enable_timing=True)
    ev0.record(stream)
    ctx.calc_steps(args.steps)
    ev1.record(stream)
    torch.cuda.synchronize()
    launches = rg.kernel_launch_count() - l0
    clk = clocks.stop()
    barrier(world)
    el = max_over_ranks(ev0.elapsed_time(ev1) / 1e3, world)
    value = N_PART * args.steps * world / el

    # ---- dominant kernel: the persistent wave solve (source, 20 substeps, gradient in one
    # launch), timed alone on the same stream with L2 flushed before every launch ------------------
    ctx.synchronize()
    probe = rg.WaveParams.make(grid.dx, diss_base=wave.diss_base, wave_speed=wave.wave_speed,
                               iterations=SUBSTEPS, steady_check_step=10 ** 9)
    ctx.set_wave_params(probe)  # no host-synchronised steady check inside the timed launches
    flush = torch.empty(256 * 2 ** 20, dtype=torch.uint8, device=f"cuda:{dev}")
    reps = 50
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True))
          for _ in range(reps)]
    with torch.cuda.stream(stream):
        for _ in range(3):
            ctx.solve_wave_and_field(SUBSTEPS)
        for a, b in ev:
            flush.zero_()  # 256 MB > 126 MB L2
            a.record(stream)
            ctx.solve_wave_and_field(SUBSTEPS)
            b.record(stream)
    torch.cuda.synchronize()
    solve_ms = sum(a.elapsed_time(b) for a, b in ev) / reps
    cells = NX ** 3
    # Algorithmic bytes of the PM step: N * 52 B for the particles (read position 12, velocity
    # 12, mass 4; write position 12, velocity 12) + NX^3 * (20 * 16 + 16 + 12) B for the grid
    # (per substep read phi^n, phi^n-1, the source and write phi^n+1: 16 B/cell; the deposit's
    # clear and write: 8 + 8; the gradient's read of phi, 12). The solve launch does the
    # substeps, the clear and the gradient: 340 B/cell. Its substeps stay on chip and in L2, so
    # this rate may exceed the HBM copy peak; the bytes that would reach DRAM once per launch
    # with nothing kept in L2 between launches (deposit in 8, other deposit cleared 8, source
    # out 4, both levels in and out 16, field out 16: 52 B/cell; the persisting L2 window keeps
    # the deposits and levels, 40 of them, on chip) and ncu's DRAM bytes are reported beside it.
    alg_bytes = (20 * 16 + 8 + 12) * cells
    min_bytes = 52 * cells
    step_bytes = 52 * N_PART + (20 * 16 + 16 + 12) * cells
    hbm, how, pk = peaks()
    achieved = alg_bytes / (solve_ms * 1e-3) / 1e9
    # the 128^3 solve runs wave_solve_kernel, or wave_solve_tb_kernel under RRG_WAVE_TB=1
    solve_kernel = ("wave_solve_tb_kernel" if os.environ.get("RRG_WAVE_TB", "0") not in ("", "0")
                    else "wave_solve_kernel")
    traffic = None
    tf = ROOT / "profiles" / "roofline_traffic.json"
    if tf.exists():
        traffic = json.loads(tf.read_text()).get(f"{solve_kernel}_bytes_per_launch")
    # the per-substep stencil of the operator path (solve_wave_equation), for comparison: its
    # algorithmic bytes are 16 B/cell (read phi, phi_old, src; write phi_new)
    ctx.solve_wave_equation(8)
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    ctx.solve_wave_equation(400)
    e1.record(stream)
    torch.cuda.synchronize()
    sub_ms = e0.elapsed_time(e1) / 400
    del flush

    # ---- end to end through the public API with host buffers ----------------------------------
    # the same run length as the device-timed region: ICs up once, K steps each followed by a
    # read of that step's diagnostics, the final snapshot down
    k_e2e = args.steps
    ctx2 = rg.Context(dev, "fp32")
    ctx2.set_stream(stream.cuda_stream)
    pin = {k: torch.from_numpy(np.ascontiguousarray(v)).pin_memory().numpy()
           for k, v in dict(pos=pos, vel=vel, mass=mass, soft2=soft2).items()}
    ctx2.init_grid(grid)
    ctx2.set_wave_params(wave)
    # each step's last particle pass also forms the conservation sums, which the per-step
    # diagnostics read then only combine
    ctx2.set_step_sums(True)
    if args.sort_interval is not None:
        ctx2.set_sort_interval(args.sort_interval)
    ctx2.load_particles(pin["pos"], pin["vel"], pin["mass"], pin["soft2"])
    ctx2.solver_init(sim)
    ctx2.precalc()
    ctx2.sync_particles_and_grid()
    ctx2.calc_steps(2)
    ctx2.synchronize()
    # each step's diagnostics come down into pinned host memory asynchronously; the host reads
    # step k's while steps k + 1 .. k + DEPTH - 1 are queued (DEPTH slots, one CUDA event each:
    # ~10 ms of GPU work, longer than a scheduler time slice on a contended host), so a host
    # thread that the shared host deschedules for a moment does not stall the GPU. The whole leg
    # runs seven times and the median counts: it is timed on the host clock, and a shared host
    # now and then stretches a run to twice its time.
    # One event per group of 8 steps keeps the host's per-step work to the two library calls
    # and a read of that step's kinetic energy, Ek = sum m v^2 / 2 (rrg_conservation_from_sums
    # does the same); a slot is read 56-63 steps before the kernel of step k + 64 rewrites it.
    depth, group = 64, 8
    sums = torch.zeros((depth, 12), dtype=torch.float64).pin_memory().numpy()
    done = [torch.cuda.Event() for _ in range(depth // group)]
    # the final snapshot (positions and velocities, FP64, the dump's content) lands in pinned
    # host arrays
    snap = {k: torch.zeros((N_PART, 3), dtype=torch.float64).pin_memory().numpy()
            for k in ("pos", "vel")}
    e2e_runs = []
    for rep in range(10):  # the first three runs record the one-step graphs and are not counted
        barrier(world)
        t0 = time.perf_counter()
        ctx2.load_particles(pin["pos"], pin["vel"], pin["mass"], pin["soft2"])  # H2D of the ICs
        ctx2.sync_particles_and_grid()
        energies = []
        for k in range(k_e2e):
            ctx2.calc_steps(1)
            ctx2.calc_conservation_async(sums[k % depth])  # D2H of the step's diagnostics
            if (k + 1) % group == 0:
                gi = k // group
                done[gi % len(done)].record(stream)
                g = gi - (len(done) - 1)  # the oldest group in flight
                if g >= 0:
                    done[g % len(done)].synchronize()
                    for j in range(g * group, g * group + group):
                        energies.append(0.5 * float(sums[j % depth, 0]))
        ctx2.synchronize()
        for j in range(len(energies), k_e2e):
            energies.append(0.5 * float(sums[j % depth, 0]))
        ctx2.get_particles(out=snap)  # D2H of the final snapshot
        el_rep = max_over_ranks(time.perf_counter() - t0, world)
        if rep >= 3:
            e2e_runs.append(el_rep)
        assert np.isfinite(snap["pos"]).all() and all(np.isfinite(energies))
        assert len(energies) == k_e2e
    e2e_el = sorted(e2e_runs)[len(e2e_runs) // 2]
    e2e_value = N_PART * k_e2e * world / e2e_el
    h2d = N_PART * 8 * 8 / k_e2e            # pos, vel (3 x f64), mass, soft2 (f64), once
    d2h = 12 * 8 + N_PART * 6 * 8 / k_e2e   # the step's 12 sums; pos, vel (3 x f64) once
    ctx2.close()

    # ---- secondary: direct-sum throughput at N = 65,536 (Plummer, FP32) ----------------------
    direct = None
    if rank == 0:
        nd = 65536
        p, v = rg.generate_plummer(0, nd, 1.0, 1.0, 20.0)
        cd = rg.Context(dev, "fp32")
        cd.set_stream(stream.cuda_stream)
        cd.load_particles(p, v, np.full(nd, 1.0 / nd), np.full(nd, 1e-4))
        cd.nbody_acceleration()
        cd.synchronize()
        r = 10
        e0.record(stream)
        for _ in range(r):
            cd.nbody_acceleration()
        e1.record(stream)
        torch.cuda.synchronize()
        t = e0.elapsed_time(e1) / 1e3 / r
        gp = nd * nd / t / 1e9
        fp32_peak = 148 * 128 * 2 * pk.get("sm_max_mhz", 1965.0) * 1e6 / 1e12
        direct = {"n": nd, "gpairs_per_s": gp, "ms_per_eval": t * 1e3,
                  "pairs": "ordered (N^2); the kernel evaluates each unordered pair once",
                  "tflops_at_20_per_pair": gp * 20 / 1e3,
                  "frac_fp32_peak": gp * 20 / 1e3 / fp32_peak,
                  "fp32_peak_tflops": fp32_peak, "fp32_peak_kind": "nominal at sm_max_mhz"}
        cd.close()

    # ---- the secondary forms in brief (rank 0, one GPU) ---------------------------------------
    forms = None
    if rank == 0 and world == 1 and not args.no_forms:
        from rrgsim_b200.bench_forms import bench_line_forms
        forms = bench_line_forms(torch)

    # ---- CPU leg (rank 0): the oracle checks one fused step of the workload and the forms'
    # accelerations, then times a bounded sample of the workload ---------------------------------
    cpu = error = None
    if rank == 0 and not args.no_cpu:
        error = pm_step_error(ctx, mass, grid, wave)
        if forms is not None:
            forms["precision_c3"]["acc_rel_err_vs_fp64_oracle"] = direct_errors(
                forms["precision_c3"])
        part = ctx.get_particles()
        g = ctx.get_grid()
        # the CPU restatement starts from the GPU's relaxed potential (both levels)
        state = (part["pos"], part["vel"], part["acc"], mass, g["grav"], g["grav"], grid, wave)
        threads = os.cpu_count() or 1
        v_cpu, sample = cpu_pm_sample(state, args.cpu_steps, threads)
        cpu = {"value": v_cpu, "unit": UNIT, "cores": threads, "kind": "port",
               "sample": sample}
    if forms is not None:  # (arrays the CPU leg did not take)
        forms["precision_c3"].pop("inputs", None)
        forms["precision_c3"].pop("acc0", None)
    ctx.close()

    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": 1e3 * el / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic",
            "config": {"workload": WORKLOAD, "particles": N_PART, "grid": NX,
                       "substeps": SUBSTEPS, "dt": DT, "parallelism": f"replicas{world}",
                       "l2": "per-step working set ~140 MB > 126 MB L2; steps back to back; the deposit grids and wave levels (48 MB) held in a persisting L2 window",
                       "setup_s": round(setup_s, 3),
                       "sort_interval": args.sort_interval if args.sort_interval is not None
                       else "library default"},
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": h2d,
                    "d2h_bytes_per_step": d2h, "steps": k_e2e, "statistic": "median of 7 runs",
                    "runs": [N_PART * k_e2e * world / t for t in e2e_runs]},
            "gpu_launches": int(launches),
            "roofline": {"bound": "hbm", "kernel": solve_kernel, "achieved": achieved,
                         "peak": hbm, "unit": "GB/s", "frac": achieved / hbm,
                         "traffic": traffic, "peak_kind": how,
                         "ms_per_launch": solve_ms, "alg_bytes_per_launch": alg_bytes,
                         "substeps_per_launch": SUBSTEPS,
                         "l2": "256 MB written before each launch (the persisting window over the deposit grids and wave levels survives it)",
                         "dram_min_bytes_per_launch": min_bytes,
                         "dram_min_achieved": min_bytes / (solve_ms * 1e-3) / 1e9,
                         "step": {"alg_bytes": step_bytes,
                                  "achieved": step_bytes / (el / args.steps) / 1e9,
                                  "frac": step_bytes / (el / args.steps) / 1e9 / hbm},
                         "operator_substep": {"kernel": "wave_solve_kernel (relaxation form, many "
                                                        "substeps per launch)",
                                              "ms_per_substep": sub_ms,
                                              "achieved": 16 * cells / (sub_ms * 1e-3) / 1e9}},
            "cpu_baseline": cpu,
            "error_vs_fp64": error,
            "clocks": clk,
            "direct_sum": direct,
            "forms": forms,
        }
        print(json.dumps(line), flush=True)
    if world > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3000)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="native", choices=["native", "reference"])
    ap.add_argument("--cpu-steps", type=int, default=3)
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-forms", action="store_true",
                    help="skip the secondary forms (precision, ensemble, adjoint)")
    ap.add_argument("--sort-interval", type=int, default=None,
                    help="steps between re-sorts of the particles by cell (default: the library's)")
    ap.add_argument("--setup-iterations", type=int, default=20000,
                    help="cap of the initial potential relaxation (profiling runs use fewer)")
    args = ap.parse_args()
    if args.warmup < 3:
        args.warmup = 3
    if args.impl == "reference":
        run_reference(args)
    else:
        run_native(args)


if __name__ == "__main__":
    main()
