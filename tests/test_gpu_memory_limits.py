"""What runs when the device's memory is nearly full: the pair slots of the direct sums, the adjoint
and the ensemble give way to the ordered kernels, and a load or a grid that does not fit leaves a
context that says so instead of one that runs on what is left of it."""
from contextlib import contextmanager

import numpy as np
import pytest

import rrgsim_b200 as rg
from helpers import disk, plummer, rel_err
from test_gpu_direct_sym import TOL_MAX, TOL_MEDIAN, _direct, _sample

pytestmark = pytest.mark.gpu


@contextmanager
def memory_left(mb):
    """All but about `mb` MB of the device's memory held by someone else."""
    from cuda.bindings import runtime as cudart
    ok = cudart.cudaError_t.cudaSuccess
    held = []
    try:
        part = 1 << 62
        while True:
            part = min(part, cudart.cudaMemGetInfo()[1] - (mb << 20))
            if part < 2 << 20:
                break
            err, p = cudart.cudaMalloc(part)
            if err == ok:
                held.append(p)
            else:
                cudart.cudaGetLastError()
                part //= 2
        yield
    finally:
        for p in held:
            cudart.cudaFree(p)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_direct_sum_without_room_for_pair_slots(prec):
    n = 131072
    pos, vel, m, s2 = plummer(n, seed=4)

    def forces(c):
        c.load_particles(pos, vel, m, s2)
        c.nbody_acceleration()
        return c.get_particles()["acc"]

    with rg.Context(0, prec) as c:
        pairs = forces(c)
    with rg.Context(0, prec) as c:
        # the ordered kernels once, one particle above the pair form's range
        p, v, mm, ss = plummer(n + 1, seed=4)
        c.load_particles(p, v, mm, ss)
        c.nbody_acceleration()
        c.get_particles()
        with memory_left(100):
            got = forces(c)
    at = _sample(n)
    err = rel_err(got[at], _direct(pos, m, s2, at)[0])
    assert np.median(err) <= TOL_MEDIAN[prec] and np.max(err) <= TOL_MAX[prec]
    assert not np.array_equal(got, pairs)  # the other form


def test_adjoint_without_room_for_pair_slots():
    """The ordered product's gradient against the pair form's: FP32 sums of at most 256 terms."""
    torch = pytest.importorskip("torch")
    from rrgsim_b200.adjoint import LeapfrogEngine, nbody_leapfrog
    pos, vel, m, s2 = plummer(131072, seed=4)

    def gradient(n):
        t = lambda a: torch.tensor(a[:n], dtype=torch.float32, device="cuda")  # noqa: E731
        x, v, mm = (t(a).requires_grad_(True) for a in (pos, vel, m))
        engine = LeapfrogEngine(n, 1e-3, 2, 1e-4, "fp32", 2)
        xn, _ = nbody_leapfrog(x, v, mm, 1e-4, 1e-3, 2, engine=engine)
        return torch.autograd.grad(((xn - 1.0) ** 2).sum(1).mean(), (x, v, mm))

    want = [g.cpu() for g in gradient(131072)]
    gradient(6000)  # the ordered kernels once
    with memory_left(160):
        got = [g.cpu() for g in gradient(131072)]
    assert not all(torch.equal(a, b) for a, b in zip(got, want))  # the other form
    for a, b in zip(got, want):
        assert float(torch.linalg.norm(a - b) / torch.linalg.norm(b)) <= 256 * 2.0 ** -24


def test_ensemble_without_room_for_pair_slots():
    n = 131072
    pos, vel, m, s2 = plummer(n, seed=4)

    def create():
        return rg.Ensemble([n], pos, vel, m, s2[:1], 1e-3)

    with create() as e:
        e.get()
    with memory_left(100):
        with create() as e:
            tuned, got = e.tuning(), e.get()["acc"]
    assert tuned["variant"] in (1, 2) and tuned["jchunk"] >= 8192
    at = _sample(n)
    err = rel_err(got[at], _direct(pos, m, s2, at)[0])
    assert np.median(err) <= 1e-5 and np.max(err) <= 1e-3


@pytest.mark.parametrize("wave", [0, 1])
def test_a_load_that_does_not_fit_leaves_no_particles(wave):
    sim = rg.SimParams(time_max=1.0, dt_save=0.1, dt_dynamics=1e-3, saves_without_dump=0,
                       use_wave_model=wave)
    small, big = disk(2000, seed=1), disk(1 << 20, seed=2)
    with rg.Context(0, "fp32") as c:
        c.load_particles(*big)
        c.get_particles()  # (the staging buffer has its size)
        c.load_particles(*small)
        g = rg.GridInfo.from_values(32, 0.5, 0.0)
        c.init_grid(g)
        c.set_wave_params(rg.WaveParams.make(g.dx, diss_base=0.5, wave_speed=8.0, iterations=4,
                                             setup_iterations=4))
        c.solver_init(sim)
        c.precalc()
        c.calc_steps(2)
        want = c.get_particles()
        with memory_left(50):
            with pytest.raises(rg.RRGError):
                c.load_particles(*big)
            for call in (lambda: c.calc_steps(2), lambda: c.prepare_steps(2), c.precalc, c.resume,
                         c.sync_particles_and_grid, c.nbody_acceleration, c.get_particles):
                with pytest.raises(rg.RRGError):
                    call()
        c.load_particles(*small)
        c.init_grid(g)
        c.precalc()
        c.calc_steps(2)
        got = c.get_particles()
    for k in ("pos", "vel"):
        np.testing.assert_array_equal(got[k], want[k])


def test_a_grid_that_does_not_fit_leaves_no_grid():
    sim = rg.SimParams(time_max=1.0, dt_save=0.1, dt_dynamics=1e-3, saves_without_dump=0,
                       use_wave_model=1)
    small, large = (rg.GridInfo.from_values(nx, 16.0 / nx, 0.0) for nx in (32, 192))
    with rg.Context(0, "fp32") as c:
        c.load_particles(*disk(2000, seed=1))

        def steps():
            c.init_grid(small)
            c.precalc()
            c.calc_steps(2)
            return c.get_particles()["pos"]

        c.init_grid(small)
        c.set_wave_params(rg.WaveParams.make(small.dx, diss_base=0.5, wave_speed=8.0, iterations=4,
                                             setup_iterations=4))
        c.solver_init(sim)
        c.precalc()
        c.calc_steps(2)
        with memory_left(50):
            with pytest.raises(rg.RRGError):
                c.init_grid(large)
            for call in (lambda: c.calc_steps(2), lambda: c.prepare_steps(2), c.precalc, c.resume,
                         c.sync_particles_and_grid, c.convert_particles_to_grid,
                         c.calc_acceleration_field):
                with pytest.raises(rg.RRGError):
                    call()
        c.load_particles(*disk(2000, seed=1))
        a = steps()
        c.load_particles(*disk(2000, seed=1))
        np.testing.assert_array_equal(a, steps())
