"""Wave substeps, steady check, gradient and adjoint substep on periodic grids of every row form:
rows of whole 16-byte vectors that tile a warp or do not, of two-cell vectors, of single cells,
and the narrowest grids, against the FP64 oracle and torch autograd."""
import numpy as np
import pytest

import oracle as orc
import rrgsim_b200 as rg
from helpers import disk, f32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("nx", [2, 3, 4, 5, 6, 7, 10, 12, 31, 36, 66, 100, 129, 132, 160])
def test_substeps_and_field_match_oracle(prec, nx):
    pos, vel, m, s2 = disk(3000, seed=nx)
    g = rg.GridInfo.from_values(nx, 16.0 / nx, 0.0)
    wp = rg.WaveParams.make(g.dx, diss_base=1.0 / (4 * g.dx), wave_speed=9.0,
                            steady_check_step=2, steady_hold_steps=99, tolerance=0.0)
    phi0 = -1.0 + 0.1 * np.random.default_rng(nx).standard_normal(nx ** 3)
    with rg.Context(0, prec) as c:
        c.load_particles(pos, vel, m, s2)
        c.init_grid(g)
        c.set_wave_params(wp)
        c.convert_particles_to_grid()
        c.set_boundary_periodic(1.0)
        c.set_grid_potential(phi0)
        it, rel = c.solve_wave_equation(3)  # the third substep checks
        c.calc_acceleration_field()
        got = c.get_grid()
        cur, prev = c.get_wave_state()
    assert it == 3
    og = orc.make_grid(nx, g.dx, wave_speed=9.0, diss_base=1.0 / (4 * g.dx), bc_type=1,
                       rho_mean=1.0 / 16.0 ** 3, steady_check_step=10 ** 9)
    st = orc.WaveState(nx)
    st.set_all(phi0 if prec == "fp64" else f32(phi0))
    st.solve(og, got["mass"], 3)
    # three substeps of nine roundings each on values around 1
    tol = (1e-12 if prec == "fp64" else 2e-6) * np.max(np.abs(st.curr))
    assert np.max(np.abs(cur - st.curr)) <= tol
    # the check's ratio, of this state's own levels
    want = np.max(np.abs(cur - prev)) / (np.max(np.abs(cur)) + 1e-30)
    assert abs(rel - want) <= 1e-14
    acc = orc.gradient(og, cur)
    assert np.max(np.abs(got["acc"].reshape(-1, 3) - np.asarray(acc).reshape(-1, 3))) <= tol / g.dx


@pytest.mark.parametrize("nx,every", [(9, 2), (10, 4), (14, 1), (20, 3)])
def test_adjoint_on_other_rows_matches_autograd(nx, every):
    torch = pytest.importorskip("torch")
    from rrgsim_b200.adjoint import PMEngine, pm_leapfrog
    from test_gpu_pm_adjoint import _case, torch_pm
    pos, vel, m, grid, wave, phi, coef = _case(nx=nx, n=300, substeps=6)
    steps, dt = 4, 2e-3
    t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    x0, v0, mm, ph = t(pos), t(vel), t(m), t(phi)
    eng = PMEngine(len(m), float(m.max()), grid, wave, dt, steps, "fp64", every)
    grads = []
    for ours in (True, False):
        xr, vr, mr = (a.clone().requires_grad_(True) for a in (x0, v0, mm))
        if ours:
            xN, vN = pm_leapfrog(xr, vr, mr, ph, ph, eng)
        else:
            xN, vN = torch_pm(xr, vr, mr, ph, ph, grid, coef, dt, steps, wave.iterations)
        (((xN - x0 - 1e-3) ** 2).sum(1).mean() + 0.2 * (vN ** 2).sum(1).mean()).backward()
        grads.append((xr.grad, vr.grad, mr.grad))
    for a, b in zip(*grads):
        assert float(torch.linalg.norm(a - b) / torch.linalg.norm(b)) <= 1e-6


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("nx", [32, 33, 40, 96])
@pytest.mark.parametrize("steps", [3, 4])
def test_zero_substeps_leave_the_levels_alone(prec, nx, steps):
    """Steps in a frozen potential: both levels keep their bits, and the particles follow the FP64
    context's. Bars: four roundings a step of coordinates below 8 and of velocities below 2, with
    the few roundings of the accelerations below them by dt."""
    pos, vel, m, s2 = disk(3000, seed=nx)
    g = rg.GridInfo.from_values(nx, 16.0 / nx, 0.0)
    wp = rg.WaveParams.make(g.dx, diss_base=1.0 / (4 * g.dx), wave_speed=9.0, iterations=0,
                            setup_iterations=0)
    rng = np.random.default_rng(nx)
    phi = f32(-1.0 + 0.01 * rng.standard_normal(nx ** 3))
    before = f32(phi + 0.01 * rng.standard_normal(nx ** 3))
    sim = rg.SimParams(time_max=1.0, dt_save=0.1, dt_dynamics=2e-3, saves_without_dump=0,
                       use_wave_model=1)
    got = {}
    for p in (prec, "fp64"):
        with rg.Context(0, p) as c:
            c.load_particles(f32(pos), f32(vel), m, s2)
            c.init_grid(g)
            c.set_wave_params(wp)
            c.solver_init(sim)
            c.set_wave_state(phi, before)
            c.resume()
            c.sync_particles_and_grid()
            c.calc_steps(steps)
            cur, prev = c.get_wave_state()
            got[p] = c.get_particles()
        np.testing.assert_array_equal(cur, phi)
        np.testing.assert_array_equal(prev, before)
    assert np.max(np.abs(got[prec]["pos"] - got["fp64"]["pos"])) <= steps * 4 * 2.0 ** -24 * 8
    assert np.max(np.abs(got[prec]["vel"] - got["fp64"]["vel"])) <= steps * 4 * 2.0 ** -24 * 2
