"""The operator path's wave solve in the persistent kernel (periodic FP32 / MIXED grids of 32, 64
and 128 cells) against one launch per substep: the same bits in both levels, the same stop
iteration and the same last relative difference, over runs on both sides of the shortest run that
the persistent kernel takes (8 substeps), odd and even, with and without steady checks inside."""
import numpy as np
import pytest

import rrgsim_b200 as rg
from helpers import disk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "mixed"])
@pytest.mark.parametrize("nx", [32, 64, 128])
@pytest.mark.parametrize("every,tol,runs", [(30, 0.0, [7, 8, 9, 30, 31, 32, 95]),
                                            (7, 0.0, [8, 22]), (1, 0.0, [3, 300]),
                                            (10, 3e-3, [400])])
def test_relaxation_equals_one_launch_per_substep(monkeypatch, prec, nx, every, tol, runs):
    pos, vel, m, s2 = disk(5000, seed=nx)
    g = rg.GridInfo.from_values(nx, 16.0 / nx, 0.2)
    wp = rg.WaveParams.make(g.dx, diss_base=1.0 / (4 * g.dx), wave_speed=8.0, iterations=20,
                            setup_iterations=50, tolerance=tol, steady_check_step=every)
    phi0 = -1.0 + 0.1 * np.random.default_rng(nx).standard_normal(nx ** 3)
    out = []
    for persist in ("1", "0"):
        monkeypatch.setenv("RRG_WAVE_PERSIST", persist)
        with rg.Context(0, prec) as c:
            c.load_particles(pos, vel, m, s2)
            c.init_grid(g)
            c.set_wave_params(wp)
            c.convert_particles_to_grid()
            c.set_boundary_periodic(1.0)
            c.set_grid_potential(phi0)
            got = []
            for n in runs:
                k0 = rg.kernel_launch_count()
                it, rel = c.solve_wave_equation(n)
                got.append((it, rel, *c.get_wave_state()))
                if persist == "1" and n == 95 and every == 30:
                    # one launch with its three checks
                    assert rg.kernel_launch_count() - k0 == 1
            out.append(got)
    for (it1, rel1, cur1, prev1), (it0, rel0, cur0, prev0) in zip(*out):
        assert it1 == it0 and rel1 == rel0
        np.testing.assert_array_equal(cur1, cur0)
        np.testing.assert_array_equal(prev1, prev0)
    if tol > 0:
        assert out[0][0][0] < runs[0]  # it stopped on the steady check
