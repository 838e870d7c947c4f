"""Downloads in the caller's order from particles sorted by cell, around whole blocks of 256: the
same bits as without sorting, and the masses' and softenings' order with them."""
import numpy as np
import pytest

import rrgsim_b200 as rg
from helpers import disk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 1000, 5121])
def test_sorted_download_equals_unsorted(prec, n):
    pos, vel, m, s2 = disk(n, seed=n)
    g = rg.GridInfo.from_values(12, 16.0 / 12, 0.0)
    wp = rg.WaveParams.make(g.dx, diss_base=1.0 / (4 * g.dx), wave_speed=9.0, iterations=3,
                            setup_iterations=5, steady_check_step=1000)
    sim = rg.SimParams(time_max=1.0, dt_save=0.1, dt_dynamics=2e-3, saves_without_dump=2 ** 63,
                       use_wave_model=1)
    out = []
    for interval in (0, 1):
        with rg.Context(0, prec) as c:
            c.load_particles(pos, vel, m, s2)
            c.init_grid(g)
            c.set_sort_interval(interval)
            c.set_wave_params(wp)
            c.solver_init(sim)
            c.precalc()
            c.calc_steps(3)
            out.append(c.get_particles())
    for k in ("pos", "vel", "acc", "grav"):
        np.testing.assert_array_equal(out[0][k], out[1][k])
    assert np.max(np.abs(out[1]["pos"] - pos)) < 0.1  # (the caller's order, not another)
