"""Fused solves on periodic FP32 grids whose levels do not stay in L2 (three substeps per launch)
against the FP64 solve: every remainder of the substep count, odd and even numbers of launches,
rows of whole and of ragged tiles, and the level parity over successive solves."""
import numpy as np
import pytest

import rrgsim_b200 as rg
from helpers import disk, f32

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "mixed"])
@pytest.mark.parametrize("nx,counts", [(196, (5, 6)), (198, (4, 7)), (200, (8, 11)), (226, (9, 12)),
                                       (224, (20, 3))])
def test_solves_match_fp64(prec, nx, counts):
    pos, vel, m, s2 = disk(3000, seed=nx)
    pos = f32(pos)
    g = rg.GridInfo.from_values(nx, 16.0 / nx, 0.0)
    wp = rg.WaveParams.make(g.dx, diss_base=1.0 / (4 * g.dx), wave_speed=9.0,
                            steady_check_step=10 ** 6)
    phi0 = f32(-1.0 + 0.1 * np.random.default_rng(nx).standard_normal(nx ** 3))

    def run(p):
        with rg.Context(0, p) as c:
            c.load_particles(pos, vel, m, s2)
            c.init_grid(g)
            c.set_wave_params(wp)
            c.convert_particles_to_grid()
            c.set_boundary_periodic(1.0)
            c.set_grid_potential(phi0)
            for count in counts:
                c.solve_wave_and_field(count)
            return c.get_grid()["acc"], c.get_wave_state()

    (a64, w64), (a32, w32) = run("fp64"), run(prec)
    scale = np.max(np.abs(w64[0]))
    # nine roundings per substep of values no larger than the potential, two per solve at its end
    tol = (9 * sum(counts) + 4) * 2.0 ** -24 * scale
    for x, y in zip(w32, w64):
        assert np.max(np.abs(x - y)) <= tol
    # (the levels differ by far more than the tolerance: none can stand in for the other)
    assert np.max(np.abs(w64[0] - w64[1])) > 20 * tol
    assert np.max(np.abs(a32 - a64)) <= tol / g.dx
