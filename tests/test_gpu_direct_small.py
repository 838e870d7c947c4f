"""Direct sums of few particles in one launch (up to 32 per SM, 4,736 on B200) against FP64.

Sizes sit at the edges of the groups of 4, 8, 16 and 32 particles a block holds, of the 512
particles its warps stage at a time, and of the range; masses and softenings equal or not. The
bars are those of the other direct-sum tests. FP64 forces also over 240 orders of magnitude of
separation, where the reciprocal square root's range could show."""
import numpy as np
import pytest

import rrgsim_b200 as rg
from helpers import rel_err
from test_gpu_direct_sym import TOL_MAX, TOL_MEDIAN, _case, _direct

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("n,form", [(2, "ms"), (31, ""), (33, "m"), (511, "s"), (513, "ms"),
                                    (775, ""), (1599, "ms"), (1601, ""), (3169, "s"),
                                    (4735, "ms"), (4736, ""), (4737, "ms"), (6000, "")])
def test_few_particles_match_fp64(prec, n, form):
    pos, vel, m, s2 = _case(n, form)
    at = np.unique(np.concatenate([[0, n - 1], np.random.default_rng(n).integers(0, n, 150)]))
    with rg.Context(0, prec) as c:
        c.load_particles(pos, vel, m, s2)
        c.nbody_acceleration()
        c.nbody_grav()
        got = c.get_particles()
        c.nbody_acceleration()
        again = c.get_particles()["acc"]
    acc, pot = _direct(pos, m, s2, at)
    err = rel_err(got["acc"][at], acc)
    assert np.median(err) <= TOL_MEDIAN[prec] and np.max(err) <= TOL_MAX[prec], (np.median(err), np.max(err))
    perr = np.abs(got["grav"][at] - pot) / np.abs(pot)
    assert np.max(perr) <= TOL_MEDIAN[prec], np.max(perr)
    np.testing.assert_array_equal(got["acc"], again)


def test_fp64_force_over_the_exponent_range():
    rng = np.random.default_rng(4)
    for e in np.arange(-100, 101, 20):
        r = rng.uniform(1, 10) * 10.0 ** e
        pos = np.array([[0.0, 0.0, 0.0], [0.6 * r, -0.48 * r, 0.64 * r]])
        s2 = np.full(2, 0.21 * r * r)
        with rg.Context(0, "fp64") as c:
            c.load_particles(pos, np.zeros((2, 3)), np.array([2.0, 3.0]), s2)
            c.nbody_acceleration()
            got = c.get_particles()["acc"]
        d = pos[1].astype(np.longdouble)
        want = 3.0 * d / ((d * d).sum() + s2[0]) ** np.longdouble(1.5)
        # the distance's three roundings, the root's 2 ulp tripled by the cube, the products
        assert np.max(np.abs(got[0] / want - 1)) <= 16 * 2.0 ** -53
    # a particle beyond the square root of the largest double adds nothing (and no NaN)
    pos = np.array([[0.0, 0.0, 0.0], [1.0, 0.0, 0.0], [1e160, 1e160, 0.0]])
    with rg.Context(0, "fp64") as c:
        c.load_particles(pos, np.zeros((3, 3)), np.ones(3), np.full(3, 1e-4))
        c.nbody_acceleration()
        got = c.get_particles()["acc"]
    assert np.all(np.isfinite(got)) and abs(got[0, 0] - 1.0001 ** -1.5) <= 1e-14
    assert np.all(got[2] == 0.0)
