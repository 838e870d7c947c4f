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


@pytest.mark.parametrize("n", [4000, 6000, 9000])  # one launch, ordered pairs, each pair once
def test_fp64_reciprocal_root_over_all_exponents(n):
    """Massless particles on top of one of mass 1 without softening: the potential of a particle is
    -1 / sqrt(x) of half its softening squared, with no other rounding. Within 2 ulp; the mass-1
    particle's own term at distance 0 is -inf."""
    rng = np.random.default_rng(n)
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(-1000, 1001, n))
    x[1:4] = [2.0 ** -1000, 1e300, 2.0 ** 1001]
    s2, m = 2.0 * x, np.zeros(n)
    s2[0], m[0] = 0.0, 1.0
    with rg.Context(0, "fp64") as c:
        c.load_particles(np.zeros((n, 3)), np.zeros((n, 3)), m, s2)
        c.nbody_grav()
        pot = c.get_particles()["grav"]
    assert pot[0] == -np.inf
    want = -1.0 / np.sqrt(x[1:].astype(np.longdouble))
    assert np.max(np.abs(pot[1:] - want) / np.spacing(np.abs(want.astype(np.float64)))) <= 2.0


@pytest.mark.parametrize("n", [3, 6000, 9000])
def test_fp64_potential_shows_a_particle_without_a_position(n):
    """A particle without softening has no force from itself (0 / 0), so its next position is NaN,
    and the potentials of all others show it."""
    pos, _, m, s2 = _case(n, "")
    s2 = np.array(s2)
    s2[2] = 0.0
    with rg.Context(0, "fp64") as c:
        c.load_particles(pos, np.zeros((n, 3)), m, s2)
        c.nbody_acceleration()
        c.predict_step(1e-3)
        c.nbody_grav()
        got = c.get_particles()
    assert np.flatnonzero(np.isnan(got["pos"]).any(1)).tolist() == [2]
    assert np.all(np.isnan(got["grav"]))
