"""Direct sums that evaluate each unordered pair once (7,937 to 131,072 particles) against FP64.

Sizes sit at the edges of the range, of the 256-particle j-tiles and of the i-tiles (512 to 2,048
particles), with masses and softenings equal or not. A sample of particles (tile edges among
them) is compared with an FP64 sum over all pairs; the bars are those of the other direct-sum
tests: median relative error 1e-5 (FP32), 1e-6 (MIXED), 1e-12 (FP64).
"""
import numpy as np
import pytest

import rrgsim_b200 as rg
from helpers import plummer, rel_err

pytestmark = pytest.mark.gpu

TOL_MEDIAN = {"fp32": 1e-5, "mixed": 1e-6, "fp64": 1e-12}
TOL_MAX = {"fp32": 1e-3, "mixed": 1e-3, "fp64": 1e-10}


def _case(n, form):
    pos, vel, m, s2 = plummer(n, seed=n)
    if "m" in form:
        m = m * np.where(np.arange(n) % 3 == 0, 1.7, 0.9)
        m[5::97] = 0.0
    if "s" in form:
        s2 = np.where(np.arange(n) < n // 4, 4e-4, 1e-4)
    return pos, vel, m, s2


def _sample(n):
    edges = [0, 255, 256, 511, 512, 2047, 2048, n // 2, n - 257, n - 256, n - 1]
    return np.unique(np.concatenate([edges, np.random.default_rng(n).integers(0, n, 100)]))


def _direct(pos, m, s2, at):
    acc, pot = np.empty((len(at), 3)), np.empty(len(at))
    for k, i in enumerate(at):
        d = pos - pos[i]
        inv = 1.0 / np.sqrt((d * d).sum(1) + 0.5 * (s2 + s2[i]))
        acc[k] = (m * inv ** 3) @ d
        pot[k] = -(m * inv).sum()
    return acc, pot


@pytest.mark.parametrize("prec", ["fp32", "mixed", "fp64"])
@pytest.mark.parametrize("n,form", [(7936, "ms"), (7937, ""), (8192, "ms"), (8193, "m"),
                                    (12287, "s"), (20011, "ms"), (33025, ""), (131072, "m")])
def test_each_pair_once_matches_fp64(prec, n, form):
    pos, vel, m, s2 = _case(n, form)
    at = _sample(n)
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
    # fixed-order sums: the same bits every time
    np.testing.assert_array_equal(got["acc"], again)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_reload_with_another_mass_and_size(prec):
    """Graphs recorded on one set of particles are not replayed on the next one's masses, and the
    pair slots follow the particle count."""
    sim = rg.SimParams(time_max=1.0, dt_save=0.1, dt_dynamics=1e-3, saves_without_dump=0,
                       use_wave_model=0)

    def steps(c, n, scale):
        pos, vel, m, s2 = plummer(n, seed=1)
        c.load_particles(pos, vel, scale * m, s2)
        c.precalc()
        c.calc_steps(3)
        return c.get_particles()

    with rg.Context(0, prec) as c:
        pos, vel, m, s2 = plummer(9000, seed=1)
        c.load_particles(pos, vel, m, s2)
        c.solver_init(sim)
        got = [steps(c, 9000, 1.0), steps(c, 9000, 1.125), steps(c, 16001, 1.0),
               steps(c, 600, 1.0)]
    for g, (n, scale) in zip(got, [(9000, 1.0), (9000, 1.125), (16001, 1.0), (600, 1.0)]):
        with rg.Context(0, prec) as c:
            pos, vel, m, s2 = plummer(n, seed=1)
            c.load_particles(pos, vel, scale * m, s2)
            c.solver_init(sim)
            want = steps(c, n, scale)
        for k in ("pos", "vel", "acc"):
            np.testing.assert_array_equal(g[k], want[k])


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_first_evaluation_under_capture(prec):
    """The first evaluation of a context may be one that its caller captures (in the default mode, in
    which an allocation breaks a capture); the replay gives the bits of an evaluation outside."""
    torch = pytest.importorskip("torch")
    pos, vel, m, s2 = plummer(9000, seed=3)
    with rg.Context(0, prec) as c:
        c.load_particles(pos, vel, m, s2)
        c.nbody_acceleration()
        want = c.get_particles()["acc"]
    s = torch.cuda.Stream()
    with rg.Context(0, prec) as c:
        c.load_particles(pos, vel, m, s2)
        c.synchronize()
        c.set_stream(s.cuda_stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            c.nbody_acceleration()
        with torch.cuda.stream(s):
            graph.replay()
        got = c.get_particles()["acc"]
        c.nbody_acceleration()  # outside the capture again
        again = c.get_particles()["acc"]
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(again, want)


def test_threads_with_contexts_of_their_own():
    """Eight threads that create contexts and evaluate at once get the bits of one after the other."""
    from concurrent.futures import ThreadPoolExecutor
    cases = [(prec, n) for prec in ("fp32", "mixed", "fp64") for n in (8001, 9000, 12287, 16001)]

    def acc(case):
        prec, n = case
        pos, vel, m, s2 = _case(n, "m" if n % 2 else "")
        with rg.Context(0, prec) as c:
            c.load_particles(pos, vel, m, s2)
            c.nbody_acceleration()
            return c.get_particles()["acc"]

    with ThreadPoolExecutor(8) as pool:
        got = list(pool.map(acc, cases))
    for case, g in zip(cases, got):
        np.testing.assert_array_equal(g, acc(case))
