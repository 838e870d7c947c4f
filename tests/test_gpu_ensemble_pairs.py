"""The ensemble's force forms (ordered pairs, each pair once) against the FP64 oracle."""
import numpy as np
import pytest

import oracle as orc
import rrgsim_b200 as rg
from helpers import rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ngal,nmin,nmax", [(1, 1, 1), (3, 200, 700), (9, 3, 5000)])
@pytest.mark.parametrize("masses", ["equal", "spread"])
def test_every_form_of_the_forces_matches_the_oracle(ngal, nmin, nmax, masses):
    """Galaxies of a particle to several i-tiles, equal masses or not: the accelerations that the
    autotuned form (each pair once, or ordered pairs) leaves after two steps against the FP64
    oracle's direct sum at the same positions, bar 1e-5 (median)."""
    rng = np.random.default_rng(ngal)
    counts = np.unique(np.linspace(nmin, nmax, ngal).astype(np.int64))
    pos, vel, m, s2 = [], [], [], []
    for k, n in enumerate(counts):
        p, v = rg.generate_plummer(k + 1, int(n), 1.0, 1.0, 20.0)
        pos.append(p)
        vel.append(v)
        w = np.full(n, 1.0 / n)
        m.append(w if masses == "equal" else w * rng.uniform(0.5, 1.5, n))
        s2.append((0.01 * (k + 1)) ** 2)
    P, V, M = np.vstack(pos), np.vstack(vel), np.concatenate(m)
    with rg.Ensemble(counts, P, V, M, np.array(s2), 1e-3, autotune=True) as e:
        e.step(2)
        got = e.get()
    at = 0
    for k, n in enumerate(counts):
        p = got["pos"][at:at + n]
        ref = orc.direct_acc(p, M[at:at + n], np.full(n, s2[k]))
        a = got["acc"][at:at + n]
        if n == 1:
            np.testing.assert_array_equal(a, 0.0)
        else:
            assert np.median(rel_err(a, ref)) <= 1e-5
        at += n


@pytest.fixture(scope="module")
def galaxies():
    """Twelve galaxies of 700 to 16,000 particles in no order of size: far more units than blocks
    in every form, so that runs start inside units and cross i-tiles and galaxies. The reference
    accelerations of both mass forms, of the FP32 positions, masses and softenings."""
    rng = np.random.default_rng(5)
    counts = rng.permutation(np.geomspace(700, 16000, 12).astype(np.int64))
    P, V = (np.vstack(a) for a in zip(*(rg.generate_plummer(k + 1, int(n), 1.0, 1.0, 20.0)
                                        for k, n in enumerate(counts))))
    s2 = (0.01 * (1 + np.arange(12) % 3)) ** 2
    spread = rng.uniform(0.5, 1.5, len(P))
    spread[7::101] = 0.0
    masses = {"equal": 1.0 / np.repeat(counts, counts)}
    masses["spread"] = masses["equal"] * spread
    at = np.concatenate([[0], np.cumsum(counts)])
    p32 = P.astype(np.float32).astype(np.float64)
    ref = {k: np.vstack([orc.direct_acc(p32[a:b], m[a:b], np.full(b - a, s2[g]))
                         for g, (a, b) in enumerate(zip(at, at[1:]))]) for k, m in masses.items()}
    return counts, P, V, masses, s2, ref


@pytest.mark.parametrize("form", [1, 2, 3, 4])
@pytest.mark.parametrize("masses", ["equal", "spread"])
def test_each_form_with_runs_across_tiles_and_galaxies(monkeypatch, galaxies, masses, form):
    """Every particle's acceleration in each form, bars of the direct sums (median 1e-5, maximum
    1e-3), and the same bits from another ensemble, at creation and after steps (the ordered forms
    where both settled on one j-chunk)."""
    counts, P, V, m, s2, ref = galaxies
    monkeypatch.setenv("RRG_ENSEMBLE_FORM", str(form))
    got = []
    for _ in range(2):
        with rg.Ensemble(counts, P, V, m[masses], s2, 1e-3) as e:
            tuned = e.tuning()
            assert tuned["variant"] == form
            first = e.get()
            e.step(3)
            got.append((first, e.get(), tuned["jchunk"]))
    err = rel_err(got[0][0]["acc"], ref[masses])
    assert np.median(err) <= 1e-5 and np.max(err) <= 1e-3, (np.median(err), np.max(err))
    for a, b in zip(got[0][:2], got[1][:2]) if got[0][2] == got[1][2] else ():
        for k in ("pos", "vel", "acc"):
            np.testing.assert_array_equal(a[k], b[k])


def test_download_of_many_galaxies_stages_a_bounded_piece():
    """3.1 million particles in galaxies of about 1,000: the download keeps at most 80 MB on the
    device, and every particle comes back in its place."""
    pytest.importorskip("torch")
    from cuda.bindings import runtime as cudart
    counts = np.where(np.arange(3072) % 2 == 0, 1021, 1030).astype(np.int64)
    n = int(counts.sum())
    rng = np.random.default_rng(2)
    P, V = rng.standard_normal((n, 3)), rng.standard_normal((n, 3))
    with rg.Ensemble(counts, P, V, np.full(n, 1e-6), np.full(3072, 1e-4), 1e-3,
                     autotune=False) as e:
        free = cudart.cudaMemGetInfo()[1]
        got = e.get()
        assert free - cudart.cudaMemGetInfo()[1] <= 80 << 20
    np.testing.assert_array_equal(got["pos"], P.astype(np.float32))
    np.testing.assert_array_equal(got["vel"], V.astype(np.float32))
    last = slice(n - 1030, n)
    ref = orc.direct_acc(got["pos"][last], np.full(1030, 1e-6), np.full(1030, 1e-4))
    assert np.median(rel_err(got["acc"][last], ref)) <= 1e-5


def test_a_galaxy_beyond_the_pair_slots_bound():
    """One galaxy whose pair slots would take more than 4 GiB in either pair form runs in an ordered
    form."""
    n = 786_437
    P, V = rg.generate_plummer(1, n, 1.0, 1.0, 20.0)
    with rg.Ensemble([n], P, V, np.full(n, 1.0 / n), [1e-4], 1e-3) as e:
        assert e.tuning()["variant"] in (1, 2)
        got = e.get()
    for i in (0, 255, n - 1):
        d = got["pos"] - got["pos"][i]
        r = ((d * d).sum(1) + 1e-4) ** -1.5
        want = (r[:, None] * d).sum(0) / n
        assert np.linalg.norm(got["acc"][i] - want) <= 1e-3 * np.linalg.norm(want)
