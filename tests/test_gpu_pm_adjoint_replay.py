"""The PM adjoint's recorded steps (4 steps a pass and more) with odd substep counts, where the two
levels change places every step, against torch autograd, and a second pass of the same engine on
other inputs against an engine of its own."""
import pytest

from test_gpu_pm_adjoint import _case, torch_pm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("substeps,steps,every", [(5, 5, 2), (6, 4, 4), (1, 7, 3), (5, 3, 2)])
def test_recorded_steps_match_autograd(substeps, steps, every):
    torch = pytest.importorskip("torch")
    from rrgsim_b200.adjoint import PMEngine, pm_leapfrog
    pos, vel, m, grid, wave, phi, coef = _case(nx=12, n=300, substeps=substeps)
    dt = 2e-3
    t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    x0, v0, mm, ph = t(pos), t(vel), t(m), t(phi)

    def engine():
        return PMEngine(len(m), float(m.max()), grid, wave, dt, steps, "fp64", every)

    def grads(run, shift):
        xr, vr, mr = ((a + s).clone().requires_grad_(True)
                      for a, s in ((x0, shift), (v0, -shift), (mm, 0.0)))
        xN, vN = run(xr, vr, mr)
        (((xN - x0 - 1e-3) ** 2).sum(1).mean() + 0.2 * (vN ** 2).sum(1).mean()).backward()
        return xN.detach(), vN.detach(), xr.grad, vr.grad, mr.grad

    eng = engine()
    ours = lambda e: lambda x, v, q: pm_leapfrog(x, v, q, ph, ph, e)  # noqa: E731
    for shift in (0.0, 3e-3):
        got = grads(ours(eng), shift)
        alone = grads(ours(engine()), shift)
        want = grads(lambda x, v, q: torch_pm(x, v, q, ph, ph, grid, coef, dt, steps,
                                              wave.iterations), shift)
        # the deposit is exact and the gathers in a fixed order: the same states
        assert torch.equal(got[0], alone[0]) and torch.equal(got[1], alone[1])
        for a, b, c in zip(got[2:], alone[2:], want[2:]):
            assert float(torch.linalg.norm(a - b) / torch.linalg.norm(b)) <= 1e-12  # atomics' order
            assert float(torch.linalg.norm(a - c) / torch.linalg.norm(c)) <= 1e-6
