"""The particle-mesh adjoint on enough particles and steps that it sorts them by cell: results and
gradients come back in the caller's order, against torch autograd, also when the object runs a
second set of particles in another order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from rrgsim_b200.adjoint import PMEngine, pm_leapfrog  # noqa: E402
from test_gpu_pm_adjoint import _case, torch_pm  # noqa: E402


@pytest.mark.parametrize("n,steps", [(65536, 4), (87381, 3), (87382, 3)])  # both sides of 2^18
def test_sorted_particles_match_autograd(n, steps):
    pos, vel, m, grid, wave, phi, coef = _case(nx=16, n=n, substeps=5)
    m = m * np.linspace(0.5, 1.5, n)
    dt = 2e-3
    t = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    x0, v0, mm, ph = t(pos), t(vel), t(m), t(phi)
    eng = PMEngine(n, float(m.max()), grid, wave, dt, steps, "fp64", 2)
    order = torch.randperm(n, generator=torch.Generator().manual_seed(n)).cuda()
    first = None
    for pick in (torch.arange(n, device="cuda"), order):
        grads = []
        for ours in (True, False):
            xr, vr, mr = (a[pick].clone().requires_grad_(True) for a in (x0, v0, mm))
            if ours:
                xN, vN = pm_leapfrog(xr, vr, mr, ph, ph, eng)
            else:
                xN, vN = torch_pm(xr, vr, mr, ph, ph, grid, coef, dt, steps, wave.iterations)
            target = (x0 + 1e-3 * torch.sin(1e3 * x0))[pick]
            (((xN - target) ** 2).sum(1).mean() + 0.2 * (vN ** 2).sum(1).mean()).backward()
            grads.append((xN.detach(), vN.detach(), xr.grad, vr.grad, mr.grad))
        # the int64 deposit's 2^-27 per contribution
        assert torch.max(torch.abs(grads[0][0] - grads[1][0])) <= 1e-10
        for a, b in zip(grads[0][1:], grads[1][1:]):
            assert float(torch.linalg.norm(a - b) / torch.linalg.norm(b)) <= 1e-6
        if first is None:
            first = grads[0]
        else:  # forward states do not depend on the order
            assert torch.equal(first[0][pick], grads[0][0])
            assert torch.equal(first[1][pick], grads[0][1])
