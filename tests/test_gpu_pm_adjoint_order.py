"""The PM adjoint's scatter on particles nearly in cell order (warps of 5 to 23 runs of equal cells,
which it sorts), in order (long runs) and at random, with particles on and beyond the box's faces,
against torch autograd."""
import numpy as np
import pytest

from test_gpu_pm_adjoint import _case, torch_pm

pytestmark = pytest.mark.gpu


def _runs(cell):
    c = cell[:len(cell) // 32 * 32].reshape(-1, 32)
    return 1 + (c[:, 1:] != c[:, :-1]).sum(1)


@pytest.mark.parametrize("prec,tol", [("fp64", 1e-6), ("fp32", 5e-3)])
@pytest.mark.parametrize("nx,order", [(6, "near"), (6, "cell"), (9, "near"), (9, "random")])
def test_scatter_in_any_order_matches_autograd(prec, tol, nx, order):
    torch = pytest.importorskip("torch")
    from rrgsim_b200.adjoint import PMEngine, pm_leapfrog
    n = 1000
    pos, vel, m, grid, wave, phi, coef = _case(nx=nx, n=n, substeps=4)
    rng = np.random.default_rng(nx)
    lo, hi = grid.domain_min, grid.domain_min + nx * grid.dx
    pos[:20, 0] = rng.choice([lo - 0.3 * grid.dx, lo + 0.2 * grid.dx, hi - 0.2 * grid.dx], 20)
    cell = np.clip(np.floor((pos - lo) / grid.dx - 0.5).astype(int), -1, nx - 1) @ [1, 100, 10000]
    if order != "random":
        by = np.argsort(cell, kind="stable")
        if order == "near":  # some particles change places with the one five further
            for i in range(0, n - 5, 7):
                by[i], by[i + 5] = by[i + 5], by[i]
        pos, vel, m = pos[by], vel[by], m[by]
        runs = _runs(cell[by])
        assert order == "cell" or np.sum((runs > 4) & (runs < 24)) >= 5  # warps that sort
    steps, dt = 3, 2e-3
    out = []
    for ours in (True, False):
        real = torch.float32 if ours and prec == "fp32" else torch.float64
        t = lambda a: torch.tensor(a, dtype=real, device="cuda")  # noqa: E731
        x, v, q, ph = t(pos), t(vel), t(m), t(phi)
        x, v, q = (a.requires_grad_(True) for a in (x, v, q))
        if ours:
            eng = PMEngine(n, float(m.max()), grid, wave, dt, steps, prec, 2)
            xN, vN = pm_leapfrog(x, v, q, ph, ph, eng)
        else:
            xN, vN = torch_pm(x, v, q, ph, ph, grid, coef, dt, steps, wave.iterations)
        (((xN - t(pos) - 1e-3) ** 2).sum(1).mean() + 0.2 * (vN ** 2).sum(1).mean()).backward()
        out.append([a.grad.double() for a in (x, v, q)])
    for a, b in zip(*out):
        assert float(torch.linalg.norm(a - b) / torch.linalg.norm(b)) <= tol
