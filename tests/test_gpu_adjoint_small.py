"""N-body adjoint below the sizes that evaluate each pair once: FP32 products in j-chunks shorter than
a tile, FP64 tile pairs in parts, against torch autograd on the dense FP64 leapfrog."""
import numpy as np
import pytest

from helpers import plummer

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from rrgsim_b200.adjoint import LeapfrogEngine, nbody_leapfrog  # noqa: E402


def _dense(x, v, m, s2, dt, steps):
    def acc(x):
        d = x[None] - x[:, None]
        r2 = (d ** 2).sum(2) + 0.5 * (s2[None] + s2[:, None])
        return (m[None, :, None] * d * (r2 ** -1.5)[..., None]).sum(1)
    a = acc(x)
    for _ in range(steps):
        x = x + dt * v + 0.5 * dt * dt * a
        b = acc(x)
        v, a = v + 0.5 * dt * (a + b), b
    return x, v


@pytest.mark.parametrize("n", [1, 3, 31, 33, 255, 257, 513, 1000, 2051, 3073])
@pytest.mark.parametrize("prec,form", [("fp32", ""), ("fp32", "ms"), ("fp64", ""), ("fp64", "ms")])
def test_gradient_matches_dense_autograd(n, prec, form):
    pos, vel, m, s2 = plummer(n, seed=n, soft=0.02)
    if "m" in form:
        m = m * np.where(np.arange(n) % 3 == 0, 1.7, 0.9)
    if "s" in form:
        s2 = np.where(np.arange(n) < n // 4, 9e-4, 4e-4)
    pos, vel, m = (np.asarray(a, np.float32).astype(np.float64) for a in (pos, vel, m))
    steps, dt = 4, 1e-3
    t = lambda a, d=torch.float64: torch.tensor(a, dtype=d, device="cuda")  # noqa: E731
    seen = t(pos + 0.05 * np.random.default_rng(n).standard_normal(pos.shape))
    out = []
    for ours in (True, False):
        dt_ = torch.float32 if ours and prec == "fp32" else torch.float64
        x, v, mm = (t(a, dt_).requires_grad_(True) for a in (pos, vel, m))
        if ours:
            eng = LeapfrogEngine(n, dt, steps, s2, prec, 4)
            xn, vn = nbody_leapfrog(x, v, mm, s2, dt, steps, engine=eng)
        else:
            xn, vn = _dense(x, v, mm, t(s2), dt, steps)
        loss = ((xn.double() - seen) ** 2).sum(1).mean() + 0.1 * (vn.double() ** 2).sum(1).mean()
        loss.backward()
        out.append([a.grad.double() for a in (x, v, mm)])
    # FP32: the direct sums' bar (1e-5 an evaluation) over eight products and sums of them
    tol = 1e-4 if prec == "fp32" else 1e-10
    for a, b in zip(*out):
        assert float(torch.linalg.norm(a - b)) <= tol * float(torch.linalg.norm(b)) + 1e-30
