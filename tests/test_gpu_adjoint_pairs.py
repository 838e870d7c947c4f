"""The FP32 N-body adjoint on the sizes that evaluate each pair once (7,937 to 131,072 particles):
gradients against the FP64 adjoint of the same loss, with equal and unequal masses and softenings,
with and without the mass gradient, checkpoints that make the reversed steps run and not."""
import numpy as np
import pytest

from helpers import plummer

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from rrgsim_b200.adjoint import LeapfrogEngine, nbody_leapfrog  # noqa: E402


@pytest.mark.parametrize("n,form,every,mass_grad", [
    (7936, "ms", 3, True), (7937, "", 3, True), (8193, "m", 1, True), (8192, "s", 5, False),
    (12289, "ms", 5, True), (20011, "", 2, False)])
def test_fp32_gradient_matches_fp64(n, form, every, mass_grad):
    pos, vel, m, s2 = plummer(n, seed=n, soft=0.02)
    if "m" in form:
        m = m * np.where(np.arange(n) % 3 == 0, 1.7, 0.9)
    if "s" in form:
        s2 = np.where(np.arange(n) < n // 4, 9e-4, 4e-4)
    # the states that FP32 holds, so that both precisions differentiate at the same point
    pos, vel, m = (np.asarray(a, np.float32).astype(np.float64) for a in (pos, vel, m))
    steps, dt = 5, 1e-3
    seen = pos + 0.05 * np.random.default_rng(n).standard_normal(pos.shape)
    got = []
    for prec, dtype in (("fp32", torch.float32), ("fp64", torch.float64)):
        eng = LeapfrogEngine(n, dt, steps, s2, prec, every)
        t = lambda a: torch.tensor(a, dtype=dtype, device="cuda")  # noqa: E731
        x, v, mm = t(pos).requires_grad_(True), t(vel).requires_grad_(True), t(m)
        if mass_grad:
            mm.requires_grad_(True)
        xn, vn = nbody_leapfrog(x, v, mm, s2, dt, steps, engine=eng)
        loss = ((xn - t(seen)) ** 2).sum(1).mean() + 0.1 * (vn ** 2).sum(1).mean()
        loss.backward()
        got.append([a.grad.double() for a in (x, v)] + ([mm.grad.double()] if mass_grad else []))
    # the direct sums' FP32 bar (1e-5 an evaluation), over ten products and sums of them
    for a, b in zip(*got):
        assert float(torch.linalg.norm(a - b) / torch.linalg.norm(b)) <= 1e-4
