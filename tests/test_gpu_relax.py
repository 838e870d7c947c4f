"""The operator path's wave solve in the persistent kernel (periodic FP32 / MIXED grids of 32, 64
and 128 cells) against one launch per substep: the same bits in both levels, the same stop
iteration and the same last relative difference, over runs on both sides of the shortest run that
the persistent kernel takes (8 substeps), odd and even, with and without steady checks inside."""
import numpy as np
import pytest

import rrgsim_b200 as rg
from helpers import disk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "mixed"])
@pytest.mark.parametrize("nx", [32, 64, 128])
@pytest.mark.parametrize("every,tol,runs", [(30, 0.0, [7, 8, 9, 30, 31, 32, 95]),
                                            (7, 0.0, [8, 22]), (1, 0.0, [3, 300]),
                                            (10, 3e-3, [400])])
def test_relaxation_equals_one_launch_per_substep(monkeypatch, prec, nx, every, tol, runs):
    pos, vel, m, s2 = disk(5000, seed=nx)
    g = rg.GridInfo.from_values(nx, 16.0 / nx, 0.2)
    wp = rg.WaveParams.make(g.dx, diss_base=1.0 / (4 * g.dx), wave_speed=8.0, iterations=20,
                            setup_iterations=50, tolerance=tol, steady_check_step=every)
    phi0 = -1.0 + 0.1 * np.random.default_rng(nx).standard_normal(nx ** 3)
    out = []
    for persist in ("1", "0"):
        monkeypatch.setenv("RRG_WAVE_PERSIST", persist)
        with rg.Context(0, prec) as c:
            c.load_particles(pos, vel, m, s2)
            c.init_grid(g)
            c.set_wave_params(wp)
            c.convert_particles_to_grid()
            c.set_boundary_periodic(1.0)
            c.set_grid_potential(phi0)
            got = []
            for n in runs:
                k0 = rg.kernel_launch_count()
                it, rel = c.solve_wave_equation(n)
                got.append((it, rel, *c.get_wave_state()))
                if persist == "1" and n == 95 and every == 30:
                    # one launch with its three checks
                    assert rg.kernel_launch_count() - k0 == 1
            out.append(got)
    for (it1, rel1, cur1, prev1), (it0, rel0, cur0, prev0) in zip(*out):
        assert it1 == it0 and rel1 == rel0
        np.testing.assert_array_equal(cur1, cur0)
        np.testing.assert_array_equal(prev1, prev0)
    if tol > 0:
        assert out[0][0][0] < runs[0]  # it stopped on the steady check


@pytest.mark.parametrize("prec,nx,kernels", [("fp32", 40, 11), ("fp64", 64, 11), ("fp32", 64, 2)])
def test_relaxation_without_a_check_adds_nothing_to_its_substeps(prec, nx, kernels):
    """A relaxation of ten substeps under capture: the source and one launch per substep (or the
    persistent one), and a cleared buffer only where the persistent kernel reads it."""
    torch = pytest.importorskip("torch")
    from cuda.bindings import runtime as cudart
    ok = cudart.cudaError_t.cudaSuccess
    pos, vel, m, s2 = disk(2000, seed=nx)
    g = rg.GridInfo.from_values(nx, 16.0 / nx, 0.2)
    s = torch.cuda.Stream()
    with rg.Context(0, prec) as c:
        c.load_particles(pos, vel, m, s2)
        c.init_grid(g)
        c.set_wave_params(rg.WaveParams.make(g.dx, diss_base=1.0 / (4 * g.dx), wave_speed=8.0))
        c.convert_particles_to_grid()
        c.set_boundary_periodic(1.0)
        c.synchronize()
        c.set_stream(s.cuda_stream)
        err, = cudart.cudaStreamBeginCapture(
            s.cuda_stream, cudart.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed)
        assert err == ok
        try:
            c.solve_wave_equation(10)
        finally:
            err, graph = cudart.cudaStreamEndCapture(s.cuda_stream)
        assert err == ok
        err, _, count = cudart.cudaGraphGetNodes(graph)
        err, nodes, count = cudart.cudaGraphGetNodes(graph, count)
        assert err == ok
        kinds = [cudart.cudaGraphNodeGetType(n)[1] for n in nodes[:count]]
        cudart.cudaGraphDestroy(graph)
    types = cudart.cudaGraphNodeType
    assert kinds.count(types.cudaGraphNodeTypeKernel) == kernels
    assert len(kinds) - kernels == (1 if nx == 64 and prec == "fp32" else 0)
