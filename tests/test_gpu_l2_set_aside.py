"""The persisting L2 set-aside: which grids take a share, and that it is given back."""
import pytest

import rrgsim_b200 as rg
from helpers import disk
from test_gpu_l2 import _window

pytestmark = pytest.mark.gpu


def test_l2_set_aside_belongs_to_the_persistent_solve_grids():
    """Grids without the persistent solve put no window on the stream, and the last context with
    one gives the process's set-aside back."""
    torch = pytest.importorskip("torch")
    from cuda.bindings import runtime as cudart
    limit = cudart.cudaLimit.cudaLimitPersistingL2CacheSize
    pos, vel, m, s2 = disk(1000, seed=5)
    for prec, nx in (("fp32", 40), ("fp32", 160), ("fp64", 64)):
        s = torch.cuda.Stream()
        with rg.Context(0, prec) as c:
            c.load_particles(pos, vel, m, s2)
            c.set_stream(s.cuda_stream)
            c.init_grid(rg.GridInfo.from_values(nx, 16.0 / nx, 0.2))
            assert _window(cudart, s.cuda_stream).num_bytes == 0
    with rg.Context(0, "fp32") as c:
        c.load_particles(pos, vel, m, s2)
        c.init_grid(rg.GridInfo.from_values(64, 0.25, 0.2))
        err, held = cudart.cudaDeviceGetLimit(limit)
        assert err == cudart.cudaError_t.cudaSuccess
        c.init_grid(rg.GridInfo.from_values(40, 0.4, 0.2))  # another grid: the window goes
    err, after = cudart.cudaDeviceGetLimit(limit)
    assert err == cudart.cudaError_t.cudaSuccess and (held == 0 or after < held)


def test_l2_set_aside_returns_to_what_the_host_had():
    """A host's own set-aside stands again once the last window is gone, is never below it while
    one lives, and does not change when the only context moves to another stream."""
    torch = pytest.importorskip("torch")
    from cuda.bindings import runtime as cudart
    kind = cudart.cudaLimit.cudaLimitPersistingL2CacheSize

    def limit():
        err, v = cudart.cudaDeviceGetLimit(kind)
        assert err == cudart.cudaError_t.cudaSuccess
        return v

    torch.cuda.init()
    old = limit()
    try:
        for mb in (0, 1, 24):  # none, below and above the window's 9.4 MB at 64^3
            assert cudart.cudaDeviceSetLimit(kind, mb << 20)[0] == cudart.cudaError_t.cudaSuccess
            host = limit()
            pos, vel, m, s2 = disk(1000, seed=5)
            s = torch.cuda.Stream()
            with rg.Context(0, "fp32") as c:
                c.load_particles(pos, vel, m, s2)
                c.init_grid(rg.GridInfo.from_values(64, 0.25, 0.2))
                held = limit()
                assert held >= host
                c.set_stream(s.cuda_stream)
                assert limit() == held
                c.init_grid(rg.GridInfo.from_values(40, 0.4, 0.2))  # no window
                assert limit() == host
                c.init_grid(rg.GridInfo.from_values(64, 0.25, 0.2))
                assert limit() == held
            assert limit() == host
    finally:
        cudart.cudaDeviceSetLimit(kind, old)
