"""Plans without Picard iterations (``max_picard_iter = 0``): the step is the
initial guess, no evaporation is formed, and a warm start that was loaded serves
the first step only (``q_evap_old`` becomes the evaporation of a loop that did
not run, which is none). Every form of a plan against the oracle to 1e-10."""
import numpy as np
import pytest

from conftest import make_context, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(24, 16, 5), (64, 32, 6), (128, 72, 4), (300, 200, 4)])
@pytest.mark.parametrize("volume", [False, True])
def test_loaded_warm_start_serves_one_step(nx, ny, nz, volume):
    from oracle.sgh_oracle import OracleSolver
    from spectral_galerkin_heat_b200 import B200SpectralSolver, workloads
    from spectral_galerkin_heat_b200.laser import StraightTrack
    size = (nx * 3e-5, ny * 3e-5, 2e-4)
    if volume:
        cfg, path = workloads.nonlinear_raster(nx, ny, nz, steps=3, size=size, cap=0)
    else:
        cfg, _ = workloads.straight_track(nx=nx, ny=ny, nz=nz, steps=3, size=size)
        cfg["simulation"]["max_picard_iter"] = 0
        path = StraightTrack(0.4 * size[0], 0.45 * size[1], 0.8, 0.3, 120.0)
    ctx = make_context(cfg, path)
    q = 1e8 * np.random.default_rng(nx).random((ny, nx))
    o = OracleSolver(ctx)
    o.initialize()
    o.q_evap_old = q.copy()
    import torch
    s = B200SpectralSolver(None, ctx)
    s.initialize()
    s.state.q_evap_old.copy_(torch.from_numpy(q))
    for k in range(3):
        o.step(k * ctx.num.dt, ctx.num.dt)
        _, m = s.step(k * ctx.num.dt, ctx.num.dt)
        assert m["n_evap_iter"] == 0
        assert np.array_equal(s.state.q_evap_old.cpu().numpy(), o.q_evap_old)
        assert rel_l2(s.state.a.cpu().numpy(), o.a) < 1e-10
    s.finalize()
