"""Bounded data waits that can only run out (no GPU fault: each wait polls a
barrier that nothing completes, 2000 times at most): the volume form's slab
kernels and the face-space cluster kernels record the error, drain their
copies and return; the step says so, and the context stays usable."""
import numpy as np
import pytest

from conftest import make_context, rel_l2

pytestmark = pytest.mark.gpu


def _raster(**kw):
    from spectral_galerkin_heat_b200 import workloads
    return make_context(*workloads.nonlinear_raster(64, 32, 16, steps=6, tol=1e-6, **kw))


@pytest.mark.parametrize("cap", [200, 0])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_slab_waits_report_a_timeout(precision, cap):
    """With and without a Picard loop (without one only the step's opening and
    closing slab kernels wait): status "tensor_core_timeout", and the loop ends at once."""
    from spectral_galerkin_heat_b200 import B200SpectralSolver
    ctx = _raster(cap=cap)
    s = B200SpectralSolver(None, ctx, precision=precision)
    s.initialize()
    dt = ctx.num.dt
    s.step(0.0, dt)
    assert s.last_status in ("converged", "capped")
    s.set_wait_limit(2000, stall_test=True)
    _, m = s.step(dt, dt)
    assert s.last_status == "tensor_core_timeout"
    assert m["n_evap_iter"] == min(cap, 1) and not m["picard_converged"]
    s.finalize()
    s = B200SpectralSolver(None, ctx, precision=precision)
    s.initialize()
    s.step(0.0, dt)
    assert s.last_status in ("converged", "capped")
    assert np.isfinite(s.state.a.cpu().numpy()).all()
    s.finalize()


def _track(nx, ny, cap):
    from spectral_galerkin_heat_b200 import workloads
    from spectral_galerkin_heat_b200.laser import StraightTrack
    size = (2e-3 * nx / 64, 1e-3 * ny / 32, 0.5e-3)
    cfg, _ = workloads.straight_track(nx=nx, ny=ny, nz=8, steps=6, size=size)
    if cap > 1:
        cfg["simulation"].update({"max_picard_iter": cap, "picard_omega": 0.1, "picard_tol": 1e-4})
    return make_context(cfg, StraightTrack(0.3 * size[0], 0.5 * size[1], 1.0, 0.0, 200.0))


@pytest.mark.parametrize("nx,ny", [(24, 16), (64, 32), (256, 128)])   # clusters of 1, 4 and 16 CTAs
def test_cluster_plan_waits_write_no_results(nx, ny):
    from spectral_galerkin_heat_b200 import B200SpectralSolver
    ctx = _track(nx, ny, cap=6)
    dt = ctx.num.dt
    s = B200SpectralSolver(None, ctx)
    s.initialize()
    s.step(0.0, dt)
    before, status = s.state.q_evap_old.cpu().numpy(), s.last_status
    s.set_wait_limit(2000, stall_test=True)
    _, m = s.step(dt, dt)
    assert s.last_status == "tensor_core_timeout" and m["n_evap_iter"] == 0 and not m["picard_converged"]
    assert np.array_equal(before, s.state.q_evap_old.cpu().numpy())
    s.finalize()
    s = B200SpectralSolver(None, ctx)
    s.initialize()
    s.step(0.0, dt)
    assert s.last_status == status
    assert np.array_equal(before, s.state.q_evap_old.cpu().numpy())
    s.finalize()


@pytest.mark.parametrize("precision,cap", [("fp64", 1), ("fp64", 6), ("mixed", 6)])
def test_cluster_batch_waits_write_no_results(precision, cap):
    """Slots on clusters of 1, 4 and 16 CTAs, side by side: error flag, no results
    written, status "nonfinite"; a fresh batch steps as before."""
    from spectral_galerkin_heat_b200 import _lib
    from spectral_galerkin_heat_b200.batch import BatchSolver
    ctxs = [_track(nx, ny, cap) for nx, ny in ((24, 16), (64, 32), (256, 128))]

    def run(steps):
        b = BatchSolver(ctxs, precision)
        for i in range(len(ctxs)):
            b.start(i, 4)
        b.step(steps)
        return b

    b = run(1)
    keep = [[b.fetch(i, k) for k in ("q_evap_old", "surface")] for i in range(len(ctxs))]
    assert b.tensor_core_error() == 0
    b.set_wait_limit(2000, stall_test=True)
    b.step(1)
    b.synchronize()
    assert b.tensor_core_error() == 1
    for i, st in enumerate(b.status()):
        assert _lib.STEP_STATUS[st.last.status] == "nonfinite" and st.last.n_iter == 0
        assert np.array_equal(keep[i][0], b.fetch(i, "q_evap_old"))
        assert np.array_equal(keep[i][1], b.fetch(i, "surface"))
    b.close()
    fresh = run(1)
    assert fresh.tensor_core_error() == 0
    for i in range(len(ctxs)):
        assert np.array_equal(keep[i][0], fresh.fetch(i, "q_evap_old"))
    fresh.close()
