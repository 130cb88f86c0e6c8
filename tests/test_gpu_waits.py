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
