"""One host thread per plan: threads that step plans of different shapes at the
same time get the results of stepping them one after the other. The shapes
share kernels but need different amounts of shared memory, so a limit set for
one thread's launch must not fail another's."""
import threading

import numpy as np
import pytest

from conftest import make_context

pytestmark = pytest.mark.gpu


def _track(nx, ny, nz):
    from spectral_galerkin_heat_b200 import workloads
    from spectral_galerkin_heat_b200.laser import StraightTrack
    size = (2e-3 * nx / 64, 1e-3 * ny / 32, 0.5e-3)
    cfg, _ = workloads.straight_track(nx=nx, ny=ny, nz=nz, steps=400, size=size)
    return make_context(cfg, StraightTrack(0.3 * size[0], 0.5 * size[1], 0.5, 0.0, 180.0))


def _raster(nx, ny, nz):
    from spectral_galerkin_heat_b200 import workloads
    return make_context(*workloads.nonlinear_raster(nx, ny, nz, steps=400, tol=1e-30, cap=6))


# (contexts, steps, eager): face clusters (k_face_run, matrices kept in shared
# memory by both shapes), and the volume form launched kernel by kernel
CASES = {"face": (lambda: [_track(64, 32, 8), _track(48, 24, 8)], 400, False),
         "volume": (lambda: [_raster(64, 32, 16), _raster(40, 24, 8)], 60, True)}


@pytest.mark.parametrize("name", list(CASES))
def test_threads_with_a_plan_each(name):
    import torch
    from spectral_galerkin_heat_b200 import B200SpectralSolver
    make, steps, eager = CASES[name]
    ctxs = make()

    def solve(ctx, out, key, barrier=None):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                s = B200SpectralSolver(None, ctx)
                s.initialize()
                if barrier is not None:
                    barrier.wait(60)
                dt = ctx.num.dt
                for k in range(steps):
                    s.step(k * dt, dt, eager=True) if eager else s.step(k * dt, dt)
                out[key] = s.state.a.cpu().numpy()
                s.finalize()
        except Exception as e:  # noqa: BLE001 -- reported by the assertion below
            out[key] = e

    one, both = {}, {}
    for i, c in enumerate(ctxs):
        solve(c, one, i)
    barrier = threading.Barrier(len(ctxs))
    threads = [threading.Thread(target=solve, args=(c, both, i, barrier)) for i, c in enumerate(ctxs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(len(ctxs)):
        assert not isinstance(one[i], Exception) and not isinstance(both[i], Exception), (one[i], both[i])
        assert np.array_equal(one[i], both[i])
