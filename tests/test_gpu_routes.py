"""Which form a single-instance plan takes, on both sides of the rules that
choose it, and that either form gives the oracle's steps to 1e-10 (the bound of
every FP64 form). Faces: one cluster, or one pass per axis where the cluster's
few SMs would take longer."""
import ctypes as C

import pytest

from conftest import make_context, rel_l2

pytestmark = pytest.mark.gpu


def _counts(s):
    from spectral_galerkin_heat_b200 import _lib
    a, b, c = C.c_int32(), C.c_int32(), C.c_int32()
    _lib.check("launch_counts", _lib.lib().sgh_plan_launch_counts(s._plan, C.byref(a), C.byref(b), C.byref(c)))
    return a.value, b.value, c.value


def _against_oracle(ctx, steps=2, **kw):
    from oracle.sgh_oracle import OracleSolver
    from spectral_galerkin_heat_b200 import B200SpectralSolver
    o = OracleSolver(ctx)
    o.initialize()
    s = B200SpectralSolver(None, ctx, **kw)
    s.initialize()
    dt = ctx.num.dt
    for k in range(steps):
        _, mo = o.step(k * dt, dt)
        _, m = s.step(k * dt, dt)
        assert m["n_evap_iter"] == mo["n_evap_iter"]
    counts, err = _counts(s), rel_l2(s.state.a.cpu().numpy(), o.a)
    s.finalize()
    return counts, err


@pytest.mark.parametrize("nx,ny,cap,cluster", [
    (64, 32, 1, True), (512, 64, 1, False), (512, 64, 6, True), (256, 256, 1, False), (256, 256, 6, True),
    (160, 256, 1, True), (256, 160, 1, False), (16, 400, 1, False), (16, 400, 6, False), (16, 256, 6, True), (288, 144, 6, False), (300, 200, 1, False), (1000, 16, 6, False)])
def test_face_form(nx, ny, cap, cluster):
    from spectral_galerkin_heat_b200 import workloads
    from spectral_galerkin_heat_b200.laser import StraightTrack
    size = (nx * 3e-5, ny * 3e-5, 2e-4)
    cfg, _ = workloads.straight_track(nx=nx, ny=ny, nz=4, steps=3, size=size)
    if cap > 1:
        cfg["simulation"].update({"max_picard_iter": cap, "picard_omega": 0.1, "picard_tol": 1e-4})
    ctx = make_context(cfg, StraightTrack(0.4 * size[0], 0.45 * size[1], 0.8, 0.3, 120.0))
    counts, err = _against_oracle(ctx)
    assert (counts[1] == 0) == cluster   # a cluster iterates inside its one kernel
    assert err < 1e-10


@pytest.mark.parametrize("nx,ny,nz,precision,fused", [
    (32, 16, 8, "fp64", False), (64, 32, 8, "fp64", False), (48, 24, 16, "fp64", True), (31, 33, 17, "fp64", True),
    (67, 41, 9, "fp64", True), (100, 17, 33, "fp64", True), (17, 100, 33, "fp64", True), (23, 25, 31, "fp64", False),
    (320, 160, 8, "fp64", False), (288, 144, 8, "fp64", False), (32, 16, 8, "mixed", True), (320, 160, 8, "mixed", True)])
@pytest.mark.parametrize("latent_only", [False, True])
def test_volume_form(nx, ny, nz, precision, fused, latent_only):
    """Fused slab and column kernels: five launches an iteration (two with latent
    heat alone) against one pass per axis (14, or 8); mixed plans against
    the oracle at the 1e-5 bound of their FP32 modes."""
    from spectral_galerkin_heat_b200 import workloads
    cfg, path = workloads.nonlinear_raster(nx, ny, nz, steps=3, tol=1e-30, cap=8)
    if latent_only:
        cfg["material"].update({"k": 25.0, "Cp": 625.0})
    counts, err = _against_oracle(make_context(cfg, path), precision=precision)
    assert (counts[1] == (2 if latent_only else 5)) == fused, counts
    assert err < (1e-10 if precision == "fp64" else 1e-5)


def test_tuner_times_only_what_differs():
    """A loop without axis passes has no threshold to tune, a cluster's no kernel."""
    from spectral_galerkin_heat_b200 import workloads
    from spectral_galerkin_heat_b200.autotune import tune
    track = make_context(*workloads.straight_track(steps=8))
    r = tune(track, candidates=(1, 132), steps=3, warmup=1)
    assert list(r["candidates"]) == ["1|0"] and r["axis_cuda_cores"] == 0
    raster = make_context(*workloads.nonlinear_raster(64, 32, 16, steps=8, cap=5))
    r = tune(raster, candidates=(1, 132), steps=3, warmup=1)
    assert sorted(r["candidates"]) == ["132|1", "1|0", "1|1"]
