"""The fused grid-mode volume form (slab and column kernels on folded FP64
contractions) at sizes where it can go wrong: shortest axes, one below / at /
above the 8- and 16-wide tiles, odd lengths, ragged shares of a cluster, columns
that end inside a CTA. Against the FP64 oracle to 1e-10 (the bound of every FP64
form), and the mixed plan to 1e-4."""
import numpy as np
import pytest

from conftest import make_context, rel_l2

pytestmark = pytest.mark.gpu

SHAPES = [(2, 3, 2), (7, 5, 9), (16, 8, 16), (17, 33, 15), (40, 21, 33), (65, 31, 8), (130, 66, 5), (24, 12, 70)]


def _contexts(nx, ny, nz):
    """The T-dependent raster, and constant properties with latent heat only."""
    from spectral_galerkin_heat_b200 import workloads
    size = (nx * 15e-6, ny * 15e-6, nz * 15e-6)
    cfg, path = workloads.nonlinear_raster(nx=nx, ny=ny, nz=nz, steps=2, size=size, line_length=0.4 * size[0],
                                           hatch=0.1 * size[1], n_lines=2, tol=1e-6, cap=25)
    yield make_context(cfg, path)
    cfg, path = workloads.straight_track(nx=nx, ny=ny, nz=nz, steps=2, size=size, x0=0.4 * size[0], dt=2e-6)
    cfg["material"].update({"L_f": 2.7e5, "h_conv_bottom": 2000.0})
    cfg["simulation"].update({"max_picard_iter": 12, "picard_omega": 0.1, "picard_tol": 1e-9})
    yield make_context(cfg, path)


@pytest.mark.parametrize("nx,ny,nz", SHAPES)
def test_fused_volume_step_vs_oracle(nx, ny, nz):
    from oracle.sgh_oracle import OracleSolver
    from spectral_galerkin_heat_b200 import B200SpectralSolver
    for ctx in _contexts(nx, ny, nz):
        o = OracleSolver(ctx)
        o.initialize()
        s = B200SpectralSolver(None, ctx)
        s.initialize()
        dt = ctx.num.dt
        for k in range(2):
            mo = o.step(k * dt, dt)[1]
            m = s.step(k * dt, dt, eager=(k == 1))[1]
            assert m["n_evap_iter"] == mo["n_evap_iter"]
            assert rel_l2(s.state.a.cpu().numpy(), o.a) < 1e-10
            assert abs(m["T_surface_max"] - mo["T_surface_max"]) < 1e-10 * abs(mo["T_surface_max"])
        assert rel_l2(s.state.T_prev.cpu().numpy(), o.T_prev_full) < 1e-10
        if o.Q_modes_prev is not None and np.abs(o.Q_modes_prev).max() > 0:
            assert rel_l2(s.state.buffer("Q_modes").cpu().numpy(), o.Q_modes_prev) < 1e-8
        s.finalize()
    mixed = B200SpectralSolver(None, ctx, precision="mixed")
    mixed.initialize()
    for k in range(2):
        mixed.step(k * dt, dt)
    assert rel_l2(mixed.state.a.cpu().numpy(), o.a) < 1e-4
    mixed.finalize()
