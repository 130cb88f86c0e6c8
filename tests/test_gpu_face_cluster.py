"""The face-space step in one thread-block cluster (folded FP64 contractions):
sizes at the edges of its tiles (8-vector and 16-mode tiles, 8-slice steps,
odd lengths with a middle sample) and of its cluster sizes, against the FP64
oracle. FP64 to 1e-10 (the bound of every FP64 form), mixed batches to 1e-4
(the bound of the mixed form)."""
import numpy as np
import pytest

from conftest import make_context, rel_l2

pytestmark = pytest.mark.gpu

# (nx, ny): shortest axes, one below / at / above a tile, odd lengths, the
# shares of 1, 4, 8 and 16 CTAs with ragged last shares, faces with more
# columns than rows and the reverse
FACES = [(2, 2), (3, 5), (7, 8), (9, 16), (16, 15), (17, 33), (31, 32), (33, 31), (64, 17), (20, 100),
         (127, 65), (200, 81), (257, 120), (120, 257)]


def _ctx(nx, ny, nz, steps, cap):
    from spectral_galerkin_heat_b200 import workloads
    from spectral_galerkin_heat_b200.laser import StraightTrack
    size = (2e-3 * nx / 64, 1e-3 * ny / 32, 0.5e-3)
    cfg, _ = workloads.straight_track(nx=nx, ny=ny, nz=nz, steps=steps, size=size)
    if cap > 1:
        cfg["simulation"].update({"max_picard_iter": cap, "picard_omega": 0.1, "picard_tol": 1e-4})
    return make_context(cfg, StraightTrack(0.4 * size[0], 0.45 * size[1], 0.8, 0.3, 180.0))


@pytest.mark.parametrize("nx,ny", FACES)
def test_cluster_faces_vs_oracle(nx, ny):
    from oracle.sgh_oracle import OracleSolver
    from spectral_galerkin_heat_b200 import B200SpectralSolver
    from spectral_galerkin_heat_b200.batch import BatchSolver
    steps = 3
    ctx = _ctx(nx, ny, 5, steps, cap=12)
    o = OracleSolver(ctx)
    o.initialize()
    dt = ctx.num.dt
    mo = [o.step(k * dt, dt)[1] for k in range(steps)]
    s = B200SpectralSolver(None, ctx)
    s.initialize()
    ms = s.run(0.0, steps)
    assert [m["n_evap_iter"] for m in ms] == [m["n_evap_iter"] for m in mo]
    assert rel_l2(s.state.a.cpu().numpy(), o.a) < 1e-10
    assert rel_l2(s.surface_temperature().cpu().numpy(), o.surface_temperature()) < 1e-10
    np.testing.assert_allclose([m["P_laser"] for m in ms], [m["P_laser"] for m in mo], rtol=1e-10)
    np.testing.assert_allclose([m["T_surface_max"] for m in ms], [m["T_surface_max"] for m in mo], rtol=1e-10)
    for precision, tol in (("fp64", 1e-10), ("mixed", 1e-4)):
        b = BatchSolver([ctx, ctx], precision)
        b.start(1, steps)
        b.step(steps)
        assert b.tensor_core_error() == 0
        assert rel_l2(b.modes(1).double().cpu().numpy(), o.a) < tol
        assert [m["n_evap_iter"] for m in b.metrics(1)] == [m["n_evap_iter"] for m in mo]
        if precision == "fp64":  # a slot and a plan do the same arithmetic
            assert np.array_equal(b.modes(1).cpu().numpy(), s.state.a.cpu().numpy())
        b.close()
    s.finalize()


def test_steps_one_by_one_equal_a_run_and_wide_slots_share_a_batch():
    """A run on the device and single calls give the same bits; in one mixed
    batch, Picard slots on clusters and one-pass slots on the tensor-core
    kernels each equal themselves alone."""
    from spectral_galerkin_heat_b200 import B200SpectralSolver
    from spectral_galerkin_heat_b200.batch import BatchSolver
    steps = 4
    ctx = _ctx(70, 40, 9, steps, cap=1)
    modes = []
    for run in (True, False):
        s = B200SpectralSolver(None, ctx)
        s.initialize()
        if run:
            s.run(0.0, steps)
        else:
            for k in range(steps):
                s.step(k * ctx.num.dt, ctx.num.dt)
        modes.append(s.state.a.cpu().numpy())
        s.finalize()
    assert np.array_equal(modes[0], modes[1])
    ctxs = [ctx, _ctx(48, 24, 9, steps, cap=10), _ctx(136, 72, 9, steps, cap=10), _ctx(32, 24, 8, steps, cap=1)]
    mix = BatchSolver(ctxs, "mixed")
    for i in range(len(ctxs)):
        mix.start(i, steps)
    mix.step(steps)
    assert mix.tensor_core_error() == 0
    for i, c in enumerate(ctxs):
        alone = BatchSolver([c], "mixed")
        alone.start(0, steps)
        alone.step(steps)
        assert np.array_equal(alone.modes(0).cpu().numpy(), mix.modes(i).cpu().numpy())
        alone.close()
    mix.close()


@pytest.mark.parametrize("count,precision", [(30, "fp64"), (600, "fp64"), (600, "mixed"), (2000, "mixed")])
def test_crowded_batches(count, precision):
    """Face shares of a lightly and a heavily loaded batch: a slot among many
    (shares of up to 4096 elements; above 10 waves the tensor-core kernels from 2048 on)
    against the same slot alone. FP64 and mixed clusters to the bit; the
    tensor-core kernels to 2e-4, the bound of the mixed form on each side."""
    from spectral_galerkin_heat_b200.batch import BatchSolver
    steps = 2
    shapes = [(64, 33), (47, 32), (100, 60)]
    ctxs = [_ctx(nx, ny, 5, steps, cap=8) for nx, ny in shapes]
    waves = count / 3 * sum(x * y for x, y in shapes) / (148 * 2048)
    b = BatchSolver([ctxs[i % 3] for i in range(count)], precision)
    for i in range(count):
        b.start(i, steps)
    b.step(steps)
    for i in (0, count // 2 // 3 * 3 + 1, count - 1 - count % 3):
        one = BatchSolver([ctxs[i % 3]], precision)
        one.start(0, steps)
        one.step(steps)
        x, y = b.modes(i).cpu().numpy(), one.modes(0).cpu().numpy()
        if precision == "mixed" and waves > 10 and i % 3 != 1:
            assert rel_l2(x, y) < 2e-4
        else:
            assert np.array_equal(x, y)
        one.close()
    b.close()
