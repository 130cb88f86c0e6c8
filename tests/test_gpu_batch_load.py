"""A slot's result does not depend on the batch around it: mixed and FP64 Picard
slots alone, among so many that the chip is filled more than ten times over,
over two lanes, and moved from a small batch into a crowded one in the middle
of a request give the same bits."""
import numpy as np
import pytest

from conftest import make_context

pytestmark = pytest.mark.gpu

STEPS = 3
COUNT = 100   # 256 x 128 faces on 148 SMs: 10.8 waves of 2048 elements per SM


def _ctx(nx, ny):
    from spectral_galerkin_heat_b200 import workloads
    from spectral_galerkin_heat_b200.laser import StraightTrack
    size = (2e-3 * nx / 64, 1e-3 * ny / 32, 0.5e-3)
    cfg, _ = workloads.straight_track(nx=nx, ny=ny, nz=5, steps=STEPS, size=size)
    cfg["simulation"].update({"max_picard_iter": 8, "picard_omega": 0.1, "picard_tol": 1e-4})
    return make_context(cfg, StraightTrack(0.4 * size[0], 0.45 * size[1], 0.8, 0.3, 180.0))


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_slot_alone_in_a_crowd_over_lanes_and_moved(precision):
    from spectral_galerkin_heat_b200.batch import BatchSolver, LaneBatch
    ctx = _ctx(256, 128)
    alone = BatchSolver([ctx], precision)
    table = alone.laser_table(ctx, 0.0, STEPS)
    alone.start(0, STEPS, table=table)
    alone.step(1)
    state = alone.export_slot(0)
    alone.step(STEPS - 1)
    want = alone.modes(0).cpu().numpy()
    alone.close()

    crowd = BatchSolver([ctx] * COUNT, precision)
    for i in range(COUNT - 1):
        crowd.start(i, STEPS, table=table)
    crowd.step(STEPS)
    assert np.array_equal(crowd.modes(COUNT // 2).cpu().numpy(), want)
    crowd.import_slot(COUNT - 1, state, table)
    crowd.step(STEPS - 1)
    assert np.array_equal(crowd.modes(COUNT - 1).cpu().numpy(), want)
    crowd.close()

    lanes = LaneBatch([ctx] * COUNT, precision, lanes=2)
    for i in range(COUNT):
        lanes.start(i, STEPS, table=table)
    lanes.step(STEPS)
    lanes.synchronize()
    assert np.array_equal(lanes.modes(COUNT - 1).cpu().numpy(), want)
    lanes.close()


@pytest.mark.parametrize("nx,ny,cluster", [(512, 64, True), (64, 512, True), (600, 32, False), (1000, 16, False)])
def test_long_thin_faces_take_the_shorter_path(nx, ny, cluster):
    """Mixed Picard slots: a cluster iterates inside its kernel (no launches per
    iteration); thin faces of very long axes stay on the tensor-core kernels.
    Either against the FP64 oracle to 1e-4, the bound of the mixed form."""
    from conftest import rel_l2
    from oracle.sgh_oracle import OracleSolver
    from spectral_galerkin_heat_b200.batch import BatchSolver
    ctx = _ctx(nx, ny)
    o = OracleSolver(ctx)
    o.initialize()
    for k in range(STEPS):
        o.step(k * ctx.num.dt, ctx.num.dt)
    b = BatchSolver([ctx], "mixed")
    assert (b.launch_counts()[1] == 0) == cluster
    b.start(0, STEPS)
    b.step(STEPS)
    assert b.tensor_core_error() == 0
    assert rel_l2(b.modes(0).double().cpu().numpy(), o.a) < 1e-4
    b.close()


def test_tensor_faces_is_the_callers_choice():
    """Picard slots on the tensor cores by request: within 1e-4 of the oracle, the
    same bits alone and among others, and no state moves between the two kinds
    of batch (their bits differ); FP64 batches refuse the choice."""
    from conftest import rel_l2
    from oracle.sgh_oracle import OracleSolver
    from spectral_galerkin_heat_b200.batch import BatchSolver
    ctxs = [_ctx(128, 64), _ctx(64, 33), _ctx(100, 60)]
    o = OracleSolver(ctxs[0])
    o.initialize()
    for k in range(STEPS):
        o.step(k * ctxs[0].num.dt, ctxs[0].num.dt)

    def run(cs):
        b = BatchSolver(cs, "mixed", tensor_faces=True)
        for i in range(len(cs)):
            b.start(i, STEPS)
        b.step(STEPS)
        assert b.tensor_core_error() == 0 and b.launch_counts()[1] > 0
        return b

    mix, alone = run(ctxs), run(ctxs[:1])
    assert rel_l2(mix.modes(0).double().cpu().numpy(), o.a) < 1e-4
    assert np.array_equal(mix.modes(0).cpu().numpy(), alone.modes(0).cpu().numpy())
    plain = BatchSolver(ctxs[:1], "mixed")
    table = plain.laser_table(ctxs[0], 0.0, STEPS)
    with pytest.raises(ValueError, match="tensor_faces"):
        plain.import_slot(0, alone.export_slot(0), table)
    alone.import_slot(0, mix.export_slot(0), table)
    for b in (mix, alone, plain):
        b.close()
    with pytest.raises(ValueError, match="tensor_faces"):
        BatchSolver(ctxs[:1], "fp64", tensor_faces=True)
