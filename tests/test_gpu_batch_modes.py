"""Modes written between a slot's start and its first step are that step's initial
condition, however the writer came by the buffer: a view taken after the
start or kept from before, a raw pointer, a write reported by hand. The same
bits as a resume from those modes; and a start that nobody writes over gives the
bits of reading the volume."""
import ctypes as C

import numpy as np
import pytest

from conftest import make_context

pytestmark = pytest.mark.gpu

STEPS = 3


def _ctxs():
    from spectral_galerkin_heat_b200 import workloads
    from spectral_galerkin_heat_b200.laser import StraightTrack
    out = []
    for nx, ny, nz, cap in ((64, 32, 9, 1), (40, 25, 6, 6)):
        size = (2e-3 * nx / 64, 1e-3 * ny / 32, 0.5e-3)
        cfg, _ = workloads.straight_track(nx=nx, ny=ny, nz=nz, steps=STEPS, size=size)
        cfg["simulation"].update({"max_picard_iter": cap, "picard_omega": 0.5, "picard_tol": 1e-4})
        out.append(make_context(cfg, StraightTrack(0.4 * size[0], 0.45 * size[1], 0.8, 0.3, 180.0)))
    return out


def _raw(b, slot):
    from spectral_galerkin_heat_b200 import _lib
    ptr, nb = C.c_void_p(), C.c_uint64()
    _lib.check("buffer", _lib.lib().sgh_batch_buffer(b._h, slot, _lib.BUF["modes"], C.byref(ptr), C.byref(nb)))
    assert ptr.value == b._view(slot, "modes").data_ptr()


def _unseen(b, slot, x):
    b._view(slot, "modes").data.copy_(x)   # .data: torch counts no write


WRITES = {
    "view_after_start": lambda b, i, x, kept: b.modes(i).copy_(x),
    "view_after_start_unseen": lambda b, i, x, kept: b.modes(i).data.copy_(x),
    "kept_view": lambda b, i, x, kept: kept.copy_(x),
    "raw_pointer": lambda b, i, x, kept: (_raw(b, i), _unseen(b, i, x)),
    "reported": lambda b, i, x, kept: (kept.data.copy_(x), b.modes_written(i)),
}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("how", ["none", "raw_pointer_before_start", *WRITES])
def test_first_step_sees_the_modes_as_they_are(how, precision):
    import torch
    from spectral_galerkin_heat_b200.batch import BatchSolver
    ctxs = _ctxs()
    ref, b = BatchSolver(ctxs, precision), BatchSolver(ctxs, precision)
    for i, c in enumerate(ctxs):
        table = b.laser_table(c, 0.0, STEPS)
        b.start(i, STEPS, table=table)
        b.step(1)                       # a start that follows steps, as most do
        kept = b.modes(i)
        if how == "raw_pointer_before_start":
            _raw(b, i)
        b.start(i, STEPS, table=table)
        x = kept.clone()
        if how != "none":
            # a field above boiling: what evaporates in the first step depends on it
            x *= 11.0
            x += x[0, 0, 0] * 1e-3 * torch.randn(x.shape, dtype=x.dtype, device=x.device,
                                                 generator=torch.Generator("cuda").manual_seed(i))
        if how == "raw_pointer_before_start":
            _unseen(b, i, x)
        elif how != "none":
            WRITES[how](b, i, x, kept)
        ref.import_slot(i, {"modes": x, "q_evap_old": torch.zeros(x.shape[1:], dtype=torch.float64, device="cuda"),
                            "step": 0, "n_steps": STEPS, "precision": precision, "shape": tuple(x.shape)}, table)
        b.step(STEPS)
        ref.step(STEPS)
        assert np.array_equal(b.modes(i).cpu().numpy(), ref.modes(i).cpu().numpy())
    b.close()
    ref.close()


def test_lanes():
    import torch
    from spectral_galerkin_heat_b200.batch import BatchSolver, LaneBatch
    ctxs = _ctxs()
    lanes, ref = LaneBatch(ctxs, "mixed", lanes=2), BatchSolver(ctxs, "mixed")
    for i, c in enumerate(ctxs):
        table = ref.laser_table(c, 0.0, STEPS)
        lanes.start(i, STEPS, table=table)
        ref.start(i, STEPS, table=table)
        torch.cuda.synchronize()
        for b in (lanes, ref):
            b.modes(i).mul_(11.0)
        torch.cuda.synchronize()
    lanes.step(STEPS)
    ref.step(STEPS)
    lanes.synchronize()
    for i, c in enumerate(ctxs):
        assert np.array_equal(lanes.modes(i).cpu().numpy(), ref.modes(i).cpu().numpy())
        one = BatchSolver([c], "mixed")
        table = one.laser_table(c, 0.0, STEPS)
        one.start(0, STEPS, table=table)
        x = one.modes(0) * 11.0
        one.import_slot(0, {"modes": x, "q_evap_old": torch.zeros(x.shape[1:], dtype=torch.float64, device="cuda"),
                            "step": 0, "n_steps": STEPS, "precision": "mixed", "shape": tuple(x.shape)}, table)
        one.step(STEPS)
        assert np.array_equal(lanes.modes(i).cpu().numpy(), one.modes(0).cpu().numpy())
        one.close()
    lanes.close()
    ref.close()
