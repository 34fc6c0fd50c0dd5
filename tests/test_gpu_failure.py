"""Failure detection on the GPU without a fault: the bounded waits of the
fused RHS (on its TMA copies) and of the line passes (on the warps of a thread
group).

When a wait gives up, the CTA (the thread group) waits for its copies still in
flight, sets status bit 2 and stops.  The tests make the waits run out without
anything being wrong: with WS_TEST_STAGE_WAIT=n they poll, n times, an mbarrier
whose phase nothing ever completes.  The tests check that the
host reads the failure (ws_device_error for the drop-in entry,
ws_solver_status -> WS_ERR_TIMEOUT for the stage kernel) and that the
context stays usable: the next launches are correct against the oracle.
"""
import ctypes as C

import numpy as np
import pytest

import windstencil_b200 as ws
from windstencil_b200 import workloads as wl
from oracle.oracle import make_grid as or_grid
from tests.conftest import rel_linf

pytestmark = pytest.mark.gpu
SHAPE = (64, 32, 16)
HOLD = "64"
FUSED = (16, 8, 0, 704)        # the fused kernel's tile shape
CL, PE = ws.FACE_CLOSURE, ws.FACE_PERIODIC


def _rhs_drop_in(s, g):
    """Ghost fill, then the drop-in entry on the solver's fields."""
    lib, gc = ws.load(), g.c()
    _, du, prims = s.fields()
    ws.check(lib.ws_ghost_fill(C.byref(gc), (ws.WsField * 6)(*prims), 6, None))
    ws.check(lib.ws_du_invis_jacobian3d_tiled(C.byref(gc), ws.interior_job(g), prims[0],
                                              prims[1], prims[2], prims[3], prims[5], None, du,
                                              ws.WsTile(*FUSED), None))


def test_drop_in_wait_timeout_reported(oracle, cuda, monkeypatch):
    g = ws.Grid(*SHAPE)
    f0 = wl.fourier_state(*SHAPE, seed=41)
    s = ws.Solver(g)
    s.set_state(f0)
    assert ws.device_error() in (0, 2)            # clear whatever an earlier test left
    monkeypatch.setenv("WS_TEST_STAGE_WAIT", HOLD)
    _rhs_drop_in(s, g)
    assert ws.device_error() == 2                 # reported, and cleared by the read
    assert ws.device_error() == 0
    monkeypatch.delenv("WS_TEST_STAGE_WAIT")
    _rhs_drop_in(s, g)                            # the context is still usable
    assert ws.device_error() == 0
    ref = oracle.rhs_conserved(or_grid(*SHAPE), f0)
    assert rel_linf(s.get_rhs(), ref).max() <= 1e-12
    s.close()


def test_stage_kernel_wait_timeout_reported(oracle, cuda, monkeypatch):
    g = ws.Grid(*SHAPE)
    f0 = wl.fourier_state(*SHAPE, seed=42)
    og = or_grid(*SHAPE)
    dt = oracle.compute_dt(og, f0, 0.5)
    s = ws.Solver(g)
    s.set_tile(FUSED)
    s.set_state(f0)
    monkeypatch.setenv("WS_TEST_STAGE_WAIT", HOLD)
    s.step(dt * 0.5, 1)                           # captured with the forced wait
    assert s.status() == 6                        # WS_ERR_TIMEOUT
    monkeypatch.delenv("WS_TEST_STAGE_WAIT")
    s.set_state(f0)                               # new state, new status word
    assert s.status() == 0
    s.step(dt, 2)                                 # new dt: recaptured without it
    assert s.status() == 0
    ref = oracle.rk3_steps(og, f0, dt, 2)
    assert rel_linf(s.get_state(), ref).max() <= 1e-12
    s.close()


def _rhs_lines(s, g):
    lib, gc = ws.load(), g.c()
    _, du, prims = s.fields()
    ws.check(lib.ws_ghost_fill(C.byref(gc), (ws.WsField * 6)(*prims), 6, None))
    ws.check(lib.ws_du_invis_jacobian3d(C.byref(gc), ws.interior_job(g), prims[0], prims[1],
                                        prims[2], prims[3], prims[5], None, du, None))


@pytest.mark.parametrize("faces", [(PE,) * 6, (CL,) * 4 + (PE,) * 2])
@pytest.mark.parametrize("precision", [ws.FP64, ws.MIXED])
def test_line_pass_wait_timeout_reported(oracle, cuda, monkeypatch, precision, faces):
    g = ws.Grid(*SHAPE, faces=faces, precision=precision)
    f0 = wl.fourier_state(*SHAPE, seed=43)
    og = or_grid(*SHAPE, face_kind=faces)
    dt = oracle.compute_dt(og, f0, 0.5)
    s = ws.Solver(g)
    s.set_state(f0)
    assert ws.device_error() in (0, 2)
    monkeypatch.setenv("WS_TEST_STAGE_WAIT", HOLD)
    _rhs_lines(s, g)
    assert ws.device_error() == 2
    s.step(dt * 0.5, 1)
    assert s.status() == 6
    monkeypatch.delenv("WS_TEST_STAGE_WAIT")
    s.set_state(f0)
    _rhs_lines(s, g)
    assert ws.device_error() == 0
    tol = 1e-12 if precision == ws.FP64 else 1e-4
    assert rel_linf(s.get_rhs(), oracle.rhs_conserved(og, f0)).max() <= tol
    s.step(dt, 2)
    assert s.status() == 0
    ref = oracle.rk3_steps(og, f0, dt, 2)
    assert rel_linf(s.get_state(), ref).max() <= (1e-12 if precision == ws.FP64 else 1e-5)
    s.close()


@pytest.mark.parametrize("precision", [ws.FP64, ws.MIXED])
def test_batch_line_pass_wait_timeout_reported_for_every_grid(cuda, monkeypatch, precision):
    """A thread group that stops reports the pieces of other grids that it
    leaves undone as well: more grids than thread groups start on."""
    shapes = [(24, 12, 8), (40, 16, 5), (9, 8, 31)] * 120
    f0 = {s: wl.fourier_state(*s, seed=44) for s in shapes[:3]}

    def batch():
        b = ws.Batch([ws.Grid(*s, precision=precision) for s in shapes])
        for i, s in enumerate(shapes):
            b.set_state(i, f0[s])
        b.set_dt(b.compute_dt(0.4))
        b.step(1)
        return b
    monkeypatch.setenv("WS_TEST_STAGE_WAIT", HOLD)
    b = batch()
    assert b.status() == [6] * len(shapes)
    b.close()
    monkeypatch.delenv("WS_TEST_STAGE_WAIT")
    b = batch()
    assert b.status() == [0] * len(shapes)
    b.close()
