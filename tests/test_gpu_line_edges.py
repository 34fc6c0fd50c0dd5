"""The line passes at the edges of their work split: line counts around the
groups of 32 (FP64) and 64 (mixed) lines, march lengths around the chunks of
five points, the smallest extents, sub-jobs that start and end inside them.

FP64 against the oracle at the parity tolerance (rel. L-inf 1e-12 per field);
the mixed form within its stated budget for one RHS (rel. L2 5e-5).
"""
import numpy as np
import pytest

import windstencil_b200 as ws
from windstencil_b200 import workloads as wl
from oracle.oracle import make_grid as or_grid
from tests.conftest import rel_l2, rel_linf
from tests.test_gpu_parity import _case

pytestmark = pytest.mark.gpu

SHAPES = [(4, 4, 4), (5, 6, 9), (8, 4, 8), (9, 31, 5), (11, 8, 33), (65, 4, 16), (33, 63, 4),
          (10, 64, 11), (129, 8, 7), (16, 15, 130)]


@pytest.mark.parametrize("faces", ["periodic", "closure"])
@pytest.mark.parametrize("shape", SHAPES)
def test_rhs_and_step_at_group_and_chunk_edges(oracle, cuda, shape, faces):
    if faces == "closure" and min(shape[:2]) < 8:
        pytest.skip("a CLOSURE direction needs 8 cells")
    kinds = (ws.FACE_CLOSURE,) * 4 + (0, 0) if faces == "closure" else (0,) * 6
    f0 = wl.fourier_state(*shape, seed=31)
    og = or_grid(*shape, face_kind=kinds)
    ref = oracle.rhs_conserved(og, f0)
    dt = oracle.compute_dt(og, f0, 0.4)
    ref1 = oracle.rk3_steps(og, f0, dt, 2)
    for precision in (ws.FP64, ws.MIXED):
        s = ws.Solver(ws.Grid(*shape, faces=kinds, precision=precision))
        s.set_state(f0)
        s.rhs()
        du = s.get_rhs()
        s.step(dt, 2)
        out = s.get_state()
        assert s.status() == 0
        s.close()
        if precision == ws.FP64:
            assert rel_linf(du, ref).max() <= 1e-12
            assert rel_linf(out, ref1).max() <= 1e-12
        else:
            assert rel_l2(du, ref).max() <= 5e-5
            assert rel_l2(out, ref1).max() <= 1e-6


@pytest.mark.parametrize("box", [((4, 4, 4), (5, 5, 5)), ((6, 9, 5), (39, 10, 16)),
                                 ((9, 5, 8), (14, 38, 13)), ((37, 4, 4), (41, 69, 9))])
def test_subjobs_at_chunk_edges(oracle, cuda, box):
    shape = (40, 66, 14)
    g = ws.Grid(*shape)
    job = ws.WsJob(ws.WsDim3(*box[0]), ws.WsDim3(*box[1]))
    out, ref = _case(oracle, cuda, g, wl.fourier_state(*shape, seed=32), job=job)
    whole = np.abs(oracle.rhs_conserved(or_grid(*shape), wl.fourier_state(*shape, seed=32)))
    scale = whole.reshape(5, -1).max(axis=1)          # the field's own size: a job may be one cell
    err = np.abs(out - ref).reshape(5, -1).max(axis=1)
    assert (err <= 1e-12 * scale).all()
