"""The line passes at the edges of their groups, chunks and zones, for general
metrics (with and without CLOSURE walls) and for batches whose grids have walls.

FP64 against the oracle at the parity tolerance (rel. L-inf 1e-12 per field); the
mixed form within its budget for one RHS (rel. L2 5e-5) and, against the one-grid
solver, 1e-6 for steps."""
import numpy as np
import pytest

import windstencil_b200 as ws
from windstencil_b200 import workloads as wl
from tests.conftest import rel_l2, rel_linf
from tests.test_gpu_parity import _case

pytestmark = pytest.mark.gpu
C, P = ws.FACE_CLOSURE, ws.FACE_PERIODIC
SHAPES = [(8, 8, 4), (9, 31, 5), (11, 8, 33), (65, 9, 16), (33, 63, 4), (10, 64, 11)]


@pytest.mark.parametrize("faces", [(P,) * 6, (C,) * 4 + (P, P)])
@pytest.mark.parametrize("precision", [ws.FP64, ws.MIXED])
@pytest.mark.parametrize("shape", SHAPES)
def test_general_metrics_at_edges(oracle, cuda, shape, precision, faces):
    g = ws.Grid(*shape, metrics_uniform=False, faces=faces, precision=precision)
    rng = np.random.default_rng(95)
    shp = (shape[2] + 8, shape[1] + 8, shape[0] + 8)
    metrics = [rng.uniform(0.6, 1.4, shp) if i % 4 == 0 else rng.uniform(-0.3, 0.3, shp)
               for i in range(9)]
    out, ref = _case(oracle, cuda, g, wl.fourier_state(*shape, seed=96), metrics,
                     rng.uniform(0.5, 1.5, shp))
    if precision == ws.FP64:
        assert rel_linf(out, ref).max() <= 1e-12
    else:
        assert rel_l2(out, ref).max() <= 5e-5


@pytest.mark.parametrize("precision", [ws.FP64, ws.MIXED])
def test_batch_with_walls_is_its_grids(cuda, precision):
    kinds = [(C,) * 4 + (P, P), (P,) * 6, (P, P, C, C, P, P)]
    grids = [ws.Grid(*s, faces=kinds[i % 3], precision=precision)
             for i, s in enumerate(SHAPES * 2)]
    states = [wl.sod_state(*s, seed=97 + i) for i, s in enumerate(SHAPES * 2)]
    b = ws.Batch(grids)
    for i, f in enumerate(states):
        b.set_state(i, f)
    b.rhs()
    dus = [b.get_rhs(i) for i in range(len(grids))]
    dts = b.compute_dt(0.3)
    b.set_dt(dts)
    b.step(3)
    assert b.status() == [0] * len(grids)
    for i, (g, f) in enumerate(zip(grids, states)):
        s = ws.Solver(g)
        s.set_state(f)
        s.rhs()
        tol = 1e-13 if precision == ws.FP64 else 1e-6      # as the other batch tests
        assert rel_linf(s.get_rhs(), dus[i]).max() <= tol, i
        s.step(dts[i], 3)
        assert rel_linf(b.get_state(i), s.get_state()).max() <= tol, i
        s.close()
    b.close()
