"""Conservation of the mixed form on periodic grids.  A face's value is rounded
to FP32 once and both cells at the face take the same value, so du sums to
zero to FP64 rounding, as in FP64.

Bound: each pass rounds a cell's face difference, its product with 1/h and its
sum with du at most once each in 64 bits, so |sum du| <= 9 x 2^-53 of the
passes' own sums of magnitudes, which are below 10 sum |du| for these states:
1e-14 sum |du|.  A stage rounds the state at most four times: over two steps
of three stages |sum f - sum f0| <= 24 x 2^-53 sum |f| = 2.7e-15 and the
stages' dt du: 1e-14 sum |f|.
"""
import numpy as np
import pytest

import windstencil_b200 as ws
from windstencil_b200 import workloads as wl

pytestmark = pytest.mark.gpu

# lines of 4 to 130 cells, whole and broken chunks of five, groups of 64 lines
# whole and broken
SHAPES = [(40, 13, 9), (37, 66, 34), (8, 5, 4), (130, 16, 8), (64, 32, 16)]


def _total(f):
    return f.astype(np.longdouble).reshape(5, -1).sum(axis=1)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("state", [wl.fourier_state, wl.sod_state])
def test_mixed_rhs_and_steps_conserve(cuda, shape, state):
    f0 = state(*shape, seed=51)
    s = ws.Solver(ws.Grid(*shape, precision=ws.MIXED))
    s.set_state(f0)
    s.rhs()
    du = s.get_rhs()
    dt = s.compute_dt(0.3)
    s.step(dt, 2)
    out = s.get_state()
    assert s.status() == 0
    s.close()
    assert (abs(_total(du)) <= 1e-14 * _total(abs(du))).all()
    assert (abs(_total(out) - _total(f0)) <= 1e-14 * _total(abs(out))).all()


def test_mixed_batch_rhs_conserves(cuda):
    b = ws.Batch([ws.Grid(*s, precision=ws.MIXED) for s in SHAPES])
    for i, s in enumerate(SHAPES):
        b.set_state(i, wl.sod_state(*s, seed=60 + i))
    b.rhs()
    for i in range(len(SHAPES)):
        du = b.get_rhs(i)
        assert (abs(_total(du)) <= 1e-14 * _total(abs(du))).all(), SHAPES[i]
    b.close()
