"""A step whose line passes take their ghost values from the interior against
the same step by stages, each of which fills the ghost layers first: the same
arithmetic on the same values, so the results are the same bits."""
import numpy as np
import pytest

import windstencil_b200 as ws
from windstencil_b200 import workloads as wl

pytestmark = pytest.mark.gpu

P, E, C = ws.FACE_PERIODIC, ws.FACE_EXTRAP, ws.FACE_CLOSURE
FACES = [(P,) * 6, (E,) * 6, (C,) * 4 + (E, E), (E, P, P, E, P, E), (C, E, E, C, P, P)]


@pytest.mark.parametrize("precision", [ws.FP64, ws.MIXED])
@pytest.mark.parametrize("faces", FACES)
@pytest.mark.parametrize("shape", [(8, 8, 8), (37, 11, 9), (13, 66, 34)])
@pytest.mark.parametrize("viscous", [False, True])
def test_step_is_its_stages(cuda, precision, faces, shape, viscous):
    if viscous and C in faces:
        pytest.skip("the viscous terms take no CLOSURE faces")
    g = ws.Grid(*shape, faces=faces, precision=precision)
    f0 = wl.fourier_state(*shape, seed=41)
    outs = []
    for by_stage in (False, True):
        s = ws.Solver(g)
        s.set_state(f0)
        if viscous:
            s.set_viscous(dict(re=1e3, pr=0.72, ref_t=288.15, scheme=6))
        dt = s.compute_dt(0.3)
        for _ in range(2):
            if by_stage:
                for krk in (1, 2, 3):
                    s.stage(krk, dt)
            else:
                s.step(dt)
        outs.append(s.get_state())
        assert s.status() == 0
        s.close()
    assert np.array_equal(*outs)
