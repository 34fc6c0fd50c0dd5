"""Ghost points that the boundary closures do not read do not reach du.  At the
low end of a CLOSURE direction every face of the closure zone takes interior
points only; at the high end the WENO7 P term of the third face from the end
reads the first ghost point.  So du is the same bits whether the other ghost
points hold the zero-gradient values or NaN."""
import numpy as np
import pytest

import windstencil_b200 as ws
from windstencil_b200 import workloads as wl
from tests.test_gpu_parity import oracle_prims, to_lap
from oracle.oracle import make_grid as or_grid

pytestmark = pytest.mark.gpu
CL, PE = ws.FACE_CLOSURE, ws.FACE_PERIODIC


@pytest.mark.parametrize("precision", [ws.FP64, ws.MIXED])
@pytest.mark.parametrize("tile", [None, (16, 8, 0, 704)])
@pytest.mark.parametrize("shape", [(8, 8, 5), (40, 24, 10), (21, 67, 9)])
def test_du_ignores_closure_ghosts(oracle, cuda, shape, tile, precision):
    faces = (CL, CL, CL, CL, PE, PE)
    g = ws.Grid(*shape, faces=faces, precision=precision)
    prims = oracle_prims(oracle, or_grid(*shape, face_kind=faces), wl.sod_state(*shape, seed=71))
    out = []
    for value in (None, np.nan):
        dev = [to_lap(cuda, g, prims[i]) for i in (0, 1, 2, 3, 5)]
        if value is not None:
            for t in dev:
                t[:, :, :4] = value
                t[:, :, g.nx + 5:] = value
                t[:, :4, :] = value
                t[:, g.ny + 5:, :] = value
        du = ws.soa_tensor(g)
        ws.du_invis_jacobian3d(g, ws.interior_job(g), *dev, du, tile=tile)
        out.append(du.cpu().numpy())
    assert np.isfinite(out[0]).all()
    assert np.array_equal(*out)


@pytest.mark.parametrize("precision", [ws.FP64, ws.MIXED])
@pytest.mark.parametrize("tile", [None, (16, 8, 0, 704)])
def test_first_high_ghost_reaches_one_face(oracle, cuda, tile, precision):
    """The one ghost point that is read, three faces from the high end in x,
    reaches the two cells at that face and no other."""
    shape, faces = (19, 24, 6), (CL, CL, CL, CL, PE, PE)
    g = ws.Grid(*shape, faces=faces, precision=precision)
    prims = oracle_prims(oracle, or_grid(*shape, face_kind=faces), wl.fourier_state(*shape, seed=72))
    out = []
    for value in (None, np.nan):
        dev = [to_lap(cuda, g, prims[i]) for i in (0, 1, 2, 3, 5)]
        if value is not None:
            for t in dev:
                t[:, :, g.nx + 4] = value
        du = ws.soa_tensor(g)
        ws.du_invis_jacobian3d(g, ws.interior_job(g), *dev, du, tile=tile)
        out.append(du.cpu().numpy())
    hit = [g.nx - 4, g.nx - 3]
    assert np.isnan(out[1][..., hit]).all()
    rest = [i for i in range(g.nx) if i not in hit]
    assert np.array_equal(out[0][..., rest], out[1][..., rest])
