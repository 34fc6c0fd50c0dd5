"""Closure zones of the line passes: the closures' values stay FP64 up to the
face difference in the mixed form too, and a cell's du does not depend on the
piece of its line that it is computed in."""
import numpy as np
import pytest

import windstencil_b200 as ws
from windstencil_b200 import workloads as wl
from oracle.oracle import make_grid as or_grid
from tests.test_gpu_parity import oracle_prims, to_lap

pytestmark = pytest.mark.gpu
CL, PE = ws.FACE_CLOSURE, ws.FACE_PERIODIC


def _du(cuda, g, dev, job):
    n = [getattr(job.end, c) - getattr(job.start, c) for c in "xyz"]
    du = cuda.full((5, n[2], n[1], n[0]), np.nan, dtype=cuda.float64, device="cuda")
    ws.du_invis_jacobian3d(g, job, *dev, du)
    return du.cpu().numpy()


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("n", [8, 13, 21, 22, 40])
def test_mixed_closure_values_are_fp64(oracle, cuda, n, axis):
    """A flow along one axis, where the split mass fluxes of both signs lie
    between 1/8 and 1 in size: FP32 values there are multiples of 2^-27, so with
    1/h a power of two the mass du of a cell between two WENO faces is a multiple
    of 2^-27 / h, and one next to a closure value is not."""
    shape = (n, 9, 6) if axis == 0 else (9, n, 6)
    h = 2.0 ** -6
    faces = tuple(CL if i // 2 == axis else PE for i in range(6))
    g = ws.Grid(*shape, hx=h, hy=h, hz=h, faces=faces, precision=ws.MIXED)
    x = np.arange(n) / n
    line = [1 + 0.1 * np.sin(5 * x), 0.2 + 0.1 * np.cos(4 * x), 1 + 0.1 * np.cos(7 * x + 1)]
    sh = [1, 1, 1]
    sh[2 - axis] = n
    d, un, T = (np.broadcast_to(a.reshape(sh), shape[::-1]).copy() for a in line)
    z = np.zeros_like(d)
    f = wl.prim_to_cons(d, un if axis == 0 else z, un if axis == 1 else z, z, T)
    prims = oracle_prims(oracle, or_grid(*shape, h, h, h, face_kind=faces), f)
    dev = [to_lap(cuda, g, prims[i]) for i in (0, 1, 2, 3, 5)]
    du = _du(cuda, g, dev, ws.interior_job(g))[0] * h * 2.0 ** 27
    q = np.moveaxis(du, 2 - axis, 0).reshape(n, -1)
    whole = (q == np.round(q)).all(axis=1)
    assert whole[4:n - 4].all()
    # (the last cell has closures linear in two split values on both sides)
    assert not whole[:4].any() and not whole[n - 4:n - 1].any()


@pytest.mark.parametrize("precision", [ws.FP64, ws.MIXED])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("n", [8, 9, 12, 18, 21, 22, 23, 31])
def test_du_does_not_depend_on_the_piece(oracle, cuda, n, axis, precision):
    shape = (n, 9, 6) if axis == 0 else (70, n, 4)
    g = ws.Grid(*shape, faces=(CL,) * 4 + (PE,) * 2, precision=precision)
    prims = oracle_prims(oracle, or_grid(*shape, face_kind=g.faces), wl.fourier_state(*shape, seed=5))
    dev = [to_lap(cuda, g, prims[i]) for i in (0, 1, 2, 3, 5)]
    whole = _du(cuda, g, dev, ws.interior_job(g))
    for lo in range(n):
        for width in (1, 3, 6):
            hi = min(lo + width, n)
            start, end = [4, 4, 4], [shape[0] + 4, shape[1] + 4, shape[2] + 4]
            start[axis], end[axis] = lo + 4, hi + 4
            job = ws.WsJob(ws.WsDim3(*start), ws.WsDim3(*end))
            part = whole[..., lo:hi] if axis == 0 else whole[:, :, lo:hi]
            assert np.array_equal(_du(cuda, g, dev, job), part), (lo, hi)
