"""Kernel selection: tile_x < 0 names the line passes, a compiled tile shape the
tile sweep whatever scan_z is (a cap when positive).  The kernels agree to
rounding only, so the bits tell which one ran."""
import numpy as np
import pytest

import windstencil_b200 as ws
from windstencil_b200 import workloads as wl

pytestmark = pytest.mark.gpu
SHAPE = (48, 24, 20)
SWEEP, UNCAPPED, LINES = (16, 8, 0, 704), (16, 8, -1, 704), (-1, 0, 0, 0)


def _solver(tile):
    s = ws.Solver(ws.Grid(*SHAPE))
    s.set_tile(tile)
    s.set_state(wl.sod_state(*SHAPE, seed=81))
    s.rhs()
    out = s.get_rhs()
    s.close()
    return out


def _batch(tile):
    b = ws.Batch([ws.Grid(*SHAPE)] * 2)
    b.set_tile(tile)
    for i in range(2):
        b.set_state(i, wl.sod_state(*SHAPE, seed=81))
    b.rhs()
    out = b.get_rhs(1)
    b.close()
    return out


@pytest.mark.parametrize("run", [_solver, _batch])
def test_negative_scan_is_an_uncapped_sweep(cuda, run):
    assert np.array_equal(run(UNCAPPED), run(SWEEP))
    assert not np.array_equal(run(LINES), run(SWEEP))
    assert np.array_equal(run(LINES), run((0, 0, 0, 0)))


def test_autotune_names_the_line_passes(cuda):
    """A batch on which the line passes win by far reports tile_x = -1."""
    b = ws.Batch([ws.Grid(128, 64, 48)] * 4)
    for i in range(4):
        b.set_state(i, wl.sod_state(128, 64, 48, seed=82 + i))
    assert b.autotune() == LINES
    b.close()
