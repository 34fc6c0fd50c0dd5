"""Large but finite fluxes: the reconstruction's products of indicators stay in
range.  Density and pressure are scaled, which scales every flux; the WENO weights
of such a flow do not depend on its scale (eps is far below the indicators), so
du / scale is that of the unscaled equations."""
import numpy as np
import pytest

import windstencil_b200 as ws
from windstencil_b200 import workloads as wl
from tests.conftest import rel_l2, rel_linf

pytestmark = pytest.mark.gpu
SHAPE = (40, 24, 12)


def _rhs(scale, precision):
    rng = np.random.default_rng(91)
    n = SHAPE[::-1]
    d, p = 1.0 + 0.6 * rng.random(n), 1.0 + 0.6 * rng.random(n)
    u, v, w = (0.4 * rng.random(n) - 0.2 for _ in range(3))
    s = ws.Solver(ws.Grid(*SHAPE, precision=precision))
    s.set_state(wl.prim_to_cons(d * scale, u, v, w, 1.4 * p / d))
    s.rhs()
    out = s.get_rhs()
    s.close()
    return out / scale


def test_mixed_flux_range(cuda):
    """Within the mixed form's budget for one RHS.  The energy's split flux is the
    largest, 1.25 rho c^3 to 4 rho c^3 from cell to cell here, so its differences
    are up to 3 scales: 3e9 of the 5e9 that the FP32 products take."""
    ref = _rhs(1e6, ws.FP64)
    for scale in (1e6, 3e8, 1e9):
        out = _rhs(scale, ws.MIXED)
        assert np.isfinite(out).all()
        assert rel_l2(out, ref).max() <= 5e-5, scale


def test_fp64_flux_range(cuda):
    """Up to flux differences of 1e32.  Scaling by a power of two changes no
    rounding but eps' share of the indicators, below 1e-10 / 1e12 of them."""
    ref = _rhs(2.0 ** 20, ws.FP64)
    for scale in (2.0 ** 60, 2.0 ** 100, 2.0 ** 106):
        out = _rhs(scale, ws.FP64)
        assert np.isfinite(out).all()
        assert rel_linf(out, ref).max() <= 1e-12, scale
