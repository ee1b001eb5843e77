"""A series whose record number at the current time is beyond a 32-bit integer
(a short interval, a late start) stays at its last record."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
def test_short_intervals_and_a_late_start(sw2d_mod, precision):
    rows, cols, dt, dx = 12, 40, 0.05, 2.0
    z = np.zeros((rows, cols))
    with sw2d_mod.Solver(rows=rows, cols=cols, dx=dx, dy=dx, precision=precision, dt_mode=sw2d_mod.DT_FIXED, dt=dt,
                         EV_WL_min=0.01) as g:
        g.set_static(z)
        g.set_rain(sw2d_mod.RAIN_COMPAT, [1.0, 2.0, 3e-9], 1e-8)
        g.set_evaporation([5.0, 2.0, 1e-9], 1e-8)
        g.set_point_sources(np.array([17, 300], dtype=np.int32), np.array([[9.0, 9.0], [8.0, 8.0], [0.5, 0.25]]), 1e-8)
        g.set_state(z + 1.0, t0=1000.0)
        assert g.advance(20) == 20
        b, t = g.budget(), 20 * 2 * dt
        rel = 1e-12 if precision == 0 else 1e-5
        assert b["source_in"] == pytest.approx(0.75 * t, rel=rel)
        assert b["rain_in"] == pytest.approx(3e-9 / 1e-5 * t * rows * cols * dx * dx, rel=rel)
        assert b["evap_out"] == pytest.approx(1e-9 / 1e-5 * t * rows * cols * dx * dx, rel=rel)
        assert np.all(np.isfinite(g.depth()))
