"""A forcing rate that no cell takes adds nothing to the budgets.

The reference's series formula (cu:547-554, cu:589-601) divides by the time
since the last record, so at a record's own time the rate is infinite: the
cells that take it say so, but a grid without any -- a dry one under
evaporation, one whose cells are all NODATA under rain -- keeps its budgets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision, how", [(0, {}), (1, {}), (1, {"steps_per_launch": 1}), (1, {"kernel": 1}),
                                            (1, {"variant": 6, "steps_per_launch": 1})])
def test_evaporation_over_dry_ground(sw2d_mod, oracle_mod, precision, how):
    rows, cols, dt, ev, ev_dt = 40, 70, 0.5, np.array([0.3, 0.5, 0.4, 0.2, 0.6]), 2.5
    z = np.zeros((rows, cols))
    o = oracle_mod.Oracle(rows, cols, 5.0, 5.0, z, dt_mode=0, dt=dt, EV_WL_min=0.01)
    o.set_forcing(oracle_mod.OracleForcing(ev=ev, ev_dt=ev_dt))
    o.set_state(z)
    with sw2d_mod.Solver(rows=rows, cols=cols, dx=5.0, dy=5.0, precision=precision, dt_mode=sw2d_mod.DT_FIXED, dt=dt,
                         EV_WL_min=0.01, **how) as g:
        g.set_static(z)
        g.set_evaporation(ev, ev_dt)
        g.set_state(z)
        assert g.advance(12) == o.advance(12) == 12  # rates at t = 0.5, 1.5, 2.5, ...
        b = g.budget()
        assert b["evap_out"] == o.budget()["evap_out"] == 0.0
        assert b["rain_in"] == b["clamp_gain"] == 0.0 and b["nonfinite"] == 0


@pytest.mark.parametrize("precision", [0, 1])
def test_rain_over_no_cell(sw2d_mod, precision):
    z = np.full((30, 40), -9999.0)
    with sw2d_mod.Solver(rows=30, cols=40, dx=5.0, dy=5.0, precision=precision, dt_mode=sw2d_mod.DT_FIXED,
                         dt=0.5) as g:
        g.set_static(z)
        g.set_rain(sw2d_mod.RAIN_COMPAT, [1.0, 4.0, 2.0], 1.5)
        g.set_state(0.0 * z)
        assert g.advance(9) == 9
        assert g.budget()["rain_in"] == 0.0


def test_rain_over_no_cell_of_a_batch(sw2d_mod):
    z = np.full((30, 40), -9999.0)
    with sw2d_mod.Batch(max_scenarios=2) as b:
        cfg = sw2d_mod.default_config(rows=30, cols=40, dx=5.0, dy=5.0, precision=sw2d_mod.PREC_F32,
                                      dt_mode=sw2d_mod.DT_CFL, dt=2.0, cfl=0.5)  # still: rates at t = 2, 6, 10, ...
        sid = b.add(cfg, z, 0.0 * z, rain_kind=sw2d_mod.RAIN_COMPAT, rain=np.array([1.0, 4.0, 2.0]), rain_dt=2.0)
        b.advance(6)
        bud = b.budget(sid)
        assert bud["t"] == 24.0 and bud["rain_in"] == 0.0
