"""The FP64 kernel at the ends of what sw2d_create takes: no wet/dry threshold
(th = 0) or a tiny one, a negative EV_WL_min, depths that are negative or
beyond single precision.  The state, the time steps and what is refused are the
oracle's."""
import numpy as np
import pytest

from helpers import same

pytestmark = pytest.mark.gpu


def _pair(O, sw2d, z, h, um=None, vn=None, **kw):
    rows, cols = z.shape
    o = O.Oracle(rows, cols, 5.0, 4.0, z, **kw)
    o.set_state(h, um, vn)
    g = sw2d.Solver(rows=rows, cols=cols, dx=5.0, dy=4.0, precision=sw2d.PREC_F64, **kw)
    g.set_static(z)
    g.set_state(h, um, vn)
    return o, g


def _rain_and_evaporation(O, sw2d, o, g):
    o.set_forcing(O.OracleForcing(rain_kind=O.RAIN_STEP, rain=[60.0], rain_dt=1e6, ev=[0.4, 0.5], ev_dt=3600.0))
    g.set_rain(sw2d.RAIN_STEP, [60.0], 1e6)
    g.set_evaporation([0.4, 0.5], 3600.0)


def _equal(o, g):
    a, b = o.state(), g.state()
    for k in ("h", "um", "vn"):
        assert same(a[k], b[k]), (k, np.max(np.abs(a[k] - b[k])))
    assert g.budget()["t"] == a["t"] and g.budget()["cmax"] == o.budget()["cmax"]


@pytest.mark.parametrize("shape", [(3, 5), (40, 33), (300, 280)])
@pytest.mark.parametrize("th", [0.0, -0.0, 1e-80, 1e-20])
def test_small_thresholds_on_wet_ground(oracle_mod, sw2d_mod, shape, th):
    rng = np.random.default_rng(shape[0])
    z = rng.uniform(0.0, 0.3, shape)
    h = 10.0 ** rng.uniform(-30.0, 0.0, shape) if th else rng.uniform(0.6, 1.0, shape)
    o, g = _pair(oracle_mod, sw2d_mod, z, h, th=th, dt_mode=1, dt=0.5, cfl=0.5, manning=0.04, south_open=1)
    _rain_and_evaporation(oracle_mod, sw2d_mod, o, g)
    for _ in range(3):
        assert o.advance(5) == g.advance(5) == 5
        _equal(o, g)
    g.close()


def test_no_threshold_on_dry_ground_is_refused_as_before(oracle_mod, sw2d_mod):
    """0 / 0 at a dry face beside a wet one: not a number in the oracle, reported here."""
    rng = np.random.default_rng(3)
    z = rng.uniform(0.0, 0.3, (30, 40))
    h = np.where(rng.random(z.shape) < 0.5, 0.0, 1.0)
    o, g = _pair(oracle_mod, sw2d_mod, z, h, th=0.0, dt_mode=0, dt=0.01)
    o.advance(10)
    assert not np.all(np.isfinite(o.state()["um"]))
    with pytest.raises(sw2d_mod.SW2DError) as e:
        g.advance(10)
    assert e.value.status == sw2d_mod.native.ERR_NONFINITE
    g.close()


@pytest.mark.parametrize("evmin", [-1.0, -1e-3, -5e-324, -0.0, 0.0])
def test_negative_depths_and_evaporation_level(oracle_mod, sw2d_mod, evmin):
    rng = np.random.default_rng(11)
    z = rng.uniform(0.0, 0.1, (40, 50))
    h = rng.choice([-0.0, 0.0, -1e-3, -0.5, 0.05, 0.3], z.shape)
    o, g = _pair(oracle_mod, sw2d_mod, z, h, EV_WL_min=evmin, INT=0.1, INF=0.3, LWL=0.05, dt_mode=0, dt=0.05)
    _rain_and_evaporation(oracle_mod, sw2d_mod, o, g)
    for n in (1, 9):
        assert o.advance(n) == g.advance(n) == n
        _equal(o, g)
    bo, bg = o.budget(), g.budget()
    for k in ("rain_in", "evap_out"):
        assert bg[k] == pytest.approx(bo[k], rel=1e-12, abs=1e-14), k
    g.close()


@pytest.mark.parametrize("top", [1e30, 1e37, 1e38, 1e40, 1e80])
def test_wave_speed_beyond_single_precision(oracle_mod, sw2d_mod, top):
    """Deep and fast faces on which FP32 overflows beside ones on which it does
    not: the CFL bound is the FP64 maximum."""
    rng = np.random.default_rng(5)
    shape = (20, 37)
    for um_scale in (0.0, 1.0, 1e8, 1e30):
        z = np.zeros(shape)
        h = 10.0 ** rng.uniform(np.log10(top) - 3.0, np.log10(top), shape)
        h[rng.random(shape) < 0.5] = 1.0
        um = um_scale * rng.uniform(-1.0, 1.0, (shape[0] + 1, shape[1]))
        o, g = _pair(oracle_mod, sw2d_mod, z, h, um=um, dt_mode=1, dt=1e-30, cfl=0.5)
        assert o.advance(2) == g.advance(2) == 2
        _equal(o, g)
        g.close()
