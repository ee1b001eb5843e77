"""The batch cuts its resident scenarios' strips anew with every admission and
retirement: a scenario's state and budgets do not depend on it, a caller's
strip height stays, and the unit table's limit refuses what it refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (17, 30), (64, 64), (130, 95), (300, 210)]


def _scenario(rows, cols):
    rng = np.random.default_rng(rows * 1000 + cols)
    z = 0.05 * np.arange(rows)[::-1, None] + rng.uniform(0.0, 0.3, (rows, cols))
    z[rng.random(z.shape) < 0.03] = -9999.0
    return z, rng.choice([0.03, 0.08], z.shape), np.where(rng.random(z.shape) < 0.3, 0.0, rng.uniform(0, 0.2, z.shape))


def _cfg(sw2d, rows, cols, **kw):
    return sw2d.default_config(rows=rows, cols=cols, dx=5.0, dy=5.0, precision=sw2d.PREC_F32, dt_mode=sw2d.DT_CFL,
                               dt=2.0, cfl=0.5, south_open=1, EV_WL_min=0.02, INT=0.1, **kw)


def _add(sw2d, b, rows, cols, **kw):
    z, n, h = _scenario(rows, cols)
    return b.add(_cfg(sw2d, rows, cols, **kw), z, h, manning=n, rain_kind=sw2d.RAIN_STEP, rain=[90.0], rain_dt=3600.0)


def _read(b, sid):
    return [b.field(sid, f) for f in (0, 1, 2)], b.budget(sid)


@pytest.mark.parametrize("own", [0, 5])
def test_results_do_not_depend_on_the_strips(sw2d_mod, own):
    """Alone, in company that comes and goes, and in strips of the caller's."""
    alone = {}
    for rows, cols in SHAPES:
        with sw2d_mod.Batch(device=0, max_scenarios=2) as b:
            sid = _add(sw2d_mod, b, rows, cols)
            b.advance(60)
            alone[rows, cols] = _read(b, sid)
    with sw2d_mod.Batch(device=0, max_scenarios=16, strip_h=own) as b:
        first = [_add(sw2d_mod, b, *s) for s in SHAPES]
        b.advance(20)
        late = _add(sw2d_mod, b, 512, 480)
        b.advance(20)
        b.remove(late)
        b.advance(20)
        for s, sid in zip(SHAPES, first):
            (f, bud), (f0, bud0) = _read(b, sid), alone[s]
            for x, y in zip(f, f0):
                assert np.array_equal(x, y), s
            assert bud["t"] == bud0["t"] and bud["steps"] == bud0["steps"] == 60
            # exact counts and one FP32 value a column, summed in FP64 in another order
            for k in ("rain_in", "evap_out", "outflow"):
                assert bud[k] == pytest.approx(bud0[k], rel=1e-6 if k == "outflow" else 1e-12, abs=1e-12), k


def test_unit_table_limit_is_the_size_rules(sw2d_mod):
    """64 x 64 cells count 3 tiles x 4 strips of 16 rows, whatever is cut."""
    with sw2d_mod.Batch(device=0, max_scenarios=8, max_units=12) as b:
        sid = _add(sw2d_mod, b, 64, 64)
        with pytest.raises(sw2d_mod.SW2DError):
            _add(sw2d_mod, b, 64, 64)
        b.advance(30)
        got = _read(b, sid)
    with sw2d_mod.Batch(device=0, max_scenarios=8) as b:
        sid = _add(sw2d_mod, b, 64, 64)
        b.advance(30)
        want = _read(b, sid)
    for x, y in zip(got[0], want[0]):
        assert np.array_equal(x, y)
