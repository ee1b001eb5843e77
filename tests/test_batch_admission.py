"""Admitting and removing a scenario beside many resident ones: the strips are
chosen anew each time, in a time that does not grow with the residents, and the
heights of all of them reach the device at once."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIDE = 40


def _add(sw2d, b, side=SIDE, seed=0, **kw):
    rng = np.random.default_rng(seed)
    z = 0.05 * np.arange(side)[::-1, None] + rng.uniform(0.0, 0.3, (side, side))
    cfg = sw2d.default_config(rows=side, cols=side, dx=5.0, dy=5.0, precision=sw2d.PREC_F32, dt_mode=sw2d.DT_CFL,
                              dt=2.0, cfl=0.5, south_open=1, manning=0.05, **kw)
    return b.add(cfg, z, rng.uniform(0.0, 0.2, z.shape), rain_kind=sw2d.RAIN_STEP, rain=[60.0], rain_dt=3600.0)


def test_cost_does_not_grow_with_the_residents(sw2d_mod):
    """Some two thirds more for 900 residents than for 30 when each admission went
    over all of them 17 times."""
    best = {}
    for residents in (30, 900):
        with sw2d_mod.Batch(max_scenarios=1024) as b:
            ids = [_add(sw2d_mod, b) for _ in range(residents)]
            for _ in range(7):
                t = time.perf_counter()
                for _ in range(10):
                    b.remove(ids.pop(0))
                    ids.append(_add(sw2d_mod, b))
                best[residents] = min(best.get(residents, 1.0), time.perf_counter() - t)
    assert best[900] < 1.35 * best[30], best


def test_changed_heights_reach_all_residents_in_one_copy(sw2d_mod):
    """Two large scenarios leave and the others' height changes: 20 times as long for
    900 residents as for 20 with a copy for each."""
    best = {}
    for residents in (20, 900):
        with sw2d_mod.Batch(max_scenarios=1024) as b:
            for _ in range(residents):
                _add(sw2d_mod, b)
            for _ in range(7):
                large = [_add(sw2d_mod, b, side=700) for _ in range(2)]
                t = time.perf_counter()
                for sid in large:
                    b.remove(sid)
                best[residents] = min(best.get(residents, 1.0), time.perf_counter() - t)
    assert best[900] < 6.0 * best[20], best


def test_every_resident_takes_the_new_heights(sw2d_mod):
    """A large scenario comes and goes, and with it the height of all the others
    (one row alone, taller beside it); a caller's height stays."""
    alone = {}
    for seed in range(6):
        with sw2d_mod.Batch(max_scenarios=1) as b:
            sid = _add(sw2d_mod, b, seed=seed)
            b.advance(36)
            alone[seed] = [b.field(sid, f) for f in (0, 1, 2)]
    with sw2d_mod.Batch(max_scenarios=64) as b:
        ids = {_add(sw2d_mod, b, seed=seed, strip_h=7 if seed == 3 else 0): seed for seed in range(6)}
        b.advance(12)
        large = [_add(sw2d_mod, b, side=900, seed=9) for _ in range(8)]
        b.advance(12)
        for sid in large:
            b.remove(sid)
        b.advance(12)
        for sid, seed in ids.items():
            for f in (0, 1, 2):
                assert np.array_equal(b.field(sid, f), alone[seed][f]), (seed, f)


def test_a_refused_scenario_leaves_the_others_as_they_were(sw2d_mod):
    with sw2d_mod.Batch(max_scenarios=8, max_units=14) as b:
        sid = _add(sw2d_mod, b, seed=1)  # 2 tiles x 3 strips of 16 rows
        other = _add(sw2d_mod, b, seed=2)
        used = b.bytes_in_use()
        for _ in range(3):
            with pytest.raises(sw2d_mod.SW2DError):
                _add(sw2d_mod, b, seed=3)
            assert b.bytes_in_use() == used
            b.advance(12)
        got = b.field(sid)
        b.remove(other)
        assert _add(sw2d_mod, b, seed=3) == other  # the place is free again
    with sw2d_mod.Batch(max_scenarios=1) as b:
        sid = _add(sw2d_mod, b, seed=1)
        b.advance(36)
        assert np.array_equal(got, b.field(sid))
