"""Scenarios of a batch that have reached their end time and stay resident: the
others are cut as if they were alone, and the finished ones keep their state,
time and budgets."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("t", "dt", "cmax", "volume", "rain_in", "evap_out", "outflow", "clamp_gain", "steps")


def _add(sw2d, b, seed, t_end):
    rng = np.random.default_rng(seed)
    rows, cols = int(64 * 2 ** rng.random()), int(64 * 2 ** rng.random())
    z = 0.05 * np.arange(rows)[::-1, None] + rng.uniform(0.0, 0.3, (rows, cols))
    cfg = sw2d.default_config(rows=rows, cols=cols, dx=5.0, dy=5.0, precision=sw2d.PREC_F32, dt_mode=sw2d.DT_CFL,
                              dt=2.0, cfl=0.5, south_open=1, manning=0.05, EV_WL_min=0.02, LWL=0.1)
    return b.add(cfg, z, rng.uniform(0.0, 0.1, z.shape), rain_kind=sw2d.RAIN_STEP, rain=[50.0], rain_dt=1e6,
                 t_end=t_end)


def _read(b, sid):
    return [b.field(sid, f) for f in (0, 1, 2)], b.budget(sid)


@pytest.mark.parametrize("how", ["advance", "poll", "unseen"])
def test_results_with_scenarios_ending_on_the_way(sw2d_mod, how):
    """Their ends are seen by the advance, by a poll or by neither; another one
    comes after some have ended, and one of the ended leaves."""
    ends = [5.0, 40.0, 1e9, 12.0, 90.0, 1e9, 0.0]
    with sw2d_mod.Batch(max_scenarios=16, chunk=6) as b:
        ids = [_add(sw2d_mod, b, k, e) for k, e in enumerate(ends)]
        final = {}
        for step in range(24):
            running = b.advance(7, wait=how == "advance")
            state = b.poll() if how == "poll" else None
            if how == "advance" and step > 0:
                assert running == sum(1 for e, i in zip(ends, ids) if i in b.shapes and b.budget(i)["t"] < e - 1e-9)
            if step == 10:
                ids.append(_add(sw2d_mod, b, 7, 1e9))
                ends.append(1e9)
                b.remove(ids[3])
            if state and step != 10:  # polled before the change
                assert set(state) == set(b.shapes)
            if step in (12, 23):
                for i in (ids[0], ids[6]):
                    got = _read(b, i)
                    if i in final:
                        assert all(np.array_equal(x, y) for x, y in zip(got[0], final[i][0]))
                        assert all(got[1][k] == final[i][1][k] for k in KEYS)
                    final[i] = got
        out = {k: _read(b, i) for k, i in enumerate(ids) if k != 3}
    for k, (fields, bud) in out.items():
        with sw2d_mod.Batch(max_scenarios=1, chunk=6) as b:
            sid = _add(sw2d_mod, b, k, ends[k])
            b.advance(7 * (24 if k < 7 else 13))
            f0, b0 = _read(b, sid)
        assert bud["t"] == b0["t"] and bud["steps"] == b0["steps"], k
        for x, y in zip(fields, f0):
            assert np.array_equal(x, y), k
        for key in ("rain_in", "outflow", "clamp_gain"):  # FP32 sums over other strips
            assert bud[key] == pytest.approx(b0[key], rel=1e-6, abs=1e-9), (k, key)


def test_the_running_ones_are_cut_for_themselves(sw2d_mod):
    """12 of 240 still run: as fast as 12 alone (nearly four times as long with heights
    chosen for all 240)."""
    best = {}
    for n in (12, 240):
        with sw2d_mod.Batch(max_scenarios=256, chunk=24) as b:
            for k in range(n):
                _add(sw2d_mod, b, k, 1e9 if k < 12 else 0.5)
            for _ in range(3):
                assert b.advance(48) in (12, n)
            for _ in range(5):
                t = time.perf_counter()
                assert b.advance(96) == 12
                best[n] = min(best.get(n, 1.0), time.perf_counter() - t)
    assert best[240] < 1.5 * best[12], best
