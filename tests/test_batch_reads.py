"""Reading a batch's scenarios after any number of launches: the budgets that the
last launch left unfolded are those that the next one folds, reads change nothing,
and a field's read does not pay for them."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("t", "dt", "cmax", "volume", "rain_in", "source_in", "evap_out", "outflow", "clamp_gain", "steps")


def _batch(sw2d, sides, **kw):
    b = sw2d.Batch(max_scenarios=max(2, len(sides)), **kw)
    ids = []
    for k, side in enumerate(sides):
        rng = np.random.default_rng(k)
        z = 0.05 * np.arange(side)[::-1, None] + rng.uniform(0.0, 0.3, (side, side))
        cfg = sw2d.default_config(rows=side, cols=side, dx=5.0, dy=5.0, precision=sw2d.PREC_F32, dt_mode=sw2d.DT_CFL,
                                  dt=2.0, cfl=0.5, south_open=1, manning=0.05, LWL=0.1, EV_WL_min=0.02)
        ids.append(b.add(cfg, z, rng.uniform(0.0, 0.2, z.shape), rain_kind=sw2d.RAIN_STEP, rain=[60.0],
                         rain_dt=3600.0, t_end=40.0 if k == 1 else 1e9))
    return b, ids


def test_reads_between_launches_change_nothing(sw2d_mod):
    """One batch read after every launch, one at the end only; a scenario that ends
    on the way among them."""
    sides, launches = (20, 45, 130), 50
    quiet, qi = _batch(sw2d_mod, sides, chunk=3)
    read, ri = _batch(sw2d_mod, sides, chunk=3)
    seen = {i: [] for i in ri}
    for _ in range(launches):
        read.advance(1)
        quiet.advance(1)
        for i in ri:
            a, b = read.budget(i), read.budget(i)
            assert all(a[k] == b[k] for k in KEYS)
            seen[i].append(a["rain_in"])
    for i, q in zip(ri, qi):
        a, b = read.budget(i), quiet.budget(q)
        # the same terms; the order in which the warps' sums reach a bucket varies
        for k in KEYS:
            assert a[k] == pytest.approx(b[k], rel=1e-12, abs=1e-12), k
        assert np.all(np.diff(seen[i]) >= 0.0) and seen[i][0] > 0.0
        for f in (0, 1, 2):
            assert np.array_equal(read.field(i, f), quiet.field(q, f))
    quiet.close()
    read.close()


def test_a_launch_accounts_for_its_own_rain(sw2d_mod):
    """Uniform rain over active cells: the budget of every iteration is rate x area x
    step, at once after its launch."""
    b, ids = _batch(sw2d_mod, (64,))
    area, rate, want = 64 * 64 * 25.0, 60.0 / 3.6e6, 0.0
    for _ in range(7):
        b.advance(1)
        bud = b.budget(ids[0])
        want += 2.0 * bud["dt"]
        # the runoff fraction of wet cells is 0.9
        assert 0.9 * rate * area * want <= bud["rain_in"] * (1 + 1e-6)
        assert bud["rain_in"] <= rate * area * want * (1 + 1e-6)
        assert bud["t"] == pytest.approx(want, rel=1e-12)
    b.close()


def test_a_small_field_costs_a_clock_copy_and_its_own(sw2d_mod):
    """Against the budget's read, which sums the volume besides: a fold kernel in both
    made a 64 x 64 field 39.6 us and a budget 47.6; 28.6 and 37.3 without."""
    b, ids = _batch(sw2d_mod, (64,) * 24)
    best = 1.0
    for _ in range(15):
        b.advance(3)
        b.budget(ids[0])
        t = time.perf_counter()
        for i in ids:
            b.field(i)
        best = min(best, (time.perf_counter() - t) / len(ids))
    with sw2d_mod.Solver(rows=64, cols=64, dx=5.0, dy=5.0, precision=sw2d_mod.PREC_F32) as g:
        g.set_static(np.zeros((64, 64)))
        g.set_state(np.ones((64, 64)))
        alone = 1.0
        for _ in range(60):
            t = time.perf_counter()
            g.depth()
            alone = min(alone, time.perf_counter() - t)
    # the handle's read is an unpacking, a copy and a wait; the batch adds a copy and a wait
    assert best < 2.2 * alone, (best, alone)
    b.close()
