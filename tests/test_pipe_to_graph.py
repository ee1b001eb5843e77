"""A fixed-step handle that has run several iterations per launch and goes over
to one (a storm is set) replays its graph from the clock slot that holds the
state, whichever of the three that is."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _handle(sw2d, steps_per_launch):
    rng = np.random.default_rng(4)
    rows, cols = 90, 120
    z = 0.05 * np.arange(rows)[::-1, None] + rng.uniform(0.0, 0.3, (rows, cols))
    g = sw2d.Solver(rows=rows, cols=cols, dx=5.0, dy=5.0, precision=sw2d.PREC_F32, dt_mode=sw2d.DT_FIXED, dt=0.1,
                    manning=0.05, south_open=1, strip_h=12, steps_per_launch=steps_per_launch)
    g.set_static(z)
    g.set_state(rng.uniform(0.0, 0.2, z.shape))
    g.set_rain(sw2d.RAIN_STEP, [40.0], 1e6)
    return g


@pytest.mark.parametrize("launches", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("steps", [47, 48, 50, 150])
def test_going_over_to_one_iteration_per_launch(sw2d_mod, launches, steps):
    out = []
    for k in (0, 1):
        with _handle(sw2d_mod, k) as g:
            if k == 0:
                assert "steps_per_launch=48" in g.describe()
            for _ in range(launches):
                assert g.advance(5) == 5
            g.set_storm(120.0, 10.0, 20.0, 2.0, 1.0, 200.0)
            assert "steps_per_launch=1" in g.describe()
            assert g.advance(steps) == steps
            mid = g.state(), g.budget()
            g.set_rain(sw2d_mod.RAIN_STEP, [40.0], 1e6)  # and back, and over again
            assert g.advance(60) == 60
            g.set_storm(120.0, 10.0, 20.0, 2.0, 1.0, 200.0)
            assert g.advance(60) == 60
            out.append((mid, (g.state(), g.budget())))
    for (a, ba), (b, bb) in zip(*out):
        assert ba["t"] == bb["t"] and ba["steps"] == bb["steps"]
        for key in ("h", "um", "vn"):
            assert np.array_equal(a[key], b[key]), key
        for key in ("rain_in", "outflow"):
            assert ba[key] == pytest.approx(bb[key], rel=1e-12), key  # FP64 sums in another order
