"""The budgets of the streaming kernel's forcing forms: the uniform form counts
cells where the others add FP32 rates, and each form leaves out the sums it does
not have. A form gives the budgets of the one that carries everything, and of
one iteration per launch those of several."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS, COLS = 73, 110
KEYS = ("rain_in", "source_in", "evap_out", "outflow", "clamp_gain")
CELLS = np.array([0, 40 * COLS + 26, 40 * COLS + 27, ROWS * COLS - 1], dtype=np.int32)
STORM = (120.0, 10.0, 20.0, 2.0, 1.0, 80.0)


def _run(sw2d, what, idle=(), steps=50, **kw):
    """`what` is set, and `idle` with rates of zero."""
    rng = np.random.default_rng(7)
    z = 0.05 * np.arange(ROWS)[::-1, None] + rng.uniform(0.0, 0.3, (ROWS, COLS))
    z[rng.random(z.shape) < 0.04] = -9999.0
    args = dict(dt_mode=sw2d.DT_CFL, dt=2.0, strip_h=9)
    args.update(kw)
    with sw2d.Solver(rows=ROWS, cols=COLS, dx=5.0, dy=4.0, precision=sw2d.PREC_F32, kernel=sw2d.KERNEL_STREAM,
                     manning=0.05, south_open=1, INT=0.1, LWL=0.05, EV_WL_min=0.02, **args) as g:
        g.set_static(z)
        g.set_state(np.where(rng.random(z.shape) < 0.3, 0.0, rng.uniform(0.0, 0.2, z.shape)))
        g.set_evaporation([0.4, 0.5], 3600.0)
        q = np.array([[0.8, 1.5, 0.1, 0.4], [0.2, 0.9, 0.3, 0.0]])
        if "storm" in what or "storm" in idle:
            g.set_storm(STORM[0] if "storm" in what else 0.0, *STORM[1:])
        elif "rain" in what:
            g.set_rain(sw2d.RAIN_STEP, [60.0], 3600.0)
        if "sources" in what or "sources" in idle:
            g.set_point_sources(CELLS, q if "sources" in what else 0.0 * q, 300.0)
        if "weights" in what or "weights" in idle:
            g.set_rain_weights(rng.uniform(0.2, 1.8, z.shape) if "weights" in what else np.ones(z.shape))
        assert g.advance(steps, 1e9) == steps
        return g.budget(), g.describe().split("form=")[1]


@pytest.mark.parametrize("what, idle, forms", [
    (("rain",), ("sources",), ("uniform", "sources")), (("rain",), ("weights",), ("uniform", "uniform")),
    (("storm",), ("sources",), ("storm", "any")), (("sources",), ("storm",), ("sources", "any")),
    (("rain", "sources"), ("weights",), ("sources", "any")), (("storm",), ("weights",), ("storm", "any"))])
@pytest.mark.parametrize("strip_h", [1, 9, 40])
def test_budgets_do_not_depend_on_the_form(sw2d_mod, what, idle, forms, strip_h):
    a, fa = _run(sw2d_mod, what, strip_h=strip_h)
    b, fb = _run(sw2d_mod, what, idle, strip_h=strip_h)
    assert (fa.split("+")[0], fb.split("+")[0]) == forms
    # counted cells against FP32 sums of a lane's rows, 32 lanes and their rounding
    tol = (strip_h + 8) * 2.0 ** -23
    for k in KEYS:
        assert a[k] == pytest.approx(b[k], rel=tol, abs=1e-12), k
    assert a["rain_in"] > 0.0 or "sources" in what
    assert (a["source_in"] > 0.0) == ("sources" in what) and a["evap_out"] > 0.0


@pytest.mark.parametrize("what", [("rain",), ("storm",), ("sources",), ("rain", "sources"), ("storm", "sources"),
                                  ("rain", "weights"), ("storm", "weights"), ("rain", "sources", "weights")])
@pytest.mark.parametrize("variant", [0, 2])
def test_budgets_of_the_pipelined_launches(sw2d_mod, what, variant):
    kw = dict(dt_mode=sw2d_mod.DT_FIXED, dt=0.2, variant=variant)
    one, _ = _run(sw2d_mod, what, steps_per_launch=1, **kw)
    many, _ = _run(sw2d_mod, what, steps_per_launch=20, **kw)
    assert one["t"] == many["t"]
    for k in KEYS:
        assert one[k] == pytest.approx(many[k], rel=1e-12, abs=1e-12), k  # FP64 sums in another order
