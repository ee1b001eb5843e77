"""The streaming kernel's forcing forms (uniform rain, moving storm, point
sources, both): the form that carries only what is set gives the bits of the
one that carries everything, reached here by setting the other forcing to a
rate of zero."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(sw2d, rows, cols, raster, strip_h):
    rng = np.random.default_rng(rows * cols)
    z = 0.05 * np.arange(rows)[::-1, None] + rng.uniform(0.0, 0.3, (rows, cols))
    z[rng.random(z.shape) < 0.04] = -9999.0
    g = sw2d.Solver(rows=rows, cols=cols, dx=5.0, dy=4.0, precision=sw2d.PREC_F32, kernel=sw2d.KERNEL_STREAM,
                    dt_mode=sw2d.DT_CFL, dt=2.0, manning=0.05, south_open=1, INT=0.1, LWL=0.05, EV_WL_min=0.02,
                    strip_h=strip_h)
    g.set_static(z, rng.choice([0.03, 0.08], z.shape) if raster else None)
    g.set_state(np.where(rng.random(z.shape) < 0.3, 0.0, rng.uniform(0.0, 0.2, z.shape)))
    g.set_evaporation([0.4, 0.5], 3600.0)
    return g


@pytest.mark.parametrize("shape, strip_h", [((1, 1), 0), ((30, 28), 1), ((65, 110), 16), ((90, 55), 30)])
@pytest.mark.parametrize("raster", [True, False])
def test_forms_agree(sw2d_mod, shape, strip_h, raster):
    rows, cols = shape
    cells = np.array([0, rows * cols // 2], dtype=np.int32)
    q = np.array([[0.8, 1.5], [0.2, 0.9]])
    storm = (120.0, 10.0, 20.0, 2.0, 1.0, 80.0)

    def both(alone, with_idle):
        out = []
        for extra in (False, True):
            g = _solver(sw2d_mod, rows, cols, raster, strip_h)
            alone(g)
            if extra:
                with_idle(g)
            assert g.advance(50, 1e9) == 50
            out.append((g.state(), g.budget()))
            g.close()
        (a, ba), (b, bb) = out
        for k in ("h", "um", "vn"):
            assert np.array_equal(a[k], b[k]), k
        assert ba["t"] == bb["t"] and ba["cmax"] == bb["cmax"]

    # storm alone; storm and sources of no inflow
    both(lambda g: g.set_storm(*storm), lambda g: g.set_point_sources(cells, 0.0 * q, 300.0))
    # sources without rain; sources and a storm of no rain
    both(lambda g: g.set_point_sources(cells, q, 300.0), lambda g: g.set_storm(0.0, *storm[1:]))


@pytest.mark.parametrize("variant", [0, 2, 3, 4, 5])
@pytest.mark.parametrize("form", ["storm", "sources", "both", "sources+weights", "storm+weights"])
def test_pipelined_forms_agree(sw2d_mod, variant, form):
    """Every form and build of the pipelined launches against one launch per
    iteration, in strips of 8 and 9 rows (8 is the least) and of 12 and 13."""
    rng = np.random.default_rng(variant)
    rows, cols = 73, 110
    z = 0.05 * np.arange(rows)[::-1, None] + rng.uniform(0.0, 0.3, (rows, cols))
    h = rng.uniform(0.0, 0.2, z.shape)
    w = rng.uniform(0.2, 1.8, z.shape)
    cells = np.array([0, 40 * cols + 26, 40 * cols + 27, rows * cols - 1], dtype=np.int32)
    for strip_h in (9, 13):
        out = []
        for k in (1, 20):
            with sw2d_mod.Solver(rows=rows, cols=cols, dx=5.0, dy=4.0, precision=sw2d_mod.PREC_F32, dt=0.2,
                                 dt_mode=sw2d_mod.DT_FIXED, kernel=sw2d_mod.KERNEL_STREAM, manning=0.05, south_open=1,
                                 strip_h=strip_h, variant=variant, steps_per_launch=k) as g:
                g.set_static(z, None)
                g.set_state(h)
                if "storm" in form or form == "both":
                    g.set_storm(120.0, 10.0, 20.0, 2.0, 1.0, 80.0)
                else:
                    g.set_rain(sw2d_mod.RAIN_STEP, [60.0], 600.0)
                if form in ("sources", "both", "sources+weights"):
                    g.set_point_sources(cells, np.array([[0.8, 1.5, 0.1, 0.4], [0.2, 0.9, 0.3, 0.0]]), 10.0)
                if "weights" in form:
                    g.set_rain_weights(w)
                assert ("stream_pipe_kernel" in g.describe()) == (k > 1)
                assert g.advance(50) == 50
                out.append((g.state(), g.budget()["t"]))
        (a, ta), (b, tb) = out
        assert ta == tb
        for key in ("h", "um", "vn"):
            assert np.array_equal(a[key], b[key]), (strip_h, key)


def test_point_sources_stay_with_the_pipelined_launches(sw2d_mod):
    with sw2d_mod.Solver(rows=100, cols=120, dx=5.0, dy=5.0, precision=sw2d_mod.PREC_F32, dt=0.2,
                         dt_mode=sw2d_mod.DT_FIXED) as g:
        g.set_point_sources(np.array([7], dtype=np.int32), np.ones((2, 1)), 10.0)
        assert "stream_pipe_kernel" in g.describe() and "steps_per_launch=48" in g.describe()
