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
