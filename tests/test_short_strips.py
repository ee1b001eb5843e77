"""Short strips of the FP32 streaming kernels, which the library picks for grids
that do not fill the GPU: the same bits as one long strip (which runs another
build of the row loop), down to one row, in every forcing form and in the
pipelined launches; and the rule that picks them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(sw2d, rows, cols, form, steps, **kw):
    from sw2d import scenarios as S
    s = S.catchment(rows, dx=5.0, seed=rows + cols, cols=cols)
    z = s["z"].copy()
    rng = np.random.default_rng(rows)
    z[rng.random(z.shape) < 0.04] = -9999.0
    h0 = np.where(rng.random(z.shape) < 0.3, 0.0, rng.uniform(0.0, 0.2, z.shape))
    g = sw2d.Solver(rows=rows, cols=cols, dx=5.0, dy=5.0, precision=sw2d.PREC_F32, south_open=1, **kw)
    g.set_static(z, s["n"])
    g.set_state(h0)
    g.set_rain(sw2d.RAIN_STEP, [90.0], 3600.0)
    if form == "storm":
        g.set_storm(120.0, 0.0, 0.0, 3.0, 3.0, 200.0)
    elif form == "weights":
        g.set_rain_weights(rng.uniform(0.0, 2.0, z.shape))
    elif form == "sources":
        g.set_point_sources(np.array([0, rows * cols // 2], dtype=np.int32), np.array([[1.0, 2.0]]), 100.0)
    assert g.advance(steps, 1e9) == steps
    out = g.state(), g.budget(), g.describe()
    g.close()
    return out


@pytest.mark.parametrize("form", ["uniform", "storm", "weights", "sources"])
@pytest.mark.parametrize("shape", [(1, 1), (2, 40), (17, 27), (33, 55), (64, 100)])
def test_short_strips_give_the_same_bits(sw2d_mod, form, shape):
    kw = dict(dt_mode=sw2d_mod.DT_CFL, dt=2.0)
    want, bw, _ = _run(sw2d_mod, *shape, form, 30, strip_h=64, **kw)
    for sh in (0, 1, 2, 3, 5, 8, 16):
        got, bg, _ = _run(sw2d_mod, *shape, form, 30, strip_h=sh, **kw)
        for k in ("h", "um", "vn"):
            assert np.array_equal(want[k], got[k]), (sh, k)
        assert bg["t"] == bw["t"] and bg["cmax"] == bw["cmax"]
        # FP32 sums of at most 64 rows a lane, in another order
        for k in ("rain_in", "outflow"):
            assert bg[k] == pytest.approx(bw[k], rel=64 * 2.0 ** -24, abs=1e-12), (sh, k)


@pytest.mark.parametrize("shape", [(5, 30), (20, 60), (41, 100), (150, 150)])
def test_short_strips_pipelined(sw2d_mod, shape):
    kw = dict(dt_mode=sw2d_mod.DT_FIXED, dt=0.2)
    want, bw, _ = _run(sw2d_mod, *shape, "uniform", 60, strip_h=150, steps_per_launch=1, **kw)
    got, bg, d = _run(sw2d_mod, *shape, "uniform", 60, **kw)
    assert "steps_per_launch=48" in d
    for k in ("h", "um", "vn"):
        assert np.array_equal(want[k], got[k]), k
    assert bg["t"] == bw["t"]


def test_strip_rule(sw2d_mod):
    """One wave, by the row steps of a strip and the warps sharing an SM."""
    def strip(rows, cols):
        with sw2d_mod.Solver(rows=rows, cols=cols, dx=1.0, dy=1.0, precision=sw2d_mod.PREC_F32,
                             dt_mode=sw2d_mod.DT_CFL, dt=1.0) as g:
            return int(g.describe().split("strip_h=")[1].split()[0])

    assert strip(64, 64) == 1
    assert 1 < strip(300, 300) < 8
    assert strip(512, 512) == 8
    assert strip(2048, 2048) == 52
    assert strip(4096, 4096) == 103  # two waves
