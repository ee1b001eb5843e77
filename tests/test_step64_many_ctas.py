"""The FP64 kernel where a grid has more CTAs than the GPU has SMs: the launches
do not overlap, and bed and mask are staged after the plan. Bit for bit the
oracle's, with every kind of roughness and forcing, and when an advance ends in
the middle of a replay, whose last launches do nothing."""
import numpy as np
import pytest

from helpers import make_pair, same, set_forcing

pytestmark = pytest.mark.gpu


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("tile, shape", [((4, 8), (150, 170)), ((8, 16), (250, 321)), ((6, 32), (301, 290)),
                                         ((10, 32), (415, 333)), ((14, 32), (423, 350)), ((16, 32), (481, 357))])
@pytest.mark.parametrize("form", ["raster", "storm", "fixed", "holes"])
def test_many_ctas_match_the_oracle(oracle_mod, sw2d_mod, tile, shape, form):
    rows, cols = shape
    assert -(-rows // tile[0]) * -(-cols // tile[1]) > _sms()
    rng = np.random.default_rng(rows * cols)
    z = 0.05 * np.arange(rows)[::-1, None] + rng.uniform(0.0, 0.2, shape)
    h = np.where(rng.random(shape) < 0.3, 0.0, rng.uniform(0.0, 0.15, shape))
    if form == "holes":
        z[rng.random(shape) < 0.06] = -9999.0
    n = rng.choice([0.0, 0.03, 0.12], shape) if form in ("raster", "holes") else None
    fixed = form == "fixed"
    kw = dict(INT=0.2, INF=0.1, LWL=0.3, EV_WL_min=0.01) if fixed else {}
    o, g = make_pair(oracle_mod, sw2d_mod, rows, cols, 4.0, z, h, n=n, manning=0.05 if fixed else 0.0,
                     south_open=form in ("raster", "fixed"), dt_mode=0 if fixed else 1, dt=0.05 if fixed else 1.0,
                     dy=3.0, tile=tile, **kw)
    if form == "storm":
        set_forcing(oracle_mod, o, g, storm={"peak": 200.0, "x0": 0.0, "y0": 0.0, "vx": 9.0, "vy": 9.0,
                                             "sigma": 300.0})
    elif fixed:
        set_forcing(oracle_mod, o, g, rain_kind=1, rain=np.array([4.0, 9.0, 2.0]), rain_dt=50.7,
                    ev=np.array([0.5, 0.7]), ev_dt=60.3, sources=np.array([0, rows * cols - 1], dtype=np.int32),
                    src_q=np.array([[0.02, 0.01], [0.05, 0.0]]), dtoq=70.1)
    else:
        set_forcing(oracle_mod, o, g, rain_kind=2, rain=np.array([120.0]), rain_dt=3600.0)
    # 11 iterations, launched one by one; then to an end time inside a replay of 48
    assert o.advance(11, 1e9) == g.advance(11, 1e9) == 11
    t_end = o.state()["t"] + (0.77 if fixed else 5.3)
    done = o.advance(10 ** 6, t_end)
    assert 0 < done == g.advance(10 ** 6, t_end) and done % 48
    a, b = o.state(), g.state()
    for k in ("h", "um", "vn"):
        assert same(a[k], b[k]), (k, np.max(np.abs(a[k] - b[k])))
    bo, bg = o.budget(), g.budget()
    assert bg["cmax"] == bo["cmax"] and bg["t"] == a["t"]
    for k in ("rain_in", "source_in", "evap_out", "outflow", "clamp_gain"):
        assert bg[k] == pytest.approx(bo[k], rel=1e-12, abs=1e-14), k  # sums in another order
    g.close()
