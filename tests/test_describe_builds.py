"""sw2d_describe names what runs: the FP64 kernel and its build, the form of the
streaming kernel for the forcing that is set, the build for short strips, the
unrolling of the pipelined one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw, build", [
    (dict(tile_h=16, tile_w=32), "step64_kernel<16,32,512,2>"), (dict(tile_h=8, tile_w=32), "step64_kernel<8,32,768,1>"),
    (dict(tile_h=4, tile_w=8), "step64_kernel<4,8,256,1>"), (dict(th=0.0), "step64_kernel<16,32,512,2,general>"),
    (dict(EV_WL_min=-1.0, tile_h=4, tile_w=8), "step64_kernel<16,32,512,2,general>")])
def test_fp64_build(sw2d_mod, kw, build):
    with sw2d_mod.Solver(rows=40, cols=60, dx=1.0, dy=1.0, **kw) as g:
        assert g.describe().endswith(" build=" + build), g.describe()


def _set(sw2d, g, what, rows, cols):
    g.set_static(np.zeros((rows, cols)))
    if "storm" in what:
        g.set_storm(50.0, 0.0, 0.0, 1.0, 0.0, 100.0)
    if "sources" in what:
        g.set_point_sources(np.array([3], dtype=np.int32), np.ones((2, 1)), 10.0)
    if "weights" in what:
        g.set_rain_weights(np.ones((rows, cols)))


FORMS = [("", "uniform"), ("storm", "storm"), ("sources", "sources"), ("storm sources", "any"),
         ("weights", "uniform"), ("weights storm", "any"), ("weights sources", "any")]


@pytest.mark.parametrize("what, form", FORMS)
@pytest.mark.parametrize("strip_h", [4, 13, 40])
def test_form_and_short_strips(sw2d_mod, what, form, strip_h):
    for variant in (0, 2, 6):
        with sw2d_mod.Solver(rows=100, cols=60, dx=1.0, dy=1.0, precision=sw2d_mod.PREC_F32, variant=variant,
                             dt_mode=sw2d_mod.DT_CFL, dt=1.0, strip_h=strip_h) as g:
            _set(sw2d_mod, g, what, 100, 60)
            tma = variant == 6 and what == ""
            skip = variant != 2 and not tma and what not in ("weights storm", "weights sources") and \
                strip_h <= (13 if what else 6)
            d = g.describe()
            assert d.endswith(" form=" + form + ("+skip" if skip else "")), d
            assert d.startswith("stream_step_tma_kernel<2,10,2> " if tma else
                                "stream_step_kernel<4,5,2> " if variant == 2 else "stream_step_kernel<2,10,2> "), d


@pytest.mark.parametrize("what, form", FORMS)
def test_pipelined_unrolling(sw2d_mod, what, form):
    with sw2d_mod.Solver(rows=100, cols=60, dx=1.0, dy=1.0, precision=sw2d_mod.PREC_F32, dt=0.1,
                         dt_mode=sw2d_mod.DT_FIXED, steps_per_launch=48) as g:
        _set(sw2d_mod, g, what, 100, 60)
        d = g.describe()
        assert d.startswith("stream_pipe_kernel<2,10,%d> " % (2 if form in ("uniform", "storm") else 1)), d
        assert d.endswith(" form=" + form), d
