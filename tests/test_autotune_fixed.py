"""A height tuned with one launch per iteration is not put on a fixed-step
handle that may take several: sw2d_create wants strips of at least 8 rows there,
refuses the others where the caller asked for several iterations, and drops to one
per launch where the library chooses."""
import pytest


def _cfg(sw2d, rows, steps, **kw):
    return sw2d.default_config(rows=rows, cols=120, dx=5.0, dy=5.0, precision=sw2d.PREC_F32, dt_mode=sw2d.DT_FIXED,
                               dt=0.1, steps_per_launch=steps, **kw)


def _cache(autotune, tmp_path, rows, strip, fixed=None):
    cache = autotune.Cache(str(tmp_path / f"{rows}-{strip}-{fixed}.json"))
    gpu = f"{autotune.gpu_name(0)}|{autotune.TABLE_VERSION}"
    cache.put(gpu, autotune.size_class(rows, 120), {"strip_h": strip, "variant": 2})
    if fixed is not None:
        cache.put(gpu, autotune.fixed_class(rows, 120), {"strip_h": strip, "variant": 2, "steps_per_launch": fixed})
    return cache


@pytest.mark.parametrize("rows, strip, kept", [(100, 1, False), (100, 4, False), (100, 8, False), (96, 8, True),
                                               (100, 16, True), (5, 1, False), (5, 16, True), (64, 9, True),
                                               (73, 8, False), (73, 9, True)])
@pytest.mark.parametrize("fixed", [None, 1, 48])
@pytest.mark.parametrize("steps", [0, 1, 2, 48])
def test_short_cached_strips(tmp_path, rows, strip, kept, fixed, steps):
    import sw2d
    from sw2d import autotune
    cfg = autotune.apply(_cfg(sw2d, rows, steps), cache=_cache(autotune, tmp_path, rows, strip, fixed))
    one = cfg.steps_per_launch == 1
    assert cfg.steps_per_launch == (fixed if steps == 0 and fixed else steps)
    assert cfg.strip_h == (strip if kept or one else 0) and cfg.variant == 2


@pytest.mark.parametrize("strip", [1, 4, 8])
def test_cfl_handles_keep_the_tuned_height(tmp_path, strip):
    import sw2d
    from sw2d import autotune
    cfg = _cfg(sw2d, 100, 0)
    cfg.dt_mode = sw2d.DT_CFL
    assert autotune.apply(cfg, cache=_cache(autotune, tmp_path, 100, strip)).strip_h == strip


@pytest.mark.gpu
@pytest.mark.parametrize("strip", [1, 8])
def test_a_tuned_fixed_step_handle_stays_pipelined(sw2d_mod, tmp_path, monkeypatch, strip):
    from sw2d import autotune
    monkeypatch.setenv("SW2D_AUTOTUNE_CACHE", str(tmp_path / "c.json"))
    kw = dict(rows=100, cols=120, dx=5.0, dy=5.0, precision=sw2d_mod.PREC_F32, dt_mode=sw2d_mod.DT_FIXED, dt=0.1)
    autotune.Cache().put(f"{autotune.gpu_name(0)}|{autotune.TABLE_VERSION}", autotune.size_class(100, 120),
                         {"strip_h": strip, "variant": 0})
    for steps in (0, 48):
        with sw2d_mod.Solver(steps_per_launch=steps, **kw) as g:
            assert "steps_per_launch=48" in g.describe()
