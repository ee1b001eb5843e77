"""What an FP64 handle holds on the device: the planes of a roughness raster
come with the first raster, and a handle that gains or loses one runs like a
new handle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_no_roughness_planes_without_a_raster(sw2d_mod):
    rows = cols = 2048
    planes = 2 * 8 * rows * cols  # of the faces, and a frame of a few per cent
    z, kw = np.zeros((rows, cols)), dict(rows=rows, cols=cols, dx=1.0, dy=1.0, manning=0.03)
    with sw2d_mod.Solver(**kw) as g:
        g.set_static(z)
        without = _free()
        g.set_static(z, z + 0.03)
        assert planes <= without - _free() < 1.1 * planes
        g.set_static(z, z + 0.05)
        g.set_static(z)
        assert planes <= without - _free() < 1.1 * planes


def test_roughness_comes_and_goes(sw2d_mod):
    rng = np.random.default_rng(2)
    shape = (130, 170)
    z, h = rng.uniform(0.0, 0.3, shape), rng.uniform(0.0, 0.4, shape)
    n = rng.choice([0.02, 0.09], shape)

    def run(g, raster):
        g.set_static(z, raster)
        g.set_state(h)
        assert g.advance(60) == 60
        return g.state()

    kw = dict(rows=shape[0], cols=shape[1], dx=4.0, dy=4.0, manning=0.04, dt_mode=sw2d_mod.DT_CFL, dt=1.0)
    with sw2d_mod.Solver(**kw) as g:
        got = [run(g, r) for r in (None, n, None, n + 0.01)]
    for raster, a in zip((None, n, None, n + 0.01), got):
        with sw2d_mod.Solver(**kw) as g:
            b = run(g, raster)
        for k in ("h", "um", "vn"):
            assert np.array_equal(a[k], b[k]), k
