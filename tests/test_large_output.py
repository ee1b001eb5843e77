"""Reading a large field into a fresh buffer and into one in use gives the same
values, whatever the buffer's alignment, and nothing beyond it is written."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 8, 4096 + 24])
def test_large_field_into_any_buffer(sw2d_mod, shift):
    rows, cols = 1700, 1301  # 17.7 MB: above the size whose pages are brought in first
    rng = np.random.default_rng(5)
    h = rng.uniform(0.1, 1.0, (rows, cols))
    with sw2d_mod.Solver(rows=rows, cols=cols, dx=1.0, dy=1.0) as g:
        g.set_static(np.zeros((rows, cols)))
        g.set_state(h)
        lib, n = sw2d_mod.load(), rows * cols * 8
        for fresh in (True, False):
            buf = np.empty(n + shift + 65536, dtype=np.uint8)
            tail = buf[shift + n:]
            if not fresh:
                buf[:] = 7
            tail[:] = 9
            out = buf[shift:shift + n]
            assert lib.sw2d_get_field(g._h, 0, out.ctypes.data_as(C.c_void_p)) == 0
            assert np.array_equal(out.view(np.float64).reshape(rows, cols), h)
            assert np.all(tail == 9)
            if not fresh:
                assert np.all(buf[:shift] == 7)
        assert np.array_equal(g.depth(), h)
