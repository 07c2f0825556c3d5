"""A frame that outgrows the renderer's buffers is marched again: the same image, bit
for bit, as with buffers that held it at once, for the first frame, for one that
needs a little more than the last and for a larger image."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage,dcol", [(0, 12), (1, 12), (1, 3)])
def test_outgrown_buffers(lib, storage, dcol):
    from plenvdb_gb300 import _lib as L
    from plenvdb_gb300.plenvdb import device_view
    from plenvdb_gb300.scene import look_at_c2w
    from test_gpu_render_status import renderer
    kw = (0.5, 1e9, 0.06, -4.6, 0.5, 1e-4, 0.7, False)

    def frames(precision):
        out, totals = [], []
        r = renderer(storage, dcol)
        r.precision = precision
        rows = C.c_void_p()
        L.call("pvdb_renderer_views", r.h, None, C.byref(rows))
        for H, W, pos in ((33, 40, (2.9, -2.1, 1.9)), (33, 40, (2.4, -1.7, 1.6)), (70, 61, (2, 2, 2))):
            r.setKwargs(*kw, H, W, t_stop=1e-3)
            r.input_a_c2w(look_at_c2w(np.array(pos, np.float64)))
            r.render_an_image()
            out.append(r.output_an_image())
            totals.append(int(device_view(rows.value, (1,), "int32", r)))
        return out, totals

    for precision in (0, 1):
        want, rows = frames(precision)
        assert 128 < rows[0] < rows[1] < rows[2]  # each frame outgrows the last one's rows
        L.call("pvdb_debug_render_exact", 1)
        try:
            got, again = frames(precision)
        finally:
            L.call("pvdb_debug_render_exact", 0)
        assert again == rows
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a, b)
