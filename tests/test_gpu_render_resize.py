"""A resize of the renderer that finds no memory for one of its frame buffers: no
frame until a later resize succeeds, and the old size then gives the old frame."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("missing", range(6))  # the buffer that gets no memory
@pytest.mark.parametrize("size", [(50, 61), (8, 8)])
def test_failed_resize(lib, missing, size):
    from plenvdb_gb300 import _lib as L
    from test_gpu_render_status import renderer
    r = renderer()
    r.render_an_image()
    image = r.output_an_image()
    H, W = r._hw
    kw = (0.5, 1e9, 0.06, -4.6, 0.5, 1e-4, 0.7, False)
    try:
        L.load().pvdb_debug_fail_allocs_after(missing, 1)
        with pytest.raises(L.PvdbError):
            r.setKwargs(*kw, *size, t_stop=1e-3)
        with pytest.raises(L.PvdbError, match="setKwargs"):
            r.render_an_image()
        # the old size finds no memory either
        L.load().pvdb_debug_fail_allocs_after(missing, 1)
        with pytest.raises(L.PvdbError):
            r.setKwargs(*kw, H, W, t_stop=1e-3)
        with pytest.raises(L.PvdbError, match="setKwargs"):
            r.render_an_image()
    finally:
        L.load().pvdb_debug_fail_next_allocs(0)
    r.setKwargs(*kw, H, W, t_stop=1e-3)
    r.render_an_image()
    np.testing.assert_array_equal(r.output_an_image(), image)
