"""The renderer reports a frame whose rgbnet gave up a bounded wait. The status
word that the kernel would set (the word two behind the sample count) is set here
from the host."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def renderer(storage=1, dcol=12):
    from plenvdb_gb300.renderer import MGRenderer
    from plenvdb_gb300.scene import look_at_c2w, rgbnet_init
    rng = np.random.default_rng(4)
    reso, W, H = (24, 24, 24), 40, 33
    act = rng.random(reso) < 0.5
    idx = np.zeros(reso, np.int32)
    idx[act] = 1 + np.arange(int(act.sum()))
    n = int(idx.max()) + 1
    net = [t.numpy().astype(np.float64) for t in rgbnet_init(c0=dcol, seed=3)]
    r = MGRenderer(dcol, 27, 128, 3)
    r.load_data(rng.normal(1.0, 1, n), rng.normal(0, 0.3, (n, dcol)), idx, n, storage=storage)
    r.load_params(*[np.ascontiguousarray(t.T) if t.ndim == 2 else t for t in net])
    r.setScene(list(reso), np.array([[36, 0, W / 2], [0, 36, H / 2], [0, 0, 1]], np.float32),
               [-1.5] * 3, [1.5] * 3)
    r.setKwargs(0.5, 1e9, 0.06, -4.6, 0.5, 1e-4, 0.7, False, H, W, t_stop=1e-3)
    r.input_a_c2w(look_at_c2w(np.array([2.9, -2.1, 1.9])))
    r.precision = 1
    return r


@pytest.mark.parametrize("storage,dcol", [(1, 12), (0, 12), (0, 3)])
def test_given_up_wait_is_reported_once(lib, storage, dcol):
    from plenvdb_gb300 import _lib as L
    from plenvdb_gb300.plenvdb import device_view
    r = renderer(storage, dcol)
    rows = C.c_void_p()
    L.call("pvdb_renderer_views", r.h, None, C.byref(rows))
    status = device_view(rows.value + 8, (1,), "int32", r)
    r.render_an_image()
    image = r.output_an_image()
    assert int(status) == 0 and int(device_view(rows.value, (1,), "int32", r)) > 128
    # taken to the host: reported there
    status.fill_(2)
    with pytest.raises(L.PvdbError, match="timed out"):
        r.output_an_image()
    np.testing.assert_array_equal(r.output_an_image(), image)
    # taken to device memory: reported by the next frame
    status.fill_(2)
    np.testing.assert_array_equal(r.output_an_image(device=True).cpu().numpy(), image)
    with pytest.raises(L.PvdbError, match="timed out"):
        r.render_an_image()
    r.render_an_image()
    np.testing.assert_array_equal(r.output_an_image(), image)
