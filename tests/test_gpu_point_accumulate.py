"""Several point backwards into one gradient: calls of different sizes, so of
different forms and with the first ones' tables and lists there, against the
fixed-scratch entry point, which sorts the (slot, corner) pairs; the same bits and
the same touched leaves after every call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [1, 3, 12])
@pytest.mark.parametrize("order", [(30000, 300, 20000, 2048, 2049, 30000), (17000, 32000, 9000, 8192)])
def test_calls_add_up(lib, channels, order):
    import torch
    from plenvdb_gb300 import ColorVDB, DensityVDB
    from plenvdb_gb300 import _lib as L
    rng = np.random.default_rng(channels + len(order))
    reso = [57, 40, 33]
    act = (rng.random(reso) < 0.3).astype(np.uint8)
    act[16:24, 8:24] = 0  # some leaves missing
    cls = DensityVDB if channels == 1 else ColorVDB
    a, b = (cls.from_mask(reso, act, background=-1.0, n=channels) for _ in range(2))
    for k, n in enumerate(order):
        # a part of the grid that moves from call to call
        lo = np.array(reso) * rng.uniform(-0.1, 0.6, 3)
        xyz = lo + rng.uniform(0, 1, (n, 3)) * np.array(reso) * (0.5 if k else 1.2)
        xyz = torch.from_numpy(xyz.astype(np.float32)).cuda()
        xs, ys, zs = (xyz[:, q].contiguous() for q in range(3))
        g = rng.normal(0, 1, (n, channels)).astype(np.float32)
        g[rng.random(n) < 0.3] = 0.0
        g = torch.from_numpy(g.reshape(-1)).cuda()
        a.backward(xs, ys, zs, g)
        L.call("pvdb_grid_sample_backward_noalloc", b.handle, L.ptr(xs), L.ptr(ys), L.ptr(zs),
               L.ptr(g), n, L.stream_of())
        ga, gb = (v.get_dense_grid(which=L.WHICH_GRAD).view(np.uint32) for v in (a, b))
        np.testing.assert_array_equal(ga, gb)
        if k == 2:  # what was touched until here is zeroed, and nothing is left of it
            for v in (a, b):
                v.zero_grad()
                left = v.get_dense_grid(which=L.WHICH_GRAD).reshape(*reso, channels)
                assert not np.any(left[act > 0])
