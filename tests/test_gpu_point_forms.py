"""The point backward on both sides of its choice of a form, against the
fixed-scratch entry point (up to 32768 points): few points for the grid's leaves
and many, with all, some and none of them carrying a gradient; the same bits and
the same touched leaves."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [1, 12])
@pytest.mark.parametrize("zero", [0.0, 0.94, 1.0])
@pytest.mark.parametrize("reso,n", [((120, 110, 97), 8192), ((120, 110, 97), 32767),
                                    ((120, 110, 97), 32768), ((71, 80, 57), 32768),
                                    ((40, 40, 40), 8191), ((40, 40, 40), 8192),
                                    ((64, 64, 56), 11468), ((64, 64, 56), 11469)])
def test_both_forms(lib, reso, n, zero, channels):
    import torch
    from plenvdb_gb300 import ColorVDB, DensityVDB
    from plenvdb_gb300 import _lib as L
    rng = np.random.default_rng(n + int(100 * zero))
    cls = DensityVDB if channels == 1 else ColorVDB
    act = np.ones(reso, np.uint8)  # (every leaf: 512 slots each)
    a, b = (cls.from_mask(list(reso), act, background=-1.0, n=channels) for _ in range(2))
    for _ in range(2):
        xyz = rng.uniform(-1.5, np.array(reso) + 0.5, (n, 3))
        xyz[:200] = np.array([9, 4, 6]) + rng.uniform(0, 0.9, (200, 3))  # many in one cell
        t = torch.from_numpy(xyz.astype(np.float32)).cuda()
        xs, ys, zs = (t[:, q].contiguous() for q in range(3))
        g = rng.normal(0, 1, (n, channels)).astype(np.float32)
        g[rng.random(n) < zero] = 0.0
        if zero < 1:
            g[n // 2], g[n - 1] = np.inf, -0.0
        gt = torch.from_numpy(g.reshape(-1)).cuda()
        a.backward(xs, ys, zs, gt)
        L.call("pvdb_grid_sample_backward_noalloc", b.handle, L.ptr(xs), L.ptr(ys), L.ptr(zs),
               L.ptr(gt), n, L.stream_of())
        ga, gb = (torch.from_numpy(v.get_dense_grid(which=L.WHICH_GRAD)) for v in (a, b))
        assert torch.equal(ga.isnan(), gb.isnan())
        assert torch.equal(ga.nan_to_num(7.0).view(torch.int32), gb.nan_to_num(7.0).view(torch.int32))
    for v in (a, b):  # the same leaves are touched
        v.zero_grad()
        assert not v.get_dense_grid(which=L.WHICH_GRAD).any()
