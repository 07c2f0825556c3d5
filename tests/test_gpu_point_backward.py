"""The point backward against the fixed-scratch entry point, which sorts the
(slot, corner) pairs: bit for bit the same gradient and the same touched
leaves, on both of its forms (one block for up to 2048 points, cells beyond),
at their edges, with points outside the lattice, on its faces, in one cell,
with zero, negative-zero, infinite and NaN gradients, and for every channel
grouping. Then the 12-channel forward against its general form."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _points(kind, n, reso, rng):
    r = np.array(reso, np.float32)
    if kind == "spread":  # also outside the lattice on every side
        return rng.uniform(-9.5, r + 9.5, (n, 3))
    if kind == "cell":    # all in one cell
        return np.array([5, 7, 15]) + rng.uniform(0, 1, (n, 3))
    if kind == "faces":   # on voxel planes and at the lattice's ends
        return rng.integers(-1, np.array(reso) + 1, (n, 3)).astype(np.float64)
    t = rng.uniform(0, 1, (n, 1))  # "line": neighbours share cells
    return (0.1 + t * 0.8) * (r - 1) + rng.uniform(-0.2, 0.2, (n, 3))


@pytest.mark.parametrize("channels", [1, 3, 12, 15])
@pytest.mark.parametrize("kind,n", [("spread", 1), ("spread", 63), ("spread", 2048),
                                    ("spread", 2049), ("line", 1500), ("line", 30000),
                                    ("cell", 700), ("cell", 5000), ("faces", 1025),
                                    ("faces", 20000)])
def test_matches_the_pair_sort(lib, channels, kind, n):
    import torch
    from plenvdb_gb300 import ColorVDB, DensityVDB
    from plenvdb_gb300 import _lib as L
    rng = np.random.default_rng(n + channels)
    reso = [37, 24, 41]
    act = (rng.random(reso) < 0.02).astype(np.uint8)
    act[16:24, :8, 32:] = 0  # some leaves missing
    cls = DensityVDB if channels == 1 else ColorVDB
    a, b = (cls.from_mask(reso, act, background=-1.0, n=channels) for _ in range(2))
    for it in range(2):  # the second call adds to the first's gradient
        xyz = torch.from_numpy(_points(kind, n, reso, rng).astype(np.float32)).cuda()
        xs, ys, zs = (xyz[:, q].contiguous() for q in range(3))
        g = rng.normal(0, 1, (n, channels)).astype(np.float32)
        g[rng.random(n) < 0.3] = 0.0
        g[rng.random(n) < 0.05] = -0.0
        if it == 1 and n > 10:
            g[3], g[5, 0] = np.inf, np.nan
        g = torch.from_numpy(g.reshape(-1)).cuda()
        a.backward(xs, ys, zs, g)
        L.call("pvdb_grid_sample_backward_noalloc", b.handle, L.ptr(xs), L.ptr(ys), L.ptr(zs),
               L.ptr(g), n, L.stream_of())
        ga, gb = (v.get_dense_grid(which=L.WHICH_GRAD).view(np.uint32) for v in (a, b))
        nan = np.isnan(ga.view(np.float32))
        np.testing.assert_array_equal(nan, np.isnan(gb.view(np.float32)))
        np.testing.assert_array_equal(ga[~nan], gb[~nan])
    # the same leaves are touched: zero_grad (which visits those alone) clears all
    for v in (a, b):
        v.zero_grad()
        # (inactive voxels of a touched leaf keep their gradient, as before)
        left = v.get_dense_grid(which=L.WHICH_GRAD).reshape(*reso, channels)
        assert not np.any(left[act > 0])


@pytest.mark.parametrize("channels", [1, 12])
def test_without_memory_for_the_cell_table(lib, channels):
    import torch
    from plenvdb_gb300 import ColorVDB, DensityVDB
    from plenvdb_gb300 import _lib as L
    rng = np.random.default_rng(channels)
    reso, n = [24, 17, 33], 3000
    act = (rng.random(reso) < 0.05).astype(np.uint8)
    cls = DensityVDB if channels == 1 else ColorVDB
    a, b = (cls.from_mask(reso, act, background=-1.0, n=channels) for _ in range(2))
    xyz = torch.from_numpy(_points("spread", n, reso, rng).astype(np.float32)).cuda()
    xs, ys, zs = (xyz[:, q].contiguous() for q in range(3))
    g = torch.from_numpy(rng.normal(0, 1, n * channels).astype(np.float32)).cuda()
    for it in range(2):  # the second call gets its table
        if it == 0:
            L.load().pvdb_debug_fail_next_allocs(1)
        try:
            a.backward(xs, ys, zs, g)
        finally:
            L.load().pvdb_debug_fail_next_allocs(0)
        b.backward(xs, ys, zs, g)
        ga, gb = (v.get_dense_grid(which=L.WHICH_GRAD).view(np.uint32) for v in (a, b))
        np.testing.assert_array_equal(ga, gb)


@pytest.mark.parametrize("n", [1, 255, 257])
def test_color_forward_12_matches_general(lib, n):
    import torch
    from plenvdb_gb300 import ColorVDB
    from plenvdb_gb300 import _lib as L
    rng = np.random.default_rng(n)
    reso = [19, 24, 9]
    act = (rng.random(reso) < 0.05).astype(np.uint8)
    g = ColorVDB.from_mask(reso, act, background=0.25, n=12)
    g.copyFromDense(rng.normal(size=reso + [12]).astype(np.float32).reshape(-1))
    xyz = torch.from_numpy(_points("spread", n, reso, rng).astype(np.float32)).cuda()
    xs, ys, zs = (xyz[:, q].contiguous() for q in range(3))
    out = g.forward(xs, ys, zs)
    # an output that is not on a 16-byte boundary takes the general form
    buf = torch.zeros(n * 12 + 1, device="cuda")
    L.call("pvdb_grid_sample", g.handle, L.ptr(xs), L.ptr(ys), L.ptr(zs), n,
           L.ptr(buf) + 4, L.MEM_DEVICE, L.stream_of())
    assert torch.equal(out, buf[1:])
