"""Voxels with many points in the point backward, which a warp sums, against the
fixed-scratch entry point, which sorts the (slot, corner) pairs: the same bits.
Point counts around the least count a warp takes, its rounds of 32 points a list
and 256 in all; lists of equal and of very different lengths, whose points come in
turn, in runs, or one list after the other; and a sort wait that gives up."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RESO = [25, 32, 17]


def _run(channels, xyz, g, fill):
    """Both entry points on the points and `fill` others far away (they choose the form)."""
    import torch
    from plenvdb_gb300 import ColorVDB, DensityVDB
    from plenvdb_gb300 import _lib as L
    rng = np.random.default_rng(len(xyz))
    cls = DensityVDB if channels == 1 else ColorVDB
    a, b = (cls.from_mask(RESO, np.ones(RESO, np.uint8), background=-1.0, n=channels)
            for _ in range(2))
    if fill:  # spread over another part of the grid, among the points
        far = np.array([0, 16, 0]) + rng.uniform(0, 1, (fill, 3)) * np.array([24, 15, 16])
        at = np.sort(rng.integers(0, len(xyz) + 1, fill))
        xyz = np.insert(xyz, at, far, axis=0)
        g = np.insert(g, at, rng.normal(0, 1, (fill, channels)), axis=0)
    t = torch.from_numpy(xyz.astype(np.float32)).cuda()
    xs, ys, zs = (t[:, q].contiguous() for q in range(3))
    gt = torch.from_numpy(g.astype(np.float32).reshape(-1)).cuda()
    a.backward(xs, ys, zs, gt)
    L.call("pvdb_grid_sample_backward_noalloc", b.handle, L.ptr(xs), L.ptr(ys), L.ptr(zs),
           L.ptr(gt), len(xyz), L.stream_of())
    ga, gb = (v.get_dense_grid(which=L.WHICH_GRAD).view(np.uint32) for v in (a, b))
    nan = np.isnan(ga.view(np.float32))
    np.testing.assert_array_equal(nan, np.isnan(gb.view(np.float32)))
    np.testing.assert_array_equal(ga[~nan], gb[~nan])
    assert ga.any()


@pytest.mark.parametrize("channels", [1, 3, 12, 15])
@pytest.mark.parametrize("fill", [0, 20000])
@pytest.mark.parametrize("kind", ["cell", "turns", "runs", "halves", "uneven"])
def test_long_voxels(lib, channels, fill, kind):
    rng = np.random.default_rng(len(kind) + channels)
    for n in (31, 32, 33, 64, 65, 255, 257, 300, 1031):
        # the cells around voxel (6, 7, 8): an edge shared by four leaves
        if kind == "cell":
            cell = np.zeros(n, int)
        elif kind == "turns":
            cell = np.arange(n) % 8
        elif kind == "runs":
            cell = (np.arange(n) // 37) % 8
        elif kind == "halves":
            cell = (np.arange(n) >= n // 2) * 7
        else:
            cell = np.where(rng.random(n) < 0.05, rng.integers(1, 8, n), 0)
        base = np.array([6, 7, 8]) - np.stack([cell >> 2, (cell >> 1) & 1, cell & 1], -1)
        xyz = base + rng.uniform(0.01, 0.99, (n, 3))
        g = rng.normal(0, 1, (n, channels))
        g[rng.random(n) < 0.1] = 0.0
        if n > 1000:
            g[5], g[700, 0] = np.inf, np.nan
        _run(channels, xyz, g, fill)


@pytest.mark.parametrize("channels", [1, 12])
def test_given_up_sort_leaves_the_gradient(lib, channels):
    import torch
    from plenvdb_gb300 import ColorVDB, DensityVDB
    from plenvdb_gb300 import _lib as L
    rng = np.random.default_rng(3)
    cls = DensityVDB if channels == 1 else ColorVDB
    n = 30000  # several sort tiles, so the look-back waits
    xyz = torch.from_numpy(rng.uniform(0, 1, (n, 3)).astype(np.float32) * 16).cuda()
    xs, ys, zs = (xyz[:, q].contiguous() for q in range(3))
    g = torch.from_numpy(rng.normal(0, 1, n * channels).astype(np.float32)).cuda()
    a, b = (cls.from_mask(RESO, np.ones(RESO, np.uint8), background=-1.0, n=channels)
            for _ in range(2))
    L.call("pvdb_debug_wait_limit", 4096, 1)
    try:
        with pytest.raises(L.PvdbError, match="timed out"):
            a.backward(xs, ys, zs, g)
    finally:
        L.call("pvdb_debug_wait_limit", 0, 0)
    assert not np.any(a.get_dense_grid(which=L.WHICH_GRAD))
    for v in (a, b):
        v.backward(xs, ys, zs, g)
    np.testing.assert_array_equal(a.get_dense_grid(which=L.WHICH_GRAD),
                                  b.get_dense_grid(which=L.WHICH_GRAD))
    assert np.any(b.get_dense_grid(which=L.WHICH_GRAD))


@pytest.mark.parametrize("channels", [1, 12, 15])
@pytest.mark.parametrize("n", [127, 128, 129, 130])
def test_at_once_and_in_rounds(lib, channels, n):
    """Points around the most that a warp orders at once, spread over the eight lists
    in every way that leaves some of them empty, long or of one point."""
    rng = np.random.default_rng(n + channels)
    for part in range(6):
        w = rng.random(8) ** (1 + 3 * part)
        w[rng.random(8) < 0.1 * part] = 0
        w[part] += 0.1
        cell = rng.choice(8, n, p=w / w.sum())
        if part == 5:
            cell.sort()  # one list after the other
        base = np.array([6, 7, 8]) - np.stack([cell >> 2, (cell >> 1) & 1, cell & 1], -1)
        xyz = base + rng.uniform(0.01, 0.99, (n, 3))
        g = rng.normal(0, 1, (n, channels))
        g[rng.random(n) < 0.05] = 0.0
        _run(channels, xyz, g, 0 if part % 2 else 20000)
