"""The point backward when one of its allocations fails: it answers with its other
form. Without any memory it gives an out-of-memory error with the gradient
unchanged; the next call is exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [5000, 20000])
@pytest.mark.parametrize("channels", [1, 3, 12])
def test_any_allocation_fails(lib, channels, n):
    import torch
    from plenvdb_gb300 import ColorVDB, DensityVDB
    from plenvdb_gb300 import _lib as L
    rng = np.random.default_rng(channels)
    reso = [24, 17, 33]
    act = (rng.random(reso) < 0.05).astype(np.uint8)
    cls = DensityVDB if channels == 1 else ColorVDB
    xyz = torch.from_numpy(rng.uniform(-2, np.array(reso) + 2.0, (n, 3)).astype(np.float32)).cuda()
    xs, ys, zs = (xyz[:, q].contiguous() for q in range(3))
    g = torch.from_numpy(rng.normal(0, 1, n * channels).astype(np.float32)).cuda()

    def grad(v):
        return v.get_dense_grid(which=L.WHICH_GRAD).view(np.uint32)

    ref = cls.from_mask(reso, act, background=-1.0, n=channels)
    ref.backward(xs, ys, zs, g)
    once = grad(ref)
    ref.backward(xs, ys, zs, g)
    twice = grad(ref)
    for skip in range(11):  # more than the call allocates
        v = cls.from_mask(reso, act, background=-1.0, n=channels)
        L.load().pvdb_debug_fail_allocs_after(skip, 1)
        try:
            v.backward(xs, ys, zs, g)
        finally:
            L.load().pvdb_debug_fail_next_allocs(0)
        np.testing.assert_array_equal(grad(v), once)
        v.backward(xs, ys, zs, g)
        np.testing.assert_array_equal(grad(v), twice)
    # no memory at all
    v = cls.from_mask(reso, act, background=-1.0, n=channels)
    L.load().pvdb_debug_fail_next_allocs(100)
    try:
        with pytest.raises(L.PvdbError, match="allocation"):
            v.backward(xs, ys, zs, g)
    finally:
        L.load().pvdb_debug_fail_next_allocs(0)
    assert not grad(v).any()
    v.backward(xs, ys, zs, g)
    np.testing.assert_array_equal(grad(v), once)
