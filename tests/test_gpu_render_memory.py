"""The renderer's load when one of its allocations fails: where only the per-voxel
features find no memory, the features stay in rows and the image is the same, bit
for bit; else load_data fails, render answers that there is no data, and the next
load works."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", [0, 1])
def test_load_without_memory(lib, storage):
    from plenvdb_gb300 import DensityVDB
    from plenvdb_gb300 import _lib as L
    from plenvdb_gb300.renderer import MGRenderer
    from plenvdb_gb300.scene import look_at_c2w, rgbnet_init
    rng = np.random.default_rng(4)
    reso, W, H, n = (24, 17, 33), 40, 33, 7
    idx = rng.integers(0, n, reso).astype(np.int32)  # voxels share rows
    idx[8:16, :8] = 0
    den, col = rng.normal(0.0, 1, n), rng.normal(0, 0.3, (n, 12))
    net = [t.numpy().astype(np.float64) for t in rgbnet_init(seed=3)]
    r = MGRenderer(12, 27, 128, 3)
    r.load_params(*[np.ascontiguousarray(t.T) if t.ndim == 2 else t for t in net])
    r.setScene(list(reso), np.array([[36, 0, W / 2], [0, 36, H / 2], [0, 0, 1]], np.float32),
               [-1.5] * 3, [1.5] * 3)
    r.setKwargs(0.5, 1e9, 0.06, -4.6, 0.5, 1e-4, 0.7, False, H, W, t_stop=1e-3)
    r.input_a_c2w(look_at_c2w(np.array([2.9, -2.1, 1.9])))

    def images():
        out = []
        for r.precision in (0, 1):
            r.render_an_image()
            out.append(r.output_an_image())
        return out

    r.load_data(den, col, idx, n, storage=storage)
    want = images()
    assert (want[0] != np.float32(0.7)).mean() > 0.2
    rows = False
    for skip in range(40):
        L.load().pvdb_debug_fail_allocs_after(skip, 1)
        try:
            r.load_data(den, col, idx, n, storage=storage)
        except L.PvdbError:
            with pytest.raises(L.PvdbError, match="load_data"):
                r.render_an_image()
            continue
        finally:
            try:  # whether the load has met the allocation that fails
                for _ in range(40):
                    DensityVDB([8, 8, 8], 1)
                met = True
            except L.PvdbError:
                met = False
            L.load().pvdb_debug_fail_next_allocs(0)
        for a, b in zip(images(), want):
            np.testing.assert_array_equal(a, b)
        rows = rows or met
        if not met:
            break
    assert rows and not met
