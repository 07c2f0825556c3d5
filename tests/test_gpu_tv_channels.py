"""TV for any number of channels: every channel of a multi-channel grid gets the
bits that a scalar grid of that channel's values gets, sparse and dense, with
missing leaves, edges inside the last leaf and inactive voxels; and in the fused
step the terms beside the gradient sums give the bits of TV added in place."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("channels", [3, 12, 15, 24])
@pytest.mark.parametrize("dense", [False, True])
@pytest.mark.parametrize("reso", [(17, 24, 9), (8, 8, 8), (31, 1, 40)])
def test_channels_as_scalar_grids(lib, channels, dense, reso):
    from plenvdb_gb300 import ColorVDB, DensityVDB
    from plenvdb_gb300 import _lib as L
    rng = np.random.default_rng(channels + reso[0])
    act = (rng.random(reso) < 0.4).astype(np.uint8)
    act[:8, :8, :8] = rng.random(act[:8, :8, :8].shape) < 0.9
    if reso[2] > 32:
        act[8:16, :, 8:16] = 0  # missing leaves
    bg = 0.0
    vals = rng.normal(0, 1.5, (*reso, channels)).astype(np.float32)
    grad = rng.normal(0, 1, (*reso, channels)).astype(np.float32)
    grad[rng.random(grad.shape) < 0.4] = 0.0
    g = ColorVDB.from_mask(list(reso), act, background=bg, n=channels)
    g.copyFromDense(vals.reshape(-1))
    g.copyFromDense(grad.reshape(-1), L.WHICH_GRAD)
    g.total_variation_add_grad(0.3, 0.7, 1.1, dense)
    got = g.get_dense_grid(which=L.WHICH_GRAD).reshape(*reso, channels)
    for c in range(channels):
        s = DensityVDB.from_mask(list(reso), act, background=bg)
        s.copyFromDense(np.ascontiguousarray(vals[..., c]).reshape(-1))
        s.copyFromDense(np.ascontiguousarray(grad[..., c]).reshape(-1), L.WHICH_GRAD)
        s.total_variation_add_grad(0.3, 0.7, 1.1, dense)
        want = s.get_dense_grid(which=L.WHICH_GRAD).reshape(reso)
        np.testing.assert_array_equal(got[..., c], want)


@pytest.mark.parametrize("c0", [3, 15])
def test_fused_step_terms(lib, c0):
    import torch
    from plenvdb_gb300.scene import (CameraConfig, SceneConfig, build_grids, random_rays,
                                     rgbnet_init)
    from plenvdb_gb300.trainer import FineStageConfig, FineStageTrainer
    ro, rd, vd = random_rays(CameraConfig(), 512, 20, seed=13)
    tgt = np.random.default_rng(14).random((512, 3)).astype(np.float32)
    dev = [torch.from_numpy(a).cuda() for a in (ro, rd, vd, tgt)]
    out = []
    for in_place, weight in ((False, 1e-2), (True, 1e-2), (False, 0.0)):
        dg, kg = build_grids(SceneConfig(reso=43, n_ellipsoids=4, seed=3, k0_dim=c0))
        cfg = FineStageConfig(reso=43, tv_weight=weight, tv_in_place=in_place)
        tr = FineStageTrainer(dg, kg, rgbnet_init(c0=c0, seed=2), cfg, max_rays=512)
        losses = [float(tr.step(*dev)) for _ in range(3)]
        out.append((losses, dg.get_dense_grid(), kg.get_dense_grid(), tr.params.cpu().numpy()))
    assert out[0][0] == out[1][0]
    for x, y in zip(out[0][1:], out[1][1:]):
        np.testing.assert_array_equal(x, y)
    assert not np.array_equal(out[0][2], out[2][2])  # (the weight moves the values)
