"""rgbnet weights that are views into a flat parameter buffer, at offsets off a
16-byte boundary: the same bits as with tensors of their own, forward and
backward, in both precisions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("c0", [3, 12, 15])
def test_weights_at_any_offset(lib, c0, precision):
    import torch
    from plenvdb_gb300 import ColorVDB, DensityVDB
    from plenvdb_gb300.march import MarchSample, MarchWorkspace, RgbNetFn, march_params
    from plenvdb_gb300.scene import CameraConfig, SceneConfig, random_rays, rgbnet_init, scene_mask
    from plenvdb_gb300.trainer import FineStageConfig
    act = scene_mask(SceneConfig(reso=40, n_ellipsoids=4, seed=3))
    ro, rd, vd = [torch.from_numpy(a).cuda() for a in random_rays(CameraConfig(), 512, 8, seed=2)]
    cfg = FineStageConfig(reso=40)
    dg = DensityVDB.from_mask([40] * 3, act, background=-10.0)
    kg = ColorVDB.from_mask([40] * 3, act, background=0.0, n=c0)
    dg.copyFromDense(np.where(act > 0, 2.0, -10.0).astype(np.float32).reshape(-1))
    p = march_params(cfg.xyz_min, cfg.xyz_max, cfg.near, cfg.stepdist, cfg.act_shift,
                     cfg.interval, cfg.fast_color_thres)
    ws = MarchWorkspace(ro.shape[0], cfg.xyz_min, cfg.xyz_max, cfg.stepdist)
    with torch.no_grad():
        _, _, k0, _ = MarchSample.apply(torch.zeros(1, device="cuda"), ws, dg, kg, ro, rd, p)
    gen = torch.Generator(device="cuda").manual_seed(c0)
    k0 = torch.randn(k0.shape, generator=gen, device="cuda")
    g = torch.randn(k0.shape[0], 3, generator=gen, device="cuda")
    params = [t.cuda() for t in rgbnet_init(c0=c0, seed=7)]
    flat = torch.cat([t.reshape(-1) for t in params])

    def run(net):
        net = [t.detach().requires_grad_() for t in net]
        x = k0.clone().requires_grad_()
        rgb = RgbNetFn.apply(x, vd, ws, 4, precision, *net)
        rgb.backward(g)
        return [rgb.detach(), x.grad] + [t.grad for t in net]

    want = run(params)
    for off in (1, 2, 3):
        buf = torch.empty(flat.numel() + off, device="cuda")
        buf[off:] = flat
        views, at = [], off
        for t in params:
            views.append(buf[at:at + t.numel()].view(t.shape))
            at += t.numel()
        assert views[2].data_ptr() % 16 == 4 * off
        for a, b in zip(want, run(views)):
            assert torch.equal(a, b)
