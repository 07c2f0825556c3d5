"""A row of the FP32 rgbnet is the same bits wherever it lies: in a 128-row tile
or in a 32-row tile of the remainder. The renderer takes its rows in the order in
which its warps finish, so a frame repeats only if this holds."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _both_kinds(rows):
    """Whether `rows` rows come to full rounds of 128-row tiles and 32-row tiles."""
    import torch
    units = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    return 0 < rows % (128 * units) <= 96 * units and rows > 128 * units


@pytest.mark.parametrize("c0", [3, 12, 15])
def test_equal_rows_give_equal_bits(lib, c0):
    import torch
    from plenvdb_gb300 import ColorVDB, DensityVDB
    from plenvdb_gb300.march import MarchSample, MarchWorkspace, RgbNetFn, march_params
    from plenvdb_gb300.scene import CameraConfig, SceneConfig, random_rays, rgbnet_init, scene_mask
    from plenvdb_gb300.trainer import FineStageConfig
    scfg = SceneConfig(reso=64, n_ellipsoids=6, seed=5)
    act = scene_mask(scfg)
    ro, rd, vd = [torch.from_numpy(a).cuda() for a in random_rays(CameraConfig(), 16384, 8, seed=2)]
    cfg = FineStageConfig(reso=64)
    dg = DensityVDB.from_mask([64] * 3, act, background=-10.0)
    kg = ColorVDB.from_mask([64] * 3, act, background=0.0, n=c0)
    dg.copyFromDense(np.where(act > 0, 2.0, -10.0).astype(np.float32).reshape(-1))
    p = march_params(cfg.xyz_min, cfg.xyz_max, cfg.near, cfg.stepdist, cfg.act_shift,
                     cfg.interval, cfg.fast_color_thres)
    dummy = torch.zeros(1, device="cuda")
    ws = MarchWorkspace(ro.shape[0], cfg.xyz_min, cfg.xyz_max, cfg.stepdist)
    with torch.no_grad():
        _, _, k0, rid = MarchSample.apply(dummy, ws, dg, kg, ro, rd, p)
        n = int(rid[40000]) + 1
        _, _, k0, rid = MarchSample.apply(dummy, ws, dg, kg, ro[:n], rd[:n], p)
        M = k0.shape[0]
        assert _both_kinds(M)
        # 61 kinds of rows, all with the same view direction
        gen = torch.Generator(device="cuda").manual_seed(c0)
        kinds = torch.randn(61, c0, generator=gen, device="cuda")
        which = torch.arange(M, device="cuda") % 61
        params = [t.cuda() for t in rgbnet_init(c0=c0, seed=7)]
        rgb = RgbNetFn.apply(kinds[which].contiguous(), vd[:1].expand(n, 3).contiguous(), ws, 4, 0,
                             *params)
    assert torch.equal(rgb, rgb[:61][which])


def test_frame_repeats(lib):
    from plenvdb_gb300 import _lib as L
    from plenvdb_gb300.plenvdb import device_view
    from plenvdb_gb300.renderer import MGRenderer
    from plenvdb_gb300.scene import look_at_c2w, rgbnet_init
    rng = np.random.default_rng(8)
    reso, W, H = (48, 48, 48), 131, 120
    act = rng.random(reso) < 0.6
    idx = np.zeros(reso, np.int32)
    idx[act] = 1 + np.arange(int(act.sum()))
    n = int(idx.max()) + 1
    net = [t.numpy().astype(np.float64) for t in rgbnet_init(seed=3)]
    r = MGRenderer(12, 27, 128, 3)
    r.load_data(rng.normal(0.5, 1, n), rng.normal(0, 0.3, (n, 12)), idx, n)
    r.load_params(*[np.ascontiguousarray(t.T) if t.ndim == 2 else t for t in net])
    r.setScene(list(reso), np.array([[150, 0, W / 2], [0, 150, H / 2], [0, 0, 1]], np.float32),
               [-1.5] * 3, [1.5] * 3)
    r.input_a_c2w(look_at_c2w(np.array([2.9, -2.1, 1.9])))
    r.setKwargs(0.5, 1e9, 0.03, -4.6, 0.5, 1e-4, 0.7, False, H, W, t_stop=1e-3)
    r.render_an_image()
    rows = C.c_void_p()
    L.load().pvdb_renderer_views(r.h, None, C.byref(rows))
    total = int(device_view(rows.value, (1,), "int32", r))
    # the image rows that give frames with both kinds of tile
    h, frames = H, []
    while not _both_kinds(total) and h > 8:
        h -= 4
        r.setKwargs(0.5, 1e9, 0.03, -4.6, 0.5, 1e-4, 0.7, False, h, W, t_stop=1e-3)
        r.render_an_image()
        total = int(device_view(rows.value, (1,), "int32", r))
    assert _both_kinds(total)
    for _ in range(8):
        r.render_an_image()
        frames.append(r.output_an_image())
    for f in frames[1:]:
        np.testing.assert_array_equal(frames[0].view(np.uint32), f.view(np.uint32))
