"""FP32 rgbnet kernels against an FP64 torch reference, at row counts around the
edges of their 32- and 128-row tiles and of the rounds over the SMs, and at
both channel paddings (12 and 16)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

C0S = [3, 12, 15]


@pytest.fixture(scope="module")
def scene(lib):
    import torch
    from plenvdb_gb300.scene import CameraConfig, SceneConfig, random_rays, scene_mask
    scfg = SceneConfig(reso=64, n_ellipsoids=6, seed=5)
    ro, rd, vd = random_rays(CameraConfig(), 16384, 8, seed=2)
    return scfg, scene_mask(scfg), [torch.from_numpy(a).cuda() for a in (ro, rd, vd)]


# 1 row of one tile; a few tiles; 32-row tiles only; full rounds of 128-row
# tiles, a remainder of 32-row tiles, and one large enough for 128-row tiles
@pytest.mark.parametrize("c0", C0S)
@pytest.mark.parametrize("rows", [1, 31, 33, 129, 4000, 14600, 19461, 34100, 38913, 40000])
def test_f32_rgbnet_matches_fp64(scene, c0, rows):
    import torch
    from plenvdb_gb300 import ColorVDB, DensityVDB
    from plenvdb_gb300.march import MarchSample, MarchWorkspace, RgbNetFn, march_params
    from plenvdb_gb300.scene import rgbnet_init
    from plenvdb_gb300.trainer import FineStageConfig
    scfg, act, (ro, rd, vd) = scene
    cfg = FineStageConfig(reso=64)
    dg = DensityVDB.from_mask([64] * 3, act, background=-10.0)
    kg = ColorVDB.from_mask([64] * 3, act, background=0.0, n=c0)
    dens = np.where(act > 0, 2.0, -10.0).astype(np.float32)
    dg.copyFromDense(dens.reshape(-1))
    p = march_params(cfg.xyz_min, cfg.xyz_max, cfg.near, cfg.stepdist, cfg.act_shift,
                     cfg.interval, cfg.fast_color_thres)
    dummy = torch.zeros(1, device="cuda")
    R = ro.shape[0]
    ws = MarchWorkspace(R, cfg.xyz_min, cfg.xyz_max, cfg.stepdist)
    with torch.no_grad():
        _, _, k0, rid = MarchSample.apply(dummy, ws, dg, kg, ro, rd, p)
        assert k0.shape[0] >= 40000
        # as many of the first rays as give at least `rows` rows
        n = int(rid[rows - 1]) + 1
        _, _, k0, rid = MarchSample.apply(dummy, ws, dg, kg, ro[:n], rd[:n], p)
    M = k0.shape[0]
    assert rows <= M < rows + 300
    gen = torch.Generator(device="cuda").manual_seed(rows * 17 + c0)
    k0 = torch.randn(M, c0, generator=gen, device="cuda")
    params = [t.cuda() for t in rgbnet_init(c0=c0, seed=7)]
    g = torch.randn(M, 3, generator=gen, device="cuda")
    # reference, and the rows with a pre-activation near enough to zero that FP32
    # rounding could flip its ReLU: those carry no gradient here
    P = [t.double().requires_grad_() for t in params]
    x0 = k0.double().requires_grad_()
    freq = 2.0 ** torch.arange(4, dtype=torch.float64, device="cuda")
    v = vd[:n].double()
    emb = (v.unsqueeze(-1) * freq).flatten(-2)
    pe = torch.cat([v, emb.sin(), emb.cos()], -1)[rid.long()]
    z0 = torch.cat([x0, pe], -1) @ P[0].T + P[1]
    z1 = torch.relu(z0) @ P[2].T + P[3]
    ref = torch.sigmoid(torch.relu(z1) @ P[4].T + P[5])
    # an accumulated FP32 dot product of 128 terms of size ~1 is off by < 128 * 2^-24 * 4
    near = (z0.abs().amin(-1) < 3e-5) | (z1.abs().amin(-1) < 3e-5)
    g[near] = 0
    (ref * g.double()).sum().backward()
    net = [t.clone().requires_grad_() for t in params]
    k0r = k0.clone().requires_grad_()
    rgb = RgbNetFn.apply(k0r, vd[:n], ws, 4, 0, *net)
    rgb.backward(g)
    assert (rgb.double() - ref).abs().max().item() < 1e-5
    # row gradients: sums of at most 3 * 128 products; weight gradients: sums over
    # the rows, errors add like a random walk (relative to the gradient's norm)
    def rel(a, b):
        return ((a.double() - b).norm() / b.norm().clamp(min=1e-30)).item()
    if (~near).any():
        assert rel(k0r.grad, x0.grad) < 3e-6
        for a, b in zip(net, P):
            assert rel(a.grad, b.grad) < 3e-6
    assert k0r.grad[near].abs().sum().item() == 0
    # the same call again gives the same bits
    net2 = [t.clone().requires_grad_() for t in params]
    k0s = k0.clone().requires_grad_()
    rgb2 = RgbNetFn.apply(k0s, vd[:n], ws, 4, 0, *net2)
    rgb2.backward(g)
    assert torch.equal(rgb, rgb2) and torch.equal(k0r.grad, k0s.grad)
    assert all(torch.equal(a.grad, b.grad) for a, b in zip(net, net2))
