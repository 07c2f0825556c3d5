"""The merged-index renderer where its march skips empty blocks and its rows
are laid out by voxel or by row id: odd image sizes (edges of the 8 x 4 pixel
tiles), sparse and empty indices, cameras outside and inside the volume, fine
and coarse steps, and channel counts on both layouts, against the
float-mirroring oracle (equal up to libm ulps; a libm ulp may flip a threshold
on a handful of pixels)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _index(kind, reso, rng):
    act = np.zeros(reso, bool)
    if kind == "voxels":      # isolated voxels: most blocks empty
        act[tuple(rng.integers(0, r, 60) for r in reso)] = True
    elif kind == "slabs":     # thin slabs on block faces
        act[7:9] = True
        act[:, :, 16] = True
        act[-1] = True
    elif kind == "full":
        act[:] = True
    idx = np.zeros(reso, np.int32)
    idx[act] = 1 + rng.permutation(int(act.sum()))
    return idx


@pytest.mark.parametrize("kind,reso,W,H,dcol,storage,inside,stepscale", [
    ("voxels", (41, 37, 50), 33, 21, 12, 0, False, 1.0),
    ("voxels", (40, 40, 40), 61, 3, 12, 0, True, 0.05),
    ("slabs", (40, 33, 47), 7, 70, 12, 1, False, 1.0),
    ("slabs", (24, 24, 24), 40, 40, 3, 0, False, 4.0),
    ("slabs", (24, 24, 24), 25, 31, 15, 1, True, 0.5),
    ("full", (17, 20, 9), 45, 19, 12, 0, False, 1.0),
    ("empty", (16, 16, 16), 9, 5, 12, 1, False, 1.0),
])
def test_render_matches_oracle(lib, kind, reso, W, H, dcol, storage, inside, stepscale):
    import torch
    from plenvdb_gb300.renderer import MGRenderer
    from plenvdb_gb300.scene import look_at_c2w, rgbnet_init
    rng = np.random.default_rng(len(kind) * 100 + W)
    idx = _index(kind, reso, rng)
    n = int(idx.max()) + 1
    den = rng.normal(4.0, 1.0, n).astype(np.float32)
    den[0] = -6.0  # the empty row has a value of its own
    col = rng.normal(0, 0.3, (n, dcol)).astype(np.float32)
    if storage == 1:  # features that BF16 holds exactly
        col = torch.from_numpy(col).to(torch.bfloat16).float().numpy()
    net = [t.numpy().astype(np.float64) for t in rgbnet_init(c0=dcol, seed=3)]
    pos = np.array([0.11, -0.23, 0.31]) if inside else np.array([2.9, -2.1, 1.9])
    pose = look_at_c2w(pos)
    K = np.array([[0.9 * W, 0, W / 2], [0, 0.9 * W, H / 2], [0, 0, 1]], np.float32)
    step = stepscale * 3.0 / max(reso) / 2
    lo, hi = [-1.5, -1.4, -1.5], [1.5, 1.5, 1.3]
    near = 0.0 if inside else 0.5
    kw = dict(near=near, stepdist=step, act_shift=-4.6, interval=0.5, thres=1e-4, bg=0.7,
              t_stop=1e-3)
    r = MGRenderer(dcol, 27, 128, 3)
    r.load_data(den, col, idx, n, storage=storage)
    r.load_params(*[np.ascontiguousarray(t.T) if t.ndim == 2 else t for t in net])
    r.setScene(list(reso), K, lo, hi)
    r.setKwargs(near, 1e9, step, -4.6, 0.5, 1e-4, 0.7, False, H, W, t_stop=1e-3)
    imgs = []
    for precision in (0, 1):
        r.precision = precision
        r.input_a_c2w(pose)
        r.render_an_image()
        imgs.append(r.output_an_image().reshape(-1, 3).astype(np.float64))
    o32, ncol, _ = O.render_pixels(idx, den, col, O.MLPWeights(*net, c0=dcol, pe=4), K, pose, lo,
                                   hi, H, W, fp32=True, **kw)
    assert (ncol > 0).any() == (kind != "empty")
    np.testing.assert_array_equal(imgs[0][ncol == 0], np.float32(0.7))
    far = np.abs(imgs[0] - o32).max(axis=1) > 1e-5
    assert far.mean() <= 0.01, f"{far.sum()} of {far.size} pixels off the fp32 oracle"
    # BF16 rgbnet on the same samples
    assert np.abs(imgs[1] - imgs[0]).max() < 5e-2
