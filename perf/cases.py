"""Performance cases: the work a user of this framework has it do, through its
public entry points.

A case is a dict with a "kind":

  step     one fine-stage training iteration (FineStageTrainer.step): rays in,
           loss and updated grids / rgbnet / Adam moments out. The trainer is in
           mid-run: every voxel has moments, the optimisers' counters are at
           2000. precision 0 is the default FP32 method, 1 the BF16 one.
  staged   the drop-in path of the reference's training loop: the autograd
           stages MarchSample (with a mask cache), RgbNetFn and CompositeFn,
           the losses in torch, and backward; gradients out.
  density  density-only forward and backward (composited alpha against a
           target), the coarse-geometry form of the march.
  points   the plugin API's grid calls: zero_grad, forward and backward at given
           points: all samples of the rays for the density grid (samples outside
           the scene carry zero gradients, as the alpha threshold leaves them),
           the samples inside the scene for the 12-channel colour grid.
  render   one frame of the merged-VDB renderer: pose in, image out.
  opt      gradient in, TV and voxel Adam on both grids (coarse-stage grids: every
           voxel active).

Scenes follow plenvdb_gb300/scene.py's recipe (bbox [-1.5, 1.5]^3, unions of
seeded ellipsoids, optionally a thin shell, raw density N(2,1) over background
-10, features N(0,0.1), cameras on the sphere of radius 4.03 with focal 1111.1),
made on the GPU. The topology is the same for every seed; values, rays, targets
and gradients come from the seed.
"""
import math

import numpy as np
import torch

BBOX = 1.5
BACKGROUND = -10.0
C0, PE, WIDTH = 12, 4, 128
DIN = C0 + 3 + 6 * PE
STEPSIZE, INTERVAL, ACT_SHIFT, THRES = 0.5, 0.5, -4.6, 1e-4
NEAR, FOCAL, RADIUS = 2.0, 1111.1, 4.03
T_STOP_TRAIN, T_STOP_RENDER = 1e-3, 1e-4
LR_DENSITY, LR_K0, LR_NET = 0.1, 0.075, 1e-3
BETAS, EPS, TV = (0.9, 0.99), 1e-8, 1e-4
W_MAIN, W_ENTROPY, W_RGBPER = 1.0, 1e-3, 1e-2
STEP0 = 2000     # optimiser steps taken before the timed ones
BATCHES = 4      # ray batches (or poses) a state goes through in turn


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest step the tests train with: launches and latency
        dict(name="step_fp32_40_601", kind="step", reso=40, ellipsoids=4, shell=False, rays=601, precision=0),
        # the headline workload, BF16 and the default FP32 method
        dict(name="step_bf16_160_8192", kind="step", reso=160, ellipsoids=8, shell=False, rays=8192, precision=1),
        dict(name="step_fp32_160_8192", kind="step", reso=160, ellipsoids=8, shell=False, rays=8192, precision=0),
        # the larger sparse grid of the benchmark
        dict(name="step_bf16_320_65536", kind="step", reso=320, ellipsoids=32, shell=True, rays=65536, precision=1),
        # the reference's own loop over the drop-in stages, a grid of the progressive scaling
        dict(name="staged_fp32_100_5003", kind="staged", reso=100, ellipsoids=8, shell=False, rays=5003, precision=0),
        # the density-only configuration
        dict(name="density_160_8192", kind="density", reso=160, ellipsoids=8, shell=False, rays=8192),
        # the plugin API's calls of one training iteration, and a short one
        dict(name="points_density_160_8192", kind="points", reso=160, ellipsoids=8, shell=False, rays=8192, channels=1),
        dict(name="points_color_160_8192", kind="points", reso=160, ellipsoids=8, shell=False, rays=8192, channels=12),
        dict(name="points_color_40_203", kind="points", reso=40, ellipsoids=4, shell=False, rays=203, channels=12),
        # the render benchmark's frame, and an odd-sized preview with the default FP32 method
        dict(name="render_bf16_800x800", kind="render", reso=160, ellipsoids=8, shell=False, width=800, height=800, precision=1),
        dict(name="render_fp32_397x301", kind="render", reso=160, ellipsoids=8, shell=False, width=397, height=301, precision=0),
        # the coarse stage's optimiser work (100^3 voxels, all active, dense TV)
        dict(name="opt_100_dense_tv", kind="opt", reso=100, mode=1, dense_tv=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "staged", "density", "points", "points", "render", "opt"])
    if kind == "opt":
        return dict(kind=kind, reso=_log_int(rng, 32, 144), mode=rng.choice([0, 1, 1]), dense_tv=rng.choice([True, False]))
    reso = _log_int(rng, 32, 280)
    case = dict(kind=kind, reso=reso, ellipsoids=rng.choice([4, 8, 16]), shell=False)
    if kind in ("step", "staged"):
        case["precision"] = rng.choice([0, 1])
        # FP32 iterations of large batches would cost more than the largest listed case
        most = 2.4e6 if case["precision"] == 0 else 9e6
        case["rays"] = _log_int(rng, 200, min(40000, most / reso))
        case["shell"] = case["precision"] == 1 and reso >= 200 and rng.random() < 0.5
    elif kind == "density":
        case["rays"] = _log_int(rng, 200, min(40000, 6e6 / reso))
    elif kind == "points":
        case["channels"] = rng.choice([1, 12])
        case["rays"] = _log_int(rng, 100, min(30000, 2e6 / reso))
    else:
        case["precision"] = rng.choice([0, 1])
        side = 420 if case["precision"] == 0 else 900
        case["reso"] = _log_int(rng, 48, 200)
        case["width"], case["height"] = _log_int(rng, 60, side), _log_int(rng, 60, side)
    return case


# ------------------------------------------------------------------ inputs
def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + salt)
    return g


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda")


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda")


def _active(c):
    """Active voxels [R,R,R] (bool): the same for every seed."""
    R = c["reso"]
    if c["kind"] == "opt":
        return torch.ones(R, R, R, dtype=torch.bool, device="cuda")
    rng = np.random.default_rng(0)
    centres = rng.uniform(-1, 1, (c["ellipsoids"], 3))
    radii = rng.uniform(0.15, 0.5, (c["ellipsoids"], 3))
    x = torch.arange(R, device="cuda", dtype=torch.float64) / (R - 1) * (2 * BBOX) - BBOX
    act = torch.zeros(R, R, R, dtype=torch.bool, device="cuda")
    for ce, ra in zip(centres, radii):
        q = [((x - ce[a]) / ra[a]) ** 2 for a in range(3)]
        act |= q[0][:, None, None] + q[1][None, :, None] + q[2][None, None, :] <= 1.0
    if c["shell"]:
        s = x * x
        act |= ((s[:, None, None] + s[None, :, None] + s[None, None, :]).sqrt() - 1.3).abs() < 0.02
    return act


def _values(c, seed, act):
    """Dense density [R,R,R] and features [R,R,R,12], float32."""
    g = _gen(seed, 1)
    R = c["reso"]
    dens = torch.where(act, _randn(g, R, R, R) + 2.0, torch.full((), BACKGROUND, device="cuda"))
    k0 = _randn(g, R, R, R, C0) * 0.1 * act[..., None]
    return dens, k0


def _moments(c, seed, act, channels, salt):
    """First and second moments of a mid-run optimiser, of the size its gradients have."""
    g = _gen(seed, salt)
    R = c["reso"]
    s = 10.0 ** (_rand(g, R, R, R, channels) * 2 - 8)
    return 0.3 * s * _randn(g, R, R, R, channels) * act[..., None], s * s * act[..., None]


def _poses(n, rng):
    """Camera-to-world matrices on the sphere, looking at the origin."""
    out = []
    for _ in range(n):
        p = rng.normal(size=3)
        back = p / np.linalg.norm(p)
        up = np.array([0.0, 0.0, 1.0]) if abs(back[2]) < 0.999 else np.array([0.0, 1.0, 0.0])
        right = np.cross(up, back)
        right /= np.linalg.norm(right)
        m = np.eye(4)
        m[:3, 0], m[:3, 1], m[:3, 2], m[:3, 3] = right, np.cross(back, right), back, RADIUS * back
        out.append(m.astype(np.float32))
    return np.stack(out)


def _rays(n, seed, salt):
    """n rays over random (view, pixel) of 100 cameras: origins, directions, unit directions."""
    poses = torch.from_numpy(_poses(100, np.random.default_rng([int(seed), salt]))).cuda()
    g = _gen(seed, 100 + salt)
    view = torch.randint(0, 100, (n,), generator=g, device="cuda")
    px = torch.randint(0, 800, (n, 2), generator=g, device="cuda").float() + 0.5
    d = torch.stack([(px[:, 0] - 400) / FOCAL, -(px[:, 1] - 400) / FOCAL, -torch.ones_like(px[:, 0])], -1)
    rot = poses[view, :3, :3]
    rd = (d[:, None, :] * rot).sum(-1)
    return poses[view, :3, 3].contiguous(), rd, rd / rd.norm(dim=-1, keepdim=True)


def _targets(vd, seed, salt):
    """Smooth images with some noise, in [0, 1]."""
    g = _gen(seed, 200 + salt)
    f = torch.tensor([[3.0, 1.0, 2.0], [1.0, 4.0, 2.0], [2.0, 2.0, 5.0]], device="cuda")
    return (0.5 + 0.35 * torch.sin(vd @ f) + 0.05 * _randn(g, *vd.shape)).clamp(0, 1)


def _rgbnet(seed):
    """nn.Linear's default init, final bias 0: [w0, b0, w1, b1, w2, b2]."""
    g = _gen(seed, 3)
    out = []
    for i, o in ((DIN, WIDTH), (WIDTH, WIDTH), (WIDTH, 3)):
        out += [(_rand(g, o, i) * 2 - 1) / math.sqrt(i), (_rand(g, o) * 2 - 1) / math.sqrt(i)]
    out[-1].zero_()
    return out


def _stepdist(c):
    return STEPSIZE * 2 * BBOX / c["reso"]


def _mask_cache(act):
    """Occupancy mask of the march: the active voxels and their neighbours."""
    m = torch.nn.functional.max_pool3d(act[None, None].float(), 3, 1, 1)[0, 0]
    return (m > 0).to(torch.uint8).contiguous()


def _point_count(c):
    """Points of a call: about what the rays' samples come to, the same for every seed."""
    per_ray = 1.85 if c["channels"] == 1 else 0.0142 * c["ellipsoids"]
    return int(c["rays"] * per_ray * c["reso"]) | 1


def _sample_points(c, seed, act):
    """Index-space points of the rays' samples, in ray order, and their gradients."""
    R, n = c["reso"], _point_count(c)
    o, d, _ = _rays(c["rays"] * 5 // 4, seed, 0)
    step = np.float32(_stepdist(c))
    inv = 1.0 / torch.where(d == 0, torch.full_like(d, 1e-6), d)
    a, b = (BBOX - o) * inv, (-BBOX - o) * inv
    t0 = torch.minimum(a, b).amax(-1).clamp(min=NEAR)
    t1 = torch.maximum(a, b).amin(-1)
    k = torch.arange(int(math.ceil(2 * BBOX * math.sqrt(3) / step)) + 1, device="cuda")
    t = t0[:, None] + float(step) * k / d.norm(dim=-1, keepdim=True)
    p = ((o[:, None] + d[:, None] * t[..., None] + BBOX) / (2 * BBOX) * (R - 1))[t < t1[:, None]]
    p = p[((p >= 0) & (p <= R - 1)).all(-1)]
    i = p.round().long()
    inside = act[i[:, 0], i[:, 1], i[:, 2]]
    if c["channels"] > 1:
        p, inside = p[inside], inside[inside]
    if p.shape[0] < n:
        p, inside = (x.repeat(n // p.shape[0] + 1, *[1] * (x.ndim - 1)) for x in (p, inside))
    p, inside = p[:n], inside[:n]
    g = _gen(seed, 5)
    grad = _randn(g, p.shape[0], c["channels"]) * 1e-4 * inside[:, None]
    return p.float(), grad


# ----------------------------------------------------------------- prepare
def _grids(c, seed, need_k0=True):
    from plenvdb_gb300 import ColorVDB, DensityVDB
    act = _active(c)
    dens, k0 = _values(c, seed, act)
    u8 = act.to(torch.uint8)
    reso = [c["reso"]] * 3
    dg = DensityVDB.from_mask(reso, u8, background=BACKGROUND)
    dg.copyFromDense(dens.reshape(-1))
    kg = None
    if need_k0:
        kg = ColorVDB.from_mask(reso, u8, background=0.0, n=C0)
        kg.copyFromDense(k0.reshape(-1))
    return act, dg, kg


def _fill_moments(opt, c, seed, act, channels, salt):
    """Sets the optimiser's moments; returns views of them."""
    import ctypes

    from plenvdb_gb300 import _lib as L
    from plenvdb_gb300.plenvdb import device_view
    handles = ctypes.c_void_p(), ctypes.c_void_p()
    L.call("pvdb_opt_moments", opt.h, ctypes.byref(handles[0]), ctypes.byref(handles[1]))
    n = opt.vdb.info()[2] * 512 * channels
    views = []
    for h, v in zip(handles, _moments(c, seed, act, channels, salt)):
        v = v.reshape(-1).contiguous()
        L.call("pvdb_grid_copy_from_dense", h, L.WHICH_DATA, L.ptr(v), v.numel(), L.MEM_DEVICE, L.stream_of())
        p = ctypes.c_void_p()
        L.call("pvdb_grid_device_views", h, ctypes.byref(p), None, None, None, None, None)
        views.append(device_view(p.value, (n,), "float32", opt))
    opt.setStep(STEP0)
    return views


def _net_moments(seed, n):
    g = _gen(seed, 11)
    s = 10.0 ** (_rand(g, n) * 2 - 6)
    return 0.3 * s * _randn(g, n), s * s


def _batches(c, seed, n):
    out = []
    for b in range(n):
        o, d, v = _rays(c["rays"], seed, b)
        out.append((o, d.contiguous(), v.contiguous(), _targets(v, seed, b)))
    return out


def _march_params(c, bg=0.0):
    from plenvdb_gb300.march import march_params
    return march_params([-BBOX] * 3, [BBOX] * 3, NEAR, _stepdist(c), ACT_SHIFT, INTERVAL, THRES, bg, T_STOP_TRAIN)


def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def _prepare_step(c, seed):
    from plenvdb_gb300.trainer import FineStageConfig, FineStageTrainer
    act, dg, kg = _grids(c, seed)
    cfg = FineStageConfig(reso=c["reso"], precision=c["precision"], tv_weight=TV)
    tr = FineStageTrainer(dg, kg, _rgbnet(seed), cfg, max_rays=c["rays"])
    md, vd = _fill_moments(tr.dopt, c, seed, act, 1, 21)
    mk, vk = _fill_moments(tr.kopt, c, seed, act, C0, 22)
    m, v = _net_moments(seed, tr.params.numel())
    tr.exp_avg.copy_(m)
    tr.exp_avg_sq.copy_(v)
    out = {"density": dg.device_views()[0], "k0": kg.device_views()[0], "params": tr.params, "exp_avg": tr.exp_avg,
           "exp_avg_sq": tr.exp_avg_sq, "d_avg": md, "d_avg_sq": vd, "k_avg": mk, "k_avg_sq": vk}
    dg.zero_grad()
    kg.zero_grad()
    return {"kind": "step", "trainer": tr, "batches": _batches(c, seed, BATCHES), "at": 0, "out": out}


def _prepare_staged(c, seed):
    from plenvdb_gb300.march import MarchWorkspace
    act, dg, kg = _grids(c, seed)
    net = [t.requires_grad_() for t in _rgbnet(seed)]
    ws = MarchWorkspace(c["rays"], [-BBOX] * 3, [BBOX] * 3, _stepdist(c))
    grads = dg.device_views()[1], kg.device_views()[1]
    dg.zero_grad()
    kg.zero_grad()
    return {"kind": "staged", "density": dg, "k0": kg, "net": net, "ws": ws, "params": _march_params(c),
            "mask": _mask_cache(act), "precision": c["precision"], "grads": grads,
            "dummy": torch.zeros(1, device="cuda", requires_grad=True), "batches": _batches(c, seed, BATCHES), "at": 0}


def _prepare_density(c, seed):
    from plenvdb_gb300.march import MarchWorkspace
    _, dg, _ = _grids(c, seed, need_k0=False)
    ws = MarchWorkspace(c["rays"], [-BBOX] * 3, [BBOX] * 3, _stepdist(c))
    grad = dg.device_views()[1]
    dg.zero_grad()
    batches = [(o, d.contiguous(), _rand(_gen(seed, 300 + b), c["rays"]))
               for b in range(BATCHES) for o, d, _ in [_rays(c["rays"], seed, b)]]
    return {"kind": "density", "density": dg, "ws": ws, "params": _march_params(c), "grad": grad,
            "dummy": torch.zeros(1, device="cuda", requires_grad=True), "batches": batches, "at": 0}


def _prepare_points(c, seed):
    act, dg, kg = _grids(c, seed, need_k0=c["channels"] > 1)
    grid = dg if c["channels"] == 1 else kg
    p, g = _sample_points(c, seed, act)
    grad = grid.device_views()[1]
    grid.zero_grad()
    return {"kind": "points", "grid": grid, "xyz": [p[:, a].contiguous() for a in range(3)], "g": g.reshape(-1),
            "grad": grad}


def _prepare_render(c, seed):
    from plenvdb_gb300 import MGRenderer
    R = c["reso"]
    act = _active(c)
    dens, k0 = _values(c, seed, act)
    n = int(act.sum())
    index = torch.zeros(R, R, R, dtype=torch.int32, device="cuda")
    index[act] = torch.arange(1, n + 1, dtype=torch.int32, device="cuda")
    den = torch.cat([torch.zeros(1, device="cuda"), dens[act]]).cpu().numpy()
    col = torch.cat([torch.zeros(1, C0, device="cuda"), k0[act]]).cpu().numpy()
    r = MGRenderer(C0, 3 + 6 * PE, WIDTH, 3)
    r.precision = c["precision"]
    r.load_data(den, col, index.cpu().numpy(), n + 1, storage=c["precision"])
    r.load_params(*[(t.T if t.ndim == 2 else t).contiguous().cpu().numpy() for t in _rgbnet(seed)])
    H, W = c["height"], c["width"]
    r.setScene([R] * 3, _intrinsics(c), [-BBOX] * 3, [BBOX] * 3)
    r.setKwargs(NEAR, 6.0, _stepdist(c), ACT_SHIFT, INTERVAL, THRES, 0.0, False, H, W, t_stop=T_STOP_RENDER)
    return {"kind": "render", "renderer": r, "poses": _render_poses(seed), "at": 0}


def _intrinsics(c):
    f = FOCAL * max(c["width"], c["height"]) / 800
    return np.array([[f, 0, c["width"] / 2], [0, f, c["height"] / 2], [0, 0, 1]], np.float32)


def _render_poses(seed):
    return _poses(BATCHES, np.random.default_rng([int(seed), 77]))


def _prepare_opt(c, seed):
    from plenvdb_gb300 import ColorOpt, DensityOpt
    act, dg, kg = _grids(c, seed)
    dopt = DensityOpt(dg, LR_DENSITY, EPS, *BETAS)
    kopt = ColorOpt(kg, LR_K0, EPS, *BETAS)
    md, vd = _fill_moments(dopt, c, seed, act, 1, 21)
    mk, vk = _fill_moments(kopt, c, seed, act, C0, 22)
    gd, gk = _opt_grads(c, seed)
    out = {"density": dg.device_views()[0], "k0": kg.device_views()[0], "d_avg": md, "d_avg_sq": vd, "k_avg": mk,
           "k_avg_sq": vk}
    return {"kind": "opt", "density": dg, "k0": kg, "dopt": dopt, "kopt": kopt, "gd": gd.reshape(-1),
            "gk": gk.reshape(-1), "mode": c["mode"], "dense": c["dense_tv"], "tv": _opt_tv(c), "out": out}


def _opt_grads(c, seed):
    """Gradients of an iteration: a third of the voxels got samples."""
    g = _gen(seed, 31)
    R = c["reso"]
    hit = _rand(g, R, R, R, 1) < 0.33
    return _randn(g, R, R, R, 1) * 1e-6 * hit, _randn(g, R, R, R, C0) * 1e-7 * hit


def _opt_tv(c):
    return TV / 8192 * c["reso"] / 128


# --------------------------------------------------------------------- run
def run(state):
    return _RUN[state["kind"]](state)


def _next(state, what="batches"):
    b = state[what][state["at"]]
    state["at"] = (state["at"] + 1) % len(state[what])
    return b


def _run_step(s):
    loss = s["trainer"].step(*_next(s))
    return {"loss": loss, **s["out"]}


def _run_staged(s):
    from plenvdb_gb300.march import CompositeFn, MarchSample, RgbNetFn
    o, d, v, target = _next(s)
    s["density"].zero_grad()
    s["k0"].zero_grad()
    for t in s["net"]:
        t.grad = None
    w, last, k0, ray = MarchSample.apply(s["dummy"], s["ws"], s["density"], s["k0"], o, d, s["params"], s["mask"])
    rgb = RgbNetFn.apply(k0, v, s["ws"], PE, s["precision"], *s["net"])
    marched = CompositeFn.apply(w, rgb, last, s["ws"], 0.0)
    loss = W_MAIN * torch.nn.functional.mse_loss(marched, target)
    p = last.clamp(1e-6, 1 - 1e-6)
    loss = loss + W_ENTROPY * -(p * torch.log(p) + (1 - p) * torch.log(1 - p)).mean()
    per = (rgb - target[ray.long()]).pow(2).sum(-1)
    loss = loss + W_RGBPER * (per * w.detach()).sum() / o.shape[0]
    loss.backward()
    return {"loss": loss, "rgb": marched, "density": s["grads"][0], "k0": s["grads"][1], "net": [t.grad for t in s["net"]]}


def _run_density(s):
    from plenvdb_gb300.march import MarchSample
    o, d, target = _next(s)
    s["density"].zero_grad()
    _, last, _, _ = MarchSample.apply(s["dummy"], s["ws"], s["density"], None, o, d, s["params"])
    loss = torch.nn.functional.mse_loss(1 - last, target)
    loss.backward()
    return {"loss": loss, "last": last, "density": s["grad"]}


def _run_points(s):
    s["grid"].zero_grad()
    out = s["grid"].forward(*s["xyz"])
    s["grid"].backward(*s["xyz"], s["g"])
    return {"out": out, "grad": s["grad"]}


def _run_render(s):
    r = s["renderer"]
    r.input_a_c2w(_next(s, "poses"))
    r.render_an_image()
    return r.output_an_image(device=True)


def _run_opt(s):
    s["dopt"].set_grad(s["gd"])
    s["kopt"].set_grad(s["gk"])
    s["density"].total_variation_add_grad(s["tv"], s["tv"], s["tv"], s["dense"])
    s["k0"].total_variation_add_grad(s["tv"], s["tv"], s["tv"], s["dense"])
    s["dopt"].step(s["mode"])
    s["kopt"].step(s["mode"])
    return s["out"]


_RUN = {"step": _run_step, "staged": _run_staged, "density": _run_density, "points": _run_points, "render": _run_render,
        "opt": _run_opt}


# -------------------------------------------------------------------- work
def work(case):
    """Each input read once, each output written once; the samples a ray meets
    in these scenes are taken per ray and voxel of resolution (measured: 18
    colour samples and 302 in the bbox per ray at 160^3, 95 with the shell at 320^3)."""
    c, R = case, case["reso"]
    if c["kind"] == "opt":
        n = R ** 3
        return {"bytes": n * 13 * 4.0 * (1 + 6), "flops": n * 13 * 30.0}
    active = R ** 3 * (0.19 if c["shell"] else 0.0065 * c["ellipsoids"])
    rows_per_ray = (0.3 if c["shell"] else 0.0142 * c["ellipsoids"]) * R
    row_flops = 2.0 * (DIN * WIDTH + WIDTH * WIDTH + 3 * WIDTH)
    if c["kind"] == "render":
        # a frame's pixels see less of the scene than random training pixels do
        pixels, rows = c["width"] * c["height"], c["width"] * c["height"] * rows_per_ray * 0.5
        return {"bytes": active * (4.0 + C0 * (2 if c["precision"] else 4)) + 12.0 * pixels, "flops": rows * row_flops}
    rays = c["rays"]
    if c["kind"] == "points":
        n = _point_count(c)
        seen = min(active, 2 * n)
        return {"bytes": n * (12.0 + 8 * c["channels"]) + 8.0 * seen * c["channels"], "flops": n * 32.0 * c["channels"]}
    rows = rays * rows_per_ray
    seen = min(active, 2 * rows)
    if c["kind"] == "density":
        return {"bytes": 28.0 * rays + 8.0 * seen, "flops": rays * 1.9 * R * 60}
    if c["kind"] == "staged":
        return {"bytes": 60.0 * rays + 8.0 * 13 * seen, "flops": 3 * rows * row_flops}
    return {"bytes": 48.0 * rays + 24.0 * 13 * seen, "flops": 3 * rows * row_flops}


# ------------------------------------------------------------------- exact
# The same results in 64 bits, in plain torch.
F64 = torch.float64


def _f32(x):
    """A scalar argument as the calls take it (a C float)."""
    return float(np.float32(x))


def _pad(dense, bg):
    """[R,R,R,C] -> [(R+1)^3, C] in 64 bits, one layer of background at the upper faces."""
    R, C = dense.shape[0], dense.shape[-1]
    out = torch.full((R + 1, R + 1, R + 1, C), bg, dtype=F64, device="cuda")
    out[:R, :R, :R] = dense
    return out.reshape(-1, C)


def _corners(idx, R):
    """Flat indices into the padded grid and weights of the 8 corners, [n, 8] each."""
    f = torch.floor(idx).clamp(0, R - 1)
    u = idx - f
    i = f.long()
    ii, ww = [], []
    for dx in (0, 1):
        for dy in (0, 1):
            for dz in (0, 1):
                ii.append(((i[:, 0] + dx) * (R + 1) + i[:, 1] + dy) * (R + 1) + i[:, 2] + dz)
                w = [(u[:, a] if e else 1 - u[:, a]) for a, e in enumerate((dx, dy, dz))]
                ww.append(w[0] * w[1] * w[2])
    return torch.stack(ii, 1), torch.stack(ww, 1)


def _trilinear(grid, idx, R):
    i, w = _corners(idx, R)
    v = torch.index_select(grid, 0, i.reshape(-1)).reshape(*i.shape, grid.shape[1])
    return (v * w[..., None]).sum(1)


def _alpha(sigma):
    return 1 - (1 + torch.exp(sigma + _f32(ACT_SHIFT))) ** -INTERVAL


def _pe(v):
    x = (v[..., None] * (2.0 ** torch.arange(PE, device="cuda", dtype=F64))).reshape(v.shape[0], -1)
    return torch.cat([v, torch.sin(x), torch.cos(x)], -1)


def _mlp(net, k0, pe):
    h = torch.relu(torch.cat([k0, pe], -1) @ net[0].T + net[1])
    return torch.sigmoid(torch.relu(h @ net[2].T + net[3]) @ net[4].T + net[5])


def _leaves(act):
    """Flat voxel indices [nleaf, 512] of the leaves (Morton order; -1 outside the resolution)."""
    R = act.shape[0]
    L = (R + 7) // 8
    a = torch.zeros(8 * L, 8 * L, 8 * L, dtype=torch.bool, device="cuda")
    a[:R, :R, :R] = act
    lc = a.reshape(L, 8, L, 8, L, 8).any(5).any(3).any(1).nonzero()
    code = torch.zeros(lc.shape[0], dtype=torch.long, device="cuda")
    for b in range(10):
        for ax in range(3):
            code |= ((lc[:, ax] >> b) & 1) << (3 * b + 2 - ax)
    lc = lc[torch.argsort(code)]
    v = torch.arange(512, device="cuda")
    x = lc[:, None, :] * 8 + torch.stack([v >> 6, (v >> 3) & 7, v & 7], -1)[None]
    flat = (x[..., 0] * R + x[..., 1]) * R + x[..., 2]
    return torch.where((x < R).all(-1), flat, torch.full_like(flat, -1))


def _to_leaves(dense, leaves, outside):
    """[R^3, C] -> [nleaf, 512, C]."""
    v = dense[leaves.clamp(min=0)]
    return torch.where((leaves >= 0)[..., None], v, torch.full((), outside, dtype=dense.dtype, device="cuda"))


def _unpad(g, R):
    return g.reshape(R + 1, R + 1, R + 1, -1)[:R, :R, :R].reshape(R ** 3, -1)


def _march64(c, dens, o, d, mask):
    """Kept samples of a chunk of rays: (ray, slot) and index-space positions, and the slots' width."""
    R, step, thr = c["reso"], _f32(_stepdist(c)), _f32(THRES)
    inv = torch.where(d == 0, torch.full_like(d, 1e-6), d)
    a, b = (BBOX - o) / inv, (-BBOX - o) / inv
    t0 = torch.minimum(a, b).amax(-1).clamp(min=NEAR, max=1e9)
    t1 = torch.maximum(a, b).amin(-1).clamp(min=NEAR, max=1e9)
    norm = d.norm(dim=-1)
    n = torch.ceil((t1 - t0) * norm / step).clamp(min=1)
    cap = int(n.max())
    k = torch.arange(cap, device="cuda", dtype=F64)
    p = (o + d * t0[:, None])[:, None] + (d / norm[:, None])[:, None] * (step * k)[None, :, None]
    ok = (k[None] < n[:, None]) & (p.abs() <= BBOX).all(-1)
    if mask is not None:
        j = torch.round((p + BBOX) / (2 * BBOX) * (R - 1)).long().clamp(0, R - 1)
        ok &= mask[j[..., 0], j[..., 1], j[..., 2]] > 0
    idx = (p + BBOX) / (2 * BBOX) * (R - 1)
    al = torch.zeros(ok.shape, dtype=F64, device="cuda")
    al[ok] = _alpha(_trilinear(dens, idx[ok], R)[:, 0])
    kept = al > thr
    T = torch.cumprod(torch.where(kept, 1 - al, torch.ones_like(al)), 1)
    before = torch.cat([torch.ones_like(T[:, :1]), T[:, :-1]], 1)
    kept &= before >= _f32(T_STOP_TRAIN)
    slot = torch.cumsum(kept, 1) - 1
    ray = kept.nonzero()[:, 0]
    return ray, slot[kept], idx[kept], int(kept.sum(1).max()) if kept.numel() else 0


def _composite64(c, dens, o, d, mask):
    """Weights [rays, slots], alphainv_last [rays], and the kept samples."""
    with torch.no_grad():
        ray, slot, idx, width = _march64(c, dens.detach(), o, d, mask)
    al = torch.zeros(o.shape[0], max(width, 1), dtype=F64, device="cuda")
    al = al.index_put((ray, slot), _alpha(_trilinear(dens, idx, c["reso"])[:, 0]))
    T = torch.cumprod(1 - al, 1)
    w = torch.cat([torch.ones_like(T[:, :1]), T[:, :-1]], 1) * al
    return w, T[:, -1], ray, slot, idx


def _fine64(c, dens, k0, net, batch, mask):
    """Loss (its backward done) and marched colours of a batch, in chunks of rays."""
    R, n = c["reso"], c["rays"]
    total, marched = 0.0, []
    for s in range(0, n, 4096):
        o, d, v, target = (x[s:s + 4096].to(F64) for x in batch)
        w, last, ray, slot, idx = _composite64(c, dens, o, d, mask)
        w = w[ray, slot]
        col = (w > _f32(THRES)).nonzero()[:, 0]
        w, ray, idx = w[col], ray[col], idx[col]
        rgb = _mlp(net, _trilinear(k0, idx, R), _pe(v)[ray])
        out = torch.zeros(o.shape[0], 3, dtype=F64, device="cuda").index_add(0, ray, w[:, None] * rgb)
        loss = W_MAIN * (out - target).pow(2).sum() / (3 * n)
        p = last.clamp(1e-6, 1 - 1e-6)
        loss = loss - W_ENTROPY * (p * torch.log(p) + (1 - p) * torch.log(1 - p)).sum() / n
        loss = loss + W_RGBPER * ((rgb - target[ray]).pow(2).sum(-1) * w.detach()).sum() / n
        loss.backward()
        total += float(loss)
        marched.append(out.detach())
    return torch.tensor(total, dtype=F64, device="cuda"), torch.cat(marched)


def _tv64(p, grad, act, bg, w, dense):
    """grad + the TV terms, [R,R,R,C]; p reads bg outside the active voxels."""
    add = torch.zeros_like(p)
    for ax in range(3):
        df = (p.narrow(ax, 1, p.shape[ax] - 1) - p.narrow(ax, 0, p.shape[ax] - 1)).clamp(-1, 1)
        add.narrow(ax, 1, p.shape[ax] - 1).add_(df)
        add.narrow(ax, 0, p.shape[ax] - 1).sub_(df)
    add = add * (_f32(w) / 6)
    return torch.where(act[..., None] if dense else act[..., None] & (grad != 0), grad + add, grad)


def _adam64(p, m, v, g, act, lr, step, mode):
    b0, b1 = _f32(BETAS[0]), _f32(BETAS[1])
    size = _f32(lr) * math.sqrt(1 - b1 ** step) / (1 - b0 ** step)
    if p.shape[-1] > 1 and mode == 1:  # a voxel's channels are skipped by threes
        live = (g.reshape(*g.shape[:-1], -1, 3) != 0).any(-1, keepdim=True).expand(*g.shape[:-1], -1, 3).reshape(g.shape)
    else:
        live = (g != 0) if mode == 1 else torch.ones_like(g, dtype=torch.bool)
    live = live & act[..., None]
    m2 = b0 * m + (1 - b0) * g
    v2 = b1 * v + (1 - b1) * g * g
    p2 = p - size * m2 / (_f32(EPS) + v2.sqrt())
    return torch.where(live, p2, p), torch.where(live, m2, m), torch.where(live, v2, v)


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, seed)


def _leaf_state(names, states, leaves, bg):
    """Updated dense (p, m, v) as the leaf views hold them."""
    p, m, v = (x.reshape(-1, x.shape[-1]) for x in states)
    return {names[0]: _to_leaves(p, leaves, bg), names[1]: _to_leaves(m, leaves, 0.0).reshape(-1),
            names[2]: _to_leaves(v, leaves, 0.0).reshape(-1)}


def _exact_step(c, seed):
    R, n = c["reso"], c["rays"]
    act = _active(c)
    dens, k0 = (x.to(F64) for x in _values(c, seed, act))
    dens = dens[..., None]
    dp, kp = _pad(dens, BACKGROUND).requires_grad_(), _pad(k0, 0.0).requires_grad_()
    net = [t.to(F64).requires_grad_() for t in _rgbnet(seed)]
    loss, _ = _fine64(c, dp, kp, net, _batches(c, seed, 1)[0], None)
    leaves = _leaves(act)
    out = {"loss": loss.reshape(1)}
    tv = TV / n * R / 128
    for names, pad, p, bg, lr, salt in ((("density", "d_avg", "d_avg_sq"), dp, dens, BACKGROUND, LR_DENSITY, 21),
                                        (("k0", "k_avg", "k_avg_sq"), kp, k0, 0.0, LR_K0, 22)):
        g = _unpad(pad.grad, R).reshape(p.shape)
        pad.grad = None
        g = _tv64(p, g, act, bg, tv, False)
        m, v = (x.to(F64) for x in _moments(c, seed, act, p.shape[-1], salt))
        out.update(_leaf_state(names, _adam64(p, m, v, g, act, lr, STEP0 + 1, 1), leaves, bg))
    flat = torch.cat([t.detach().reshape(-1) for t in net])
    g = torch.cat([t.grad.reshape(-1) for t in net])
    m, v = (x.to(F64) for x in _net_moments(seed, flat.numel()))
    one = torch.ones(1, dtype=torch.bool, device="cuda")
    p, m, v = _adam64(flat[:, None], m[:, None], v[:, None], g[:, None], one, LR_NET, 1, 0)
    out.update(params=p[:, 0], exp_avg=m[:, 0], exp_avg_sq=v[:, 0])
    return out


def _exact_staged(c, seed):
    R = c["reso"]
    act = _active(c)
    dens, k0 = _values(c, seed, act)
    dp, kp = _pad(dens[..., None], BACKGROUND).requires_grad_(), _pad(k0, 0.0).requires_grad_()
    net = [t.to(F64).requires_grad_() for t in _rgbnet(seed)]
    loss, rgb = _fine64(c, dp, kp, net, _batches(c, seed, 1)[0], _mask_cache(act))
    leaves = _leaves(act)
    return {"loss": loss, "rgb": rgb, "density": _to_leaves(_unpad(dp.grad, R), leaves, 0.0),
            "k0": _to_leaves(_unpad(kp.grad, R), leaves, 0.0), "net": [t.grad for t in net]}


def _exact_density(c, seed):
    act = _active(c)
    dens, _ = _values(c, seed, act)
    dp = _pad(dens[..., None], BACKGROUND).requires_grad_()
    o, d, _ = _rays(c["rays"], seed, 0)
    target = _rand(_gen(seed, 300), c["rays"]).to(F64)
    total, lasts = 0.0, []
    for s in range(0, c["rays"], 4096):
        _, last, _, _, _ = _composite64(c, dp, o[s:s + 4096].to(F64), d[s:s + 4096].to(F64), None)
        loss = (1 - last - target[s:s + 4096]).pow(2).sum() / c["rays"]
        loss.backward()
        total += float(loss)
        lasts.append(last.detach())
    return {"loss": torch.tensor(total, dtype=F64), "last": torch.cat(lasts),
            "density": _to_leaves(_unpad(dp.grad, c["reso"]), _leaves(act), 0.0)}


def _exact_points(c, seed):
    R = c["reso"]
    act = _active(c)
    dens, k0 = _values(c, seed, act)
    grid = _pad(dens[..., None], BACKGROUND) if c["channels"] == 1 else _pad(k0, 0.0)
    p, g = _sample_points(c, seed, act)
    i, w = _corners(p.to(F64), R)
    grad = torch.zeros_like(grid)
    for q in range(8):
        grad.index_add_(0, i[:, q], g.to(F64) * w[:, q:q + 1])
    return {"out": _trilinear(grid, p.to(F64), R).reshape(-1),
            "grad": _to_leaves(_unpad(grad, R), _leaves(act), 0.0)}


def _exact_render(c, seed):
    R, H, W = c["reso"], c["height"], c["width"]
    act = _active(c)
    dens, k0 = _values(c, seed, act)
    dens = _pad((dens * act)[..., None], 0.0)  # the empty row is zero
    k0 = _pad(k0, 0.0)
    net = [t.to(F64) for t in _rgbnet(seed)]
    K = torch.from_numpy(_intrinsics(c)).to("cuda", F64)
    m = torch.from_numpy(_render_poses(seed)[0]).to("cuda", F64)
    pix = torch.arange(H * W, device="cuda")
    step, thr = _f32(_stepdist(c)), _f32(THRES)
    out = []
    for s in range(0, H * W, 32768):
        q = pix[s:s + 32768]
        x, y = (q % W).to(F64) + 0.5, torch.div(q, W, rounding_mode="floor").to(F64) + 0.5
        d = torch.stack([(x - K[0, 2]) / K[0, 0], -(y - K[1, 2]) / K[1, 1], -torch.ones_like(x)], -1) @ m[:3, :3].T
        norm = d.norm(dim=-1, keepdim=True)
        o, u = (m[:3, 3] + BBOX) / (2 * BBOX), d / (2 * BBOX)
        inv = torch.where(u == 0, torch.full_like(u, 1e-6), u)
        a, b = (1 - o) / inv, -o / inv
        t0 = torch.minimum(a, b).amax(-1).clamp(min=NEAR, max=1e9)
        t1 = torch.maximum(a, b).amin(-1).clamp(min=NEAR, max=1e9)
        n = max(1, int(torch.ceil(((t1 - t0).clamp(min=0) * norm[:, 0] / step).max())) + 1)
        k = torch.arange(n, device="cuda", dtype=F64)
        prev = t0[:, None] + k * (step / norm)
        p = o + u[:, None] * (prev + step / norm)[..., None]
        ok = (prev < t1[:, None]) & ((p >= 0) & (p <= 1)).all(-1)
        idx = p * (R - 1)
        j = torch.round(idx).long().clamp(0, R - 1)
        ok &= act[j[..., 0], j[..., 1], j[..., 2]]
        al = torch.zeros(ok.shape, dtype=F64, device="cuda")
        al[ok] = _alpha(_trilinear(dens, idx[ok], R)[:, 0])
        al = torch.where(al > thr, al, torch.zeros_like(al))
        T = torch.cumprod(1 - al, 1)
        w = torch.cat([torch.ones_like(T[:, :1]), T[:, :-1]], 1) * al
        col = w > thr
        # a ray ends at the first colour sample behind which T is below the limit
        ends = torch.cumsum((col & (T < _f32(T_STOP_RENDER))).long(), 1)
        col &= torch.cat([torch.zeros_like(ends[:, :1]), ends[:, :-1]], 1) == 0
        ray = col.nonzero()[:, 0]
        rgb = _mlp(net, _trilinear(k0, idx[col], R), _pe(d / norm)[ray])
        out.append(torch.zeros(q.shape[0], 3, dtype=F64, device="cuda").index_add(0, ray, w[col][:, None] * rgb))
    return torch.cat(out).reshape(-1)


def _exact_opt(c, seed):
    act = _active(c)
    dens, k0 = (x.to(F64) for x in _values(c, seed, act))
    leaves = _leaves(act)
    out = {}
    for names, p, g, bg, lr, salt in ((("density", "d_avg", "d_avg_sq"), dens[..., None], 0, BACKGROUND, LR_DENSITY, 21),
                                      (("k0", "k_avg", "k_avg_sq"), k0, 1, 0.0, LR_K0, 22)):
        g = _tv64(p, _opt_grads(c, seed)[g].to(F64), act, bg, _opt_tv(c), c["dense_tv"])
        m, v = (x.to(F64) for x in _moments(c, seed, act, p.shape[-1], salt))
        out.update(_leaf_state(names, _adam64(p, m, v, g, act, lr, STEP0 + 1, c["mode"]), leaves, bg))
    return out
