"""Workloads timed for performance work: what a user has this package do.

Each case is a plain dict; ``prepare`` builds what a user's program holds
before the call (inputs on the GPU, the model, optimizer, trainer or server
it keeps), ``run`` makes one pass through the public entry points.  Kinds:

  sample   a training batch's ray samples and their mask lookup, the
           drop-in ops under the reference's own sample_ray
  weights  alpha compositing weights of those samples, forward and
           backward (drop-in ops)
  interp   trilinear lookups of a DenseGrid at the samples of a ray batch
           and the gradient grid they scatter into
  sweep    one optimizer update of a voxel grid: total-variation gradient
           and Adam, with the BF16 shadow of mixed-precision training
  mlp      a colour MLP on the shaded rows of a batch, forward and backward
  train    a fine-stage training step: forward, loss and backward of the
           model, or the trainer's graph-replayed step with its optimizer
  render   views of resident scenes through the render server
  mesh     the SDF field on a dense lattice, as mesh extraction queries it

Sizes follow the benchmark configurations (96^3 to 256^3 grids, 8192 rays a
step, MLPs 128 and 192 wide, 800x600 to 1600x1200 views, 512^3 lattices).
"""
import math

import numpy as np
import torch
import torch.nn as nn
import torch.nn.functional as F

from voxurf_gb300 import configs, grid, mlp, serve, synthetic, train, utils, voxurf_fine
from voxurf_gb300 import render_utils_cuda as ru

DEV = "cuda"
BMIN, BMAX = (-1.0, -1.0, -1.0), (1.0, 1.0, 1.0)
LR, BETAS, EPS, TV = 1e-3, (0.9, 0.99), 1e-8, 1e-4
LATE_LR = 5e-6          # the decayed rate of a late step: the scene stays what it was over many passes
STEP = 4000             # mid-way through the fine schedule: s_val 0.01
ROWS_PER_RAY = 11       # shaded rows a ray has there, for work()
VIEWS = ((600, 800), (480, 640), (1200, 1600), (300, 400))


def listed():
    return [
        # the sampling of one 8192-ray training batch on the fine stage's grid
        dict(name="sample_8192", kind="sample", rays=8192, R=256, stepsize=0.5),
        # its compositing weights: about 400 samples a ray, forward and backward
        dict(name="weights_8192", kind="weights", rays=8192, mean=400),
        # feature lookups of a batch's shaded samples and their gradient grid
        dict(name="interp_k0", kind="interp", points=700_003, R=256, C=12),
        # the smallest call: a few thousand SDF lookups in a coarse grid
        dict(name="interp_small", kind="interp", points=5_003, R=64, C=1),
        # the feature grid's update, the largest sweep of a training step
        dict(name="sweep_k0", kind="sweep", X=256, Y=256, Z=256, C=12, shadow=True, nonzero=0.06),
        # rgbnet of a fine step on the shaded rows of 8192 rays, in both precisions
        dict(name="mlp_fp32", kind="mlp", rows=131_003, d_in=70, width=192, depth=4, bf16=False),
        dict(name="mlp_bf16", kind="mlp", rows=131_003, d_in=70, width=192, depth=4, bf16=True),
        # the coarse rgbnet on a small batch
        dict(name="mlp_coarse_small", kind="mlp", rows=3_001, d_in=75, width=128, depth=3, bf16=True),
        # the fine stage in the default precision, as run.py's loop calls the model
        dict(name="train_fp32", kind="train", R=256, rays=8192, bf16=False, graphed=False),
        # the whole step of the trainer in mixed precision, optimizer included
        dict(name="train_bf16", kind="train", R=256, rays=8192, bf16=True, graphed=True),
        # views of the resident scenes: one request of each resolution
        dict(name="render_views", kind="render", R=256, scenes=2, views=4, scale=1.0, tick=1 << 20),
        # the field of a mesh extraction
        dict(name="mesh_512", kind="mesh", R=256, lattice=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sample", "weights", "interp", "sweep", "mlp", "mlp", "train", "train", "render", "mesh"])
    if kind == "sample":
        return dict(kind=kind, rays=_log_int(rng, 300, 8192), R=rng.randint(64, 256),
                    stepsize=rng.choice([0.5, 1.0]))
    if kind == "weights":
        return dict(kind=kind, rays=_log_int(rng, 300, 8192), mean=_log_int(rng, 40, 400))
    if kind == "interp":
        return dict(kind=kind, points=_log_int(rng, 5_000, 700_000), R=rng.randint(64, 256), C=rng.choice([1, 12]))
    if kind == "sweep":
        C = rng.choice([1, 12])
        return dict(kind=kind, X=rng.randint(64, 256), Y=rng.randint(64, 256), Z=rng.randint(64, 256), C=C,
                    shadow=bool(C > 1 and rng.random() < 0.5), nonzero=round(rng.uniform(0.01, 0.2), 3))
    if kind == "mlp":
        return dict(kind=kind, rows=_log_int(rng, 3_000, 131_000), d_in=rng.randint(60, 75),
                    width=rng.choice([128, 192]), depth=rng.choice([3, 4]), bf16=bool(rng.random() < 0.5))
    if kind == "train":
        return dict(kind=kind, R=rng.randint(96, 224), rays=_log_int(rng, 1024, 8192), bf16=bool(rng.random() < 0.5),
                    graphed=bool(rng.random() < 0.5))
    if kind == "render":
        return dict(kind=kind, R=rng.randint(128, 224), scenes=rng.randint(1, 2), views=rng.randint(1, 4),
                    scale=round(rng.uniform(0.25, 1.0), 2), tick=1 << rng.randint(17, 20))
    return dict(kind="mesh", R=rng.randint(96, 256), lattice=_log_int(rng, 100, 500))


# ---- inputs -------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rays(n, seed):
    """n pixels of the 49 cameras that synthetic.fibonacci_poses places."""
    return tuple(torch.from_numpy(a).to(DEV) for a in synthetic.random_rays(n, seed=seed % (1 << 30)))


def _scene_sdf(shape, seed, radii=(0.45, 0.6, 0.15)):
    """SDF of a sphere inside a torus with the noise of an optimized grid."""
    ax = [torch.linspace(-1, 1, s, device=DEV) for s in shape]
    x, y, z = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    rho = x * x + y * y
    s = (rho + z * z).sqrt() - radii[0]
    t = ((rho.sqrt() - radii[1]) ** 2 + z * z).sqrt() - radii[2]
    s = torch.minimum(s, t)
    return s + 0.005 * torch.randn(s.shape, generator=_gen(seed), device=DEV)


def _model(R, bf16, seed, radii=(0.45, 0.6, 0.15)):
    """The fine model of the benchmark configuration with a scene loaded and
    the mask of the voxels within 6.4 voxels of its surface."""
    kw = configs.fine_model_kwargs(R, "bf16" if bf16 else "fp32")
    torch.manual_seed(seed)
    m = voxurf_fine.Voxurf(**kw).to(DEV)
    sdf = _scene_sdf(m.sdf.grid.shape[2:], seed, radii)
    with torch.no_grad():
        m.sdf.grid.copy_(sdf[None, None])
        m.k0.grid.copy_(0.1 * torch.randn(m.k0.grid.shape, generator=_gen(seed + 1), device=DEV))
        mask = sdf.abs() < 6.4 * 2.0 / R
        m.mask_cache = grid.MaskGrid(mask=mask, xyz_min=BMIN, xyz_max=BMAX).to(DEV)
        m.nonempty_mask = mask[None, None]
        m.density[~mask[None, None]] = -100
        m.sdf.grid[~mask[None, None]] = 1
    if bf16:
        m.refresh_k0_shadow()
    return m


def _segments(rays, mean, seed):
    """Ragged per-ray segments of alphas: a faint halo and one surface.  The
    lengths are the same ones for every seed, in another order."""
    g = _gen(seed)
    n = torch.randint(mean // 4, 2 * mean - mean // 4, (rays,), generator=_gen(rays), device=DEV)
    n = n[torch.randperm(rays, generator=g, device=DEV)]
    ray_id = torch.repeat_interleave(torch.arange(rays, device=DEV), n)
    off = torch.cumsum(n, 0) - n
    pos = torch.arange(ray_id.numel(), device=DEV) - off[ray_id]
    at = (torch.rand(rays, generator=g, device=DEV) * 1.3 * n)[ray_id]
    peak = (0.6 * torch.rand(rays, generator=g, device=DEV))[ray_id]
    alpha = peak * torch.exp(-((pos - at) / 6.0) ** 2) + 1e-3 * torch.rand(ray_id.numel(), generator=g, device=DEV)
    return alpha.clamp(0, 0.999).contiguous(), ray_id.contiguous(), n, off


def _points(n, R, seed):
    """Runs of 32 consecutive half-voxel samples along random directions."""
    g = _gen(seed)
    runs = -(-n // 32)
    o = 1.6 * torch.rand((runs, 1, 3), generator=g, device=DEV) - 0.8
    d = F.normalize(torch.randn((runs, 1, 3), generator=g, device=DEV), dim=-1)
    t = torch.arange(32, device=DEV, dtype=torch.float32)[None, :, None] * (1.0 / R)
    return (o + d * t).reshape(-1, 3)[:n].clamp(-1, 1).contiguous()


def _net(case, seed):
    torch.manual_seed(seed)
    W = case["width"]
    layers = [nn.Linear(case["d_in"], W), nn.ReLU(inplace=True)]
    for _ in range(case["depth"] - 2):
        layers.append(nn.Sequential(nn.Linear(W, W), nn.ReLU(inplace=True)))
    return nn.Sequential(*layers, nn.Linear(W, 3)).to(DEV)


def _mlp_rows(case, seed):
    """Feature rows (features and encodings within [-1, 1], zero padding) and
    the gradient of a mean-squared loss at the logits."""
    dt = torch.bfloat16 if case["bf16"] else torch.float32
    ld = mlp.row_stride(case["d_in"], dt)
    n, g = case["rows"], _gen(seed)
    x = torch.zeros((n, ld), dtype=dt, device=DEV)
    x[:, :case["d_in"]] = torch.sin(3.0 * torch.randn((n, case["d_in"]), generator=g, device=DEV)).to(dt)
    dy = torch.randn((n, 3), generator=g, device=DEV) / n
    return x, dy


# ---- prepare ------------------------------------------------------------------
def prepare(case, seed):
    k = case["kind"]
    s = {"case": case}
    if k == "sample":
        R = case["R"]
        # one set of pixels in another order: as many samples for every seed
        o, d, _ = (t[torch.randperm(case["rays"], generator=_gen(seed), device=DEV)].contiguous()
                   for t in _rays(case["rays"], 0))
        mask = grid.MaskGrid(mask=_scene_sdf((R, R, R), seed).abs() < 0.05, xyz_min=BMIN, xyz_max=BMAX).to(DEV)
        s.update(o=o, d=d, mask=mask, bmin=torch.tensor(BMIN, device=DEV), bmax=torch.tensor(BMAX, device=DEV),
                 stepdist=case["stepsize"] * 2.0 / R)
    elif k == "weights":
        alpha, ray_id, _, _ = _segments(case["rays"], case["mean"], seed)
        g = _gen(seed + 1)
        s.update(alpha=alpha, ray_id=ray_id, gw=torch.randn(alpha.shape, generator=g, device=DEV),
                 gl=torch.randn(case["rays"], generator=g, device=DEV))
    elif k == "interp":
        g = _gen(seed)
        net = grid.DenseGrid(case["C"], [case["R"]] * 3, BMIN, BMAX).to(DEV)
        with torch.no_grad():
            net.grid.copy_(0.1 * torch.randn(net.grid.shape, generator=g, device=DEV))
        out = (case["points"], case["C"]) if case["C"] > 1 else (case["points"],)
        s.update(net=net, pts=_points(case["points"], case["R"], seed + 1),
                 gout=torch.randn(out, generator=g, device=DEV))
    elif k == "sweep":
        p, g, shadow = _sweep_inputs(case, seed)
        p = nn.Parameter(p)
        opt = utils.Adam([dict(params=[p], lr=LR, name="k0", tv_weight=_tv_weight(case), tv_dense=True,
                               shadow=shadow)], betas=BETAS)
        s.update(p=p, g=g, opt=opt, shadow=shadow)
    elif k == "mlp":
        x, dy = _mlp_rows(case, seed + 1)
        s.update(net=_net(case, seed), x=x.requires_grad_(), dy=dy)
    elif k == "train":
        m = _model(case["R"], case["bf16"], seed)
        o, d, v = _rays(case["rays"], seed + 2)
        s.update(model=m, batch=(o, d, v),
                 target=torch.rand((case["rays"], 3), generator=_gen(seed + 3), device=DEV),
                 rk=dict(configs.FINE_RENDER_KWARGS))
        if case["graphed"]:
            s["trainer"] = train.FineTrainer(m, lr_sdf=LATE_LR, lr_k0=LATE_LR, lr_rgbnet=LATE_LR, lr_k_rgbnet=LATE_LR,
                                             n_rays=case["rays"], graphed=True)
    elif k == "render":
        scenes = [serve.ResidentScene(_model(case["R"], True, seed + i, configs.SERVE_SHAPES[i]),
                                      s_val=configs.trained_s_val()) for i in range(case["scenes"])]
        sizes = _view_sizes(case)
        srv = serve.RenderServer(scenes, tick_rays=case["tick"], arena_pixels=sum(h * w for h, w in sizes))
        poses = synthetic.fibonacci_poses(49)
        rng = np.random.default_rng(seed)
        s.update(server=srv, views=[(i % case["scenes"], poses[rng.integers(49)], h, w)
                                    for i, (h, w) in enumerate(sizes)])
    else:
        R = case["R"]
        s.update(sdf=_scene_sdf((R, R, R), seed).contiguous(), taps=_taps(),
                 bmin=torch.tensor(BMIN, device=DEV), bmax=torch.tensor(BMAX, device=DEV))
    return s


def _sweep_inputs(case, seed):
    shape = (1, case["C"], case["X"], case["Y"], case["Z"])
    fmt = torch.channels_last_3d if case["C"] > 1 else torch.contiguous_format
    gen = _gen(seed)
    p = torch.empty(shape, device=DEV).contiguous(memory_format=fmt).normal_(0, 0.1, generator=gen)
    # the gradient is zero at the voxels no ray of the batch came by
    hit = torch.rand((1, 1) + shape[2:], generator=gen, device=DEV) < case["nonzero"]
    g = torch.empty(shape, device=DEV).contiguous(memory_format=fmt).normal_(0, 1e-6, generator=gen).mul_(hit)
    shadow = p.to(torch.bfloat16).contiguous(memory_format=fmt) if case["shadow"] else None
    return p, g, shadow


def _taps():
    """The fine stage's smoothing kernel along one axis (5 wide, sigma 0.8)."""
    g = np.exp(-np.arange(-2, 3) ** 2 / (2 * 0.8 ** 2))
    return (g / g.sum()).astype(np.float32)


def _tv_weight(case):
    return TV / 8192 * max(case["X"], case["Y"], case["Z"]) / 128


def _view_sizes(case):
    return [tuple(max(8, int(v * case["scale"])) for v in VIEWS[i]) for i in range(case["views"])]


# ---- run ----------------------------------------------------------------------
def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "sample":
        out = ru.sample_pts_on_rays(s["o"], s["d"], s["bmin"], s["bmax"], 0.1, 1e9, s["stepdist"])
        return [*out, s["mask"](out[0])]
    if k == "weights":
        w, T, last, i0, i1 = ru.alpha2weight(s["alpha"], s["ray_id"], case["rays"])
        g = ru.alpha2weight_backward(s["alpha"], w, T, last, i0, i1, case["rays"], s["gw"], s["gl"])
        return [w, T, last, i0, i1, g]
    if k == "interp":
        s["net"].grid.grad = None
        out = s["net"](s["pts"])
        out.backward(s["gout"])
        return [out.detach(), s["net"].grid.grad]
    if k == "sweep":
        s["p"].grad = s["g"]
        s["opt"].step(zero_grad=True)
        st = s["opt"].state[s["p"]]
        out = [s["p"].detach(), st["exp_avg"], st["exp_avg_sq"]]
        return out + [s["shadow"]] if case["shadow"] else out
    if k == "mlp":
        ps = list(s["net"].parameters())
        y = mlp.apply_mlp(s["net"], s["x"])
        grads = torch.autograd.grad(y, [s["x"], *ps], s["dy"])
        return [y.detach(), *grads]
    if k == "train":
        m = s["model"]
        if case["graphed"]:
            loss, _ = s["trainer"].step(*s["batch"], s["target"], s["rk"], global_step=STEP)
            st = s["trainer"].optimizer.state
            return [loss, [p.detach() for p in _trained(m)],
                    [st[p]["exp_avg"] for p in _trained(m)]]
        for p in m.parameters():
            p.grad = None
        ret = m(*s["batch"], global_step=STEP, **s["rk"])
        loss = train.fine_loss(ret, s["target"])
        loss.backward()
        return [loss.detach(), ret["rgb_marched"].detach(), ret["rgb_marched0"].detach(),
                ret["alphainv_cum"].detach(), [p.grad for p in _trained(m)]]
    if k == "render":
        srv = s["server"]
        reqs = [srv.submit(scene, pose, h, w) for scene, pose, h, w in s["views"]]
        srv.run_until_idle()
        srv.done.clear()
        return [a for r in reqs for a in (r.rgb, r.depth)]
    sm = voxurf_fine.smooth_grid(s["sdf"], s["taps"])
    return voxurf_fine.extract_fields(sm, s["bmin"], s["bmax"], BMIN, BMAX, case["lattice"])


def _trained(m):
    return [m.sdf.grid, m.k0.grid, *m.rgbnet.parameters(), *m.k_rgbnet.parameters()]


# ---- work ---------------------------------------------------------------------
def _mlp_flops(d_in, W, depth):
    return 2 * (d_in * W + (depth - 2) * W * W + 3 * W)


def work(case):
    k = case["kind"]
    if k == "sample":
        # about 0.8 box widths a ray: points, flag, two ids; then a mask byte and a flag
        n = case["rays"] * case["R"] * 1.6 / case["stepsize"] / 2
        return {"bytes": n * (12 + 1 + 16 + 1 + 1) + case["rays"] * 40, "flops": n * 20}
    if k == "weights":
        n = case["rays"] * case["mean"]
        return {"bytes": n * (12 + 8 + 8) + case["rays"] * 28, "flops": n * 8}
    if k == "interp":
        vox = case["R"] ** 3
        n, C = case["points"], case["C"]
        return {"bytes": 4 * (n * 3 + 2 * n * C + min(8 * n, vox) * C + vox * C), "flops": n * C * 32}
    if k == "sweep":
        n = case["X"] * case["Y"] * case["Z"] * case["C"]
        return {"bytes": n * (28 + 2 * case["shadow"]), "flops": n * 35}
    if k == "mlp":
        b = 2 if case["bf16"] else 4
        f = _mlp_flops(case["d_in"], case["width"], case["depth"]) * case["rows"]
        return {"bytes": case["rows"] * (2 * b * case["d_in"] + 24), "flops": 3 * f}
    if k == "train":
        vox, rows = case["R"] ** 3, case["rays"] * ROWS_PER_RAY * case["R"] / 256
        f = 3 * rows * (_mlp_flops(70, 192, 4) + _mlp_flops(60, 192, 4))
        if case["graphed"]:
            return {"bytes": vox * (13 * 24 + 24 * case["bf16"]), "flops": f}
        return {"bytes": vox * (4 + 13 * 4), "flops": f}
    if k == "render":
        n = sum(h * w for h, w in _view_sizes(case))
        return {"bytes": n * 16, "flops": n * 5 * (_mlp_flops(70, 192, 4) + _mlp_flops(60, 192, 4))}
    n = case["lattice"] ** 3
    return {"bytes": 4 * n + 4 * case["R"] ** 3, "flops": n * 24}


# ---- the same outputs in 64 bits ------------------------------------------------
def exact(case, seed):
    """What run() returns, from plain torch in 64 bits.  None for `sample`
    (its points are defined by their 32-bit rounding), `train` and `render`
    (which samples count is decided by 32-bit thresholds on the way)."""
    k = case["kind"]
    if k == "weights":
        return _exact_weights(case, seed)
    if k == "interp":
        return _exact_interp(case, seed)
    if k == "sweep":
        return _exact_sweep(case, seed)
    if k == "mlp":
        return _exact_mlp(case, seed)
    if k == "mesh":
        return _exact_mesh(case, seed)
    return None


def _exact_weights(case, seed):
    alpha, ray_id, n, off = _segments(case["rays"], case["mean"], seed)
    g = _gen(seed + 1)
    gw = torch.randn(alpha.shape, generator=g, device=DEV).double()
    gl = torch.randn(case["rays"], generator=g, device=DEV).double()
    rays, L = case["rays"], int(n.max())
    col = torch.arange(alpha.numel(), device=DEV) - off[ray_id]
    a = torch.zeros((rays, L), dtype=torch.float64, device=DEV)
    a[ray_id, col] = alpha.double()
    inside = torch.arange(L, device=DEV)[None] < n[:, None]
    T1 = torch.cumprod(1 - a, 1)                            # after the sample
    T0 = torch.cat([torch.ones_like(T1[:, :1]), T1[:, :-1]], 1)
    below = (T1 < 1e-3) & inside                            # the march ends at the first such sample
    end = torch.where(below.any(1), below.to(torch.int8).argmax(1) + 1, n)
    live = torch.arange(L, device=DEV)[None] < end[:, None]
    w = torch.where(live, T0 * a, torch.zeros_like(a))
    last = T1.gather(1, (end - 1)[:, None])[:, 0]
    G = torch.zeros_like(a)
    G[ray_id, col] = gw
    tail = torch.flip(torch.cumsum(torch.flip(torch.where(live, G * w, torch.zeros_like(a)), [1]), 1), [1])
    after = torch.cat([tail[:, 1:], torch.zeros_like(tail[:, :1])], 1) + (gl * last)[:, None]
    # dw_i/da_i = T_i; every later weight and the last transmittance carry 1 / (1 - a_i)
    grad = torch.where(live, G * T0 - after / (1 - a), torch.zeros_like(a))
    T = torch.where(live, T0, torch.ones_like(a))
    return [w[ray_id, col], T[ray_id, col], last, None, None, grad[ray_id, col]]


def _grid_sample(vol, pts):
    """Trilinear lookups with aligned corners, the bbox [-1, 1]^3 (x the
    slowest axis, which grid_sample calls depth)."""
    q = pts.flip(-1).reshape(1, 1, 1, -1, 3)
    return F.grid_sample(vol, q, mode="bilinear", align_corners=True)[0, :, 0, 0].t()


def _exact_interp(case, seed):
    g = _gen(seed)
    C, n = case["C"], case["points"]
    like = torch.empty([1, C] + [case["R"]] * 3, device=DEV)
    if C > 1:
        like = like.contiguous(memory_format=torch.channels_last_3d)
    vol = (0.1 * torch.randn(like.shape, generator=g, device=DEV)).double().requires_grad_()
    gout = torch.randn((n, C) if C > 1 else (n,), generator=g, device=DEV).double()
    out = _grid_sample(vol, _points(n, case["R"], seed + 1).double())
    out = out if C > 1 else out[:, 0]
    out.backward(gout)
    grad = torch.empty_like(like, dtype=torch.float64).copy_(vol.grad)
    return [out.detach(), grad]


def _exact_sweep(case, seed):
    p32, g32, _ = _sweep_inputs(case, seed)
    p, w = p32.double(), _tv_weight(case) / 6
    grad = g32.double()
    for ax in (2, 3, 4):
        n = p.shape[ax]
        d = (p.narrow(ax, 1, n - 1) - p.narrow(ax, 0, n - 1)).clamp_(-1, 1).mul_(w)
        grad.narrow(ax, 1, n - 1).add_(d)
        grad.narrow(ax, 0, n - 1).sub_(d)
    del d
    m = grad * (1 - BETAS[0])
    v = grad.square_().mul_(1 - BETAS[1])
    p -= LR / (1 - BETAS[0]) * m / (v.sqrt() / math.sqrt(1 - BETAS[1]) + EPS)
    return [p, m, v] + ([p] if case["shadow"] else [])


def _exact_mlp(case, seed):
    net = _net(case, seed).double()
    x, dy = _mlp_rows(case, seed + 1)
    x = x.double().requires_grad_()
    y = net(x[:, :case["d_in"]])
    grads = torch.autograd.grad(y, [x, *net.parameters()], dy.double())
    return [y.detach(), *grads]


def _exact_mesh(case, seed):
    R, n = case["R"], case["lattice"]
    vol = _scene_sdf((R, R, R), seed).double()
    taps = [float(t) for t in _taps()]
    for ax in range(3):     # the grid's border values continue outside
        at = torch.arange(R, device=DEV)
        vol = sum(t * vol.index_select(ax, (at + i - 2).clamp(0, R - 1)) for i, t in enumerate(taps))
    axis = torch.linspace(-1, 1, n, device=DEV).double()
    out = torch.empty((n, n, n), dtype=torch.float64, device=DEV)
    yz = torch.stack(torch.meshgrid(axis, axis, indexing="ij"), -1).reshape(-1, 2)
    for i in range(n):
        pts = torch.cat([axis[i].expand(n * n, 1), yz], 1)
        out[i] = -_grid_sample(vol[None, None], pts).reshape(n, n)
    return out
