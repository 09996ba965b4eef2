"""Workloads of the Universal Beta Splatting rasteriser, each through the entry
points a program calls: training steps (eager, captured, batched over views,
with the full loss and Adam), serving requests, the drop-in operators, feature
rasterisation, the training loss, MCMC densification and viewer frames.

    listed()             the named workloads
    draw(rng)            another workload of the same ranges
    prepare(case, seed)  inputs and handles on the GPU
    run(state)           one pass; returns its outputs
    work(case)           bytes and operations one pass cannot do without
    exact(case, seed)    the outputs in 64 bits, in plain torch

Scenes, cameras and images are seeded and synthetic, with the parameter
distributions of the benchmark (bench.py)."""
import math
import os
import sys
import types

import numpy as np
import torch
import torch.nn.functional as F

sys.path.insert(0, os.path.join(os.getcwd(), "universal-beta-splatting_gb300"))

NAMES = ("xyz", "mean", "scale", "l_triangle", "opacity", "beta", "rgb")
# the training configuration's learning rates
LRS = {"xyz": 1.6e-4, "mean": 2e-3, "rgb": 2.5e-3, "opacity": 5e-2, "beta": 5e-3, "scale": 5e-3,
       "l_triangle": 1e-3}
EPS2D, ADAM_T = 0.3, 1000


def listed():
    return [
        # the headline training step: 1M primitives at 1080p, captured once
        # into a CUDA graph and replayed (a fixed view, e.g. a benchmark loop)
        dict(name="train_graph_1080p", kind="train", graph=True, n=1_000_000, dim=6, tile=16,
             views="1920x1080"),
        # the smallest configuration: 10k primitives at 256x256, kernel by
        # kernel, where launches and host work count
        dict(name="train_small_256", kind="train", graph=False, n=10_000, dim=6, tile=16,
             views="256x256"),
        # a dynamic (7-D) scene, 8 timestamped views in one step
        dict(name="train_7d_8views", kind="train", graph=False, n=500_000, dim=7, tile=16,
             views="1352x1014*8"),
        # the largest: 3M primitives, 4 views of mixed resolution in one step
        dict(name="train_3m_mixed", kind="train", graph=False, n=3_000_000, dim=6, tile=16,
             views="1920x1080,1600x1064,1280x720,960x540"),
        # one iteration of a training loop: render, L1 + SSIM loss, backward
        # and Adam over the seven groups; an odd image size
        dict(name="iterate_979x547", kind="iterate", n=300_007, dim=6, tile=16, views="979x547"),
        # a serving request: a camera not seen before, forward only
        dict(name="request_720p", kind="request", n=500_000, dim=6, tile=16, views="1280x720"),
        # the reference model's own call sequence through the drop-in
        # operators, forward and backward
        dict(name="dropin_train_1064", kind="dropin", n=300_000, dim=6, tile=16, mode="RGB",
             grad=True, views="1600x1064"),
        # the same forward only with depth, as in evaluation (7-D scene)
        dict(name="dropin_depth_640", kind="dropin", n=100_000, dim=7, tile=16, mode="RGB+D",
             grad=False, views="640x480"),
        # 16 feature channels per primitive instead of colours
        dict(name="features_16", kind="features", n=40_000, channels=16, tile=16,
             views="640x480"),
        # the training loss alone on a 1080p image, channels first
        dict(name="loss_1080p", kind="loss", views="1920x1080"),
        # densification: relocate 10% dead, add 2%, position noise
        dict(name="mcmc_1m", kind="mcmc", n=1_000_000, dim=6),
        # an interactive viewer frame with Beta quantile ranges, to the host
        dict(name="viewer_1080p", kind="viewer", n=1_000_000, dim=6, tile=16, views="1920x1080"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def size(lo, hi):
        w = log(lo, hi)
        return w, max(48, int(w * rng.uniform(0.5, 0.85)))

    kind = rng.choice(["train", "train", "train", "iterate", "request", "request", "dropin",
                       "dropin", "features", "loss", "mcmc", "viewer"])
    dim, tile = rng.choice([6, 6, 7]), rng.choice([16, 16, 16, 8, 32])
    if kind == "train":
        c = rng.choice([1, 1, 1, 2, 3, 5, 8])
        n = log(5_000, min(2_000_000, 4_000_000 // c))
        views = ",".join("%dx%d" % size(96, 1920 if c < 3 else 1200) for _ in range(c))
        return dict(kind=kind, graph=rng.random() < 0.4, n=n, dim=dim, tile=tile, views=views)
    if kind == "loss":
        return dict(kind=kind, views="%dx%d" % size(64, 2400))
    if kind == "mcmc":
        return dict(kind=kind, n=log(5_000, 2_000_000), dim=dim)
    views = "%dx%d" % size(96, 1920)
    if kind == "features":
        return dict(kind=kind, n=log(2_000, 100_000), channels=rng.choice([1, 3, 4, 5, 8, 13, 16, 32]),
                    tile=16, views="%dx%d" % size(96, 900))
    n = log(5_000, 1_500_000 if kind != "dropin" else 700_000)
    case = dict(kind=kind, n=n, dim=dim, tile=tile, views=views)
    if kind == "dropin":
        case.update(mode=rng.choice(["RGB", "RGB+D"]), grad=rng.random() < 0.6)
    return case


# ------------------------------------------------------------------- inputs
def _gen(seed, what):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + what)


def _sizes(case):
    out = []
    for v in case["views"].split(","):
        wh, _, k = v.partition("*")
        w, h = wh.split("x")
        out += [(int(w), int(h))] * int(k or 1)
    return out


def _small(case):
    """Scenes of the smallest configuration fill [-1, 1]^3 seen from 3 units,
    the others [-2, 2]^3 from 4."""
    return case["n"] <= 50_000


def _scene(case, seed):
    """Raw parameters: spatial scales exp(N(-4, 0.5)) through the inverse
    softplus, angular scales about 1, small skews and lower triangles,
    opacity logits N(0, 1), uniform colours."""
    n, dim, g = case["n"], case["dim"], _gen(seed, 1)
    k, r = dim - 3, 1.0 if _small(case) else 2.0

    def rnd(*s):
        return torch.randn(*s, generator=g, device="cuda")

    def uni(*s):
        return torch.rand(*s, generator=g, device="cuda")

    mean = uni(n, k) * 2 - 1
    if dim == 7:
        mean[:, 3] = uni(n)
    s = torch.cat([torch.exp(rnd(n, 3) * 0.5 - 4.0), 1.0 + 1e-5 * rnd(n, k)], 1)
    return {"xyz": (uni(n, 3) * 2 - 1) * r, "mean": mean, "scale": s + torch.log(-torch.expm1(-s)),
            "l_triangle": rnd(n, dim * (dim - 1) // 2) * 0.1, "opacity": rnd(n, 1),
            "beta": torch.cat([rnd(n, 1) * 0.3, rnd(n, k) * 0.5], 1), "rgb": uni(n, 3)}


def _cameras(case, seed):
    """(viewmat [4, 4], K [3, 3], width, height, timestamp) per view, on the
    host: an orbit looking at the origin."""
    rng = np.random.RandomState(int(seed) % (1 << 31))
    out = []
    for w, h in _sizes(case):
        eye = rng.standard_normal(3)
        eye *= (3.0 if _small(case) else 4.0) / np.linalg.norm(eye)
        f = -eye / np.linalg.norm(eye)
        r = np.cross(f, [0.0, 1.0, 0.0])
        r /= np.linalg.norm(r)
        vm = np.eye(4)
        vm[:3, :3] = np.stack([r, -np.cross(r, f), f])
        vm[:3, 3] = -vm[:3, :3] @ eye
        fx = (300.0 / 256 if _small(case) else 1500.0 / 1920) * w
        K = np.array([[fx, 0, w / 2], [0, fx, h / 2], [0, 0, 1]])
        out.append((torch.tensor(vm, dtype=torch.float32), torch.tensor(K, dtype=torch.float32), w, h,
                    float(np.float32(rng.uniform()))))
    return out


def _images(case, seed):
    return torch.rand(sum(w * h for w, h in _sizes(case)), 3, generator=_gen(seed, 2), device="cuda")


def _background(case, seed):
    return torch.rand(len(_sizes(case)), 3, generator=_gen(seed, 3), device="cuda")


def _projected(case, seed):
    """Projected primitives of the feature case, as a projection leaves them."""
    n, g = case["n"], _gen(seed, 4)
    (w, h), = _sizes(case)

    def uni(*s):
        return torch.rand(*s, generator=g, device="cuda")

    a, b = (torch.exp(torch.randn(1, n, generator=g, device="cuda") * 0.6) * 3.0 for _ in range(2))
    t = uni(1, n) * math.pi
    c, s = torch.cos(t), torch.sin(t)
    xx, xy, yy = a * a * c * c + b * b * s * s, (a * a - b * b) * c * s, a * a * s * s + b * b * c * c
    det = xx * yy - xy * xy
    return {"means2d": torch.stack([uni(1, n) * (w + 20) - 10, uni(1, n) * (h + 20) - 10], -1),
            "conics": torch.stack([yy / det, -xy / det, xx / det], -1),
            "colors": uni(1, n, case["channels"]), "opacities": uni(1, n) * 0.8 + 0.05,
            "betas": torch.exp(torch.randn(1, n, generator=g, device="cuda") * 0.5) * 1.5,
            "radii": torch.ceil(torch.maximum(a, b)).to(torch.int32) + 1, "depths": uni(1, n) * 8 + 0.5}


def _model(case, seed):
    """A mid-training model: parameters with Adam moments, as the reference's
    BetaModel keeps them."""
    from ubs.optim import FusedAdam
    p, g = _scene(case, seed), _gen(seed, 5)
    m = types.SimpleNamespace(params={k: torch.nn.Parameter(v) for k, v in p.items()})
    for k, v in m.params.items():
        setattr(m, "_" + k, v)
    m.optimizer = FusedAdam([{"params": [m.params[k]], "lr": LRS[k], "name": k} for k in NAMES],
                            lr=0.0, eps=1e-15)
    for k in NAMES:
        st, shape = m.optimizer.state[m.params[k]], m.params[k].shape
        st["step"] = float(ADAM_T)
        st["exp_avg"] = torch.randn(shape, generator=g, device="cuda") * 1e-7
        st["exp_avg_sq"] = torch.rand(shape, generator=g, device="cuda") * 1e-13 + 1e-14
    return m


def prepare(case, seed):
    from ubs import scene as S
    kind = case["kind"]
    st = types.SimpleNamespace(case=case)
    if kind in ("train", "iterate", "request", "dropin"):
        on = "cpu" if kind == "request" else "cuda"
        st.cams = [S.Camera(vm.to(on), K.to(on), w, h, t) for vm, K, w, h, t in _cameras(case, seed)]
    if kind in ("train", "iterate", "request"):
        from ubs.render import GraphedStep, Renderer, Views
        st.r = Renderer(dim=case["dim"], tile_size=case["tile"])
        st.bg = _background(case, seed)
        if kind != "request":
            st.views = Views(st.cams, tile_size=case["tile"], device="cuda")
            st.target = _images(case, seed)
    if kind == "train":
        from ubs.loss import l1_loss
        st.p = {k: torch.nn.Parameter(v) for k, v in _scene(case, seed).items()}
        st.loss = lambda colors, alphas: l1_loss(colors, st.target)
        if case["graph"]:
            st.step = GraphedStep(st.r, st.p, st.views, st.bg, st.loss)
    elif kind == "iterate":
        st.m = _model(case, seed)
    elif kind == "request":
        st.p = _scene(case, seed)
    elif kind == "dropin":
        st.p = {k: v.requires_grad_(case["grad"]) for k, v in _scene(case, seed).items()}
        st.rest = S.rest_indices(case["dim"], "cuda")
        st.bg = _background(case, seed)[0]
        w, h = _sizes(case)[0]
        st.target = _images(case, seed).view(h, w, 3).permute(2, 0, 1).contiguous()
    elif kind == "features":
        st.p = _projected(case, seed)
        for k in ("means2d", "conics", "colors", "opacities", "betas"):
            st.p[k].requires_grad_(True)
        (w, h), = _sizes(case)
        st.v = torch.randn(1, h, w, case["channels"], generator=_gen(seed, 6), device="cuda")
    elif kind == "loss":
        st.img, st.gt = _loss_images(case, seed)
        st.img.requires_grad_(True)
    elif kind == "mcmc":
        st.m = _model(case, seed)
        st.dead = torch.rand(case["n"], generator=_gen(seed, 7), device="cuda") < 0.1
        st.g = torch.Generator().manual_seed(int(seed))
    elif kind == "viewer":
        from ubs.viewer import FrameRenderer, ViewState
        st.p = _scene(case, seed)
        st.frames = FrameRenderer(dim=case["dim"], tile_size=case["tile"])
        st.state = ViewState(b_xyz=(5, 95), b_view=(5, 95), timestamp=_cameras(case, seed)[0][4],
                             backgrounds=(255.0, 255.0, 255.0))
        vm, K, w, h, _ = _cameras(case, seed)[0]
        st.cam = (torch.linalg.inv(vm.double()).float().numpy(), K.numpy(), w, h)
    return st


def _loss_images(case, seed):
    (w, h), = _sizes(case)
    g = _gen(seed, 8)
    gt = torch.rand(1, 3, h, w, generator=g, device="cuda")
    img = (gt + 0.2 * torch.randn(1, 3, h, w, generator=g, device="cuda")).clamp(0, 1)
    return img, gt


# --------------------------------------------------------------------- passes
def run(st):
    kind = st.case["kind"]
    if kind == "train":
        if st.case["graph"]:
            loss = st.step.replay()
        else:
            for v in st.p.values():
                v.grad = None
            loss = st.loss(*st.r.render(st.p, st.views, st.bg))
            loss.backward()
        return {"loss": loss.detach(), "grads": {k: v.grad for k, v in st.p.items()}}
    if kind == "iterate":
        from ubs.loss import l1_ssim_loss
        st.m.optimizer.zero_grad(set_to_none=True)
        colors, _ = st.r.render(st.m.params, st.views, st.bg, check=False)
        (w, h), = _sizes(st.case)
        loss = l1_ssim_loss(colors.view(h, w, 3), st.target.view(h, w, 3), channels_last=True)
        loss.backward()
        grads = {k: v.grad for k, v in st.m.params.items()}
        st.m.optimizer.step()
        return {"loss": loss.detach(), "image": colors.detach(), "grads": grads,
                "params": dict(st.m.params),
                "m": {k: st.m.optimizer.state[v]["exp_avg"] for k, v in st.m.params.items()}}
    if kind == "request":
        from ubs.render import Views
        with torch.no_grad():
            colors, alphas = st.r.render(st.p, Views(st.cams, tile_size=st.case["tile"],
                                                     device="cuda"), st.bg)
        return {"image": colors, "alpha": alphas}
    if kind == "dropin":
        return _run_dropin(st)
    if kind == "features":
        return _run_features(st)
    if kind == "loss":
        from ubs.loss import l1_ssim_loss
        st.img.grad = None
        loss = l1_ssim_loss(st.img, st.gt)
        loss.backward()
        return {"loss": loss.detach(), "grad": st.img.grad}
    if kind == "mcmc":
        return _run_mcmc(st)
    c2w, K, w, h = st.cam
    return {"image": st.frames.render(st.p, c2w, K, w, h, st.state)}


def _run_dropin(st):
    from ubs.scene import render_view
    for v in st.p.values():
        v.grad = None
    with torch.set_grad_enabled(st.case["grad"]):
        img, alphas, meta = render_view(st.p, st.cams[0], st.bg, *st.rest,
                                        render_mode=st.case["mode"], tile_size=st.case["tile"])
        out = {"image": img.detach(), "alpha": alphas.detach(), "radii": meta["radii"],
               "tiles": meta["tiles_per_gauss"], "offsets": meta["isect_offsets"]}
        if st.case["grad"]:
            loss = (img[:3] - st.target).abs().mean()
            loss.backward()
            out.update(loss=loss.detach(), grads={k: v.grad for k, v in st.p.items()})
    return out


def _run_features(st):
    from gsplat.cuda._wrapper import isect_offset_encode, isect_tiles, rasterize_to_pixels
    p, ts = st.p, st.case["tile"]
    (w, h), = _sizes(st.case)
    tw, th = -(-w // ts), -(-h // ts)
    leaves = [p[k] for k in ("means2d", "conics", "colors", "opacities", "betas")]
    for v in leaves:
        v.grad = None
    tiles, ids, order = isect_tiles(p["means2d"].detach(), p["radii"], p["depths"], ts, tw, th)
    offsets = isect_offset_encode(ids, 1, tw, th)
    img, alphas = rasterize_to_pixels(*leaves, w, h, ts, offsets, order)
    torch.autograd.backward([img], [st.v])
    return {"image": img.detach(), "alpha": alphas.detach(), "tiles": tiles, "offsets": offsets,
            "grads": [v.grad for v in leaves]}


def _run_mcmc(st):
    from ubs.mcmc import add_new_gs, perturb_xyz, relocate_gs
    m, opt = st.m, st.m.optimizer
    relocate_gs(m, st.dead, generator=st.g)
    perturb_xyz(m, 5e5 * LRS["xyz"] * 1e-3, generator=st.g)
    params, state = dict(m.params), {k: dict(opt.state[v]) for k, v in m.params.items()}
    added = add_new_gs(m, 1 << 30, generator=st.g)
    grown = {k: getattr(m, "_" + k) for k in NAMES}
    out = {"added": added, "params": {k: v.detach() for k, v in grown.items()},
           "m": {k: opt.state[v]["exp_avg"] for k, v in grown.items()}}
    # the model as it was before the growth, so that a pass can be repeated
    for group in opt.param_groups:
        k = group["name"]
        opt.state.pop(grown[k], None)
        group["params"][0] = params[k]
        opt.state[params[k]] = state[k]
        setattr(m, "_" + k, params[k])
    return out


# ----------------------------------------------------------------------- work
def work(case):
    """Bytes: every input read and every output written once.  Operations:
    the blend's per-pixel arithmetic over contributing (pixel, primitive)
    pairs (31 forward, 60 backward; about 80 pairs a pixel where the scene is
    dense, the scene's coverage where it is not), the separable window sums of
    SSIM, Adam's and the per-primitive chain's arithmetic."""
    kind = case["kind"]
    dim, n, sizes = case.get("dim", 6), case.get("n", 0), _sizes(case) if "views" in case else []
    pixels, c = sum(w * h for w, h in sizes), len(sizes)
    params = n * 4 * (3 + (dim - 3) + dim + dim * (dim - 1) // 2 + 1 + (dim - 2) + 3)
    if kind == "loss":
        return {"bytes": pixels * 36, "flops": pixels * 3 * 392}
    if kind == "mcmc":
        return {"bytes": 3 * params * 2.04 + n * 24, "flops": n * 150}
    pairs = 0
    for w, h in sizes:
        f = (300.0 / 256 if n <= 50_000 else 1500.0 / 1920) * w / (3.0 if n <= 50_000 else 4.0)
        area = 3.1 * (0.021 * f) ** 2 + 3.1 * EPS2D if kind != "features" else 40.0
        pairs += min(80.0 * w * h, 0.7 * n * area)
    ch = case.get("channels", 3)
    if kind == "features":
        return {"bytes": n * 4 * (16 + 2 * ch) + pixels * 4 * (2 * ch + 1),
                "flops": pairs * (85 + 6 * ch)}
    train = kind in ("train", "iterate") or case.get("grad", False)
    by, fl = params + pixels * 16, pairs * 31 + n * c * 600
    if train:
        by, fl = by + params + pixels * 12, fl + pairs * 60 + n * c * 1500
    if kind == "iterate":
        by, fl = by + 5 * params, fl + pixels * 3 * 392 + params / 4 * 15
    return {"bytes": by, "flops": fl}


# ------------------------------------------------------- 64-bit restatement
class _Whiten(torch.autograd.Function):
    """y = L^-1 x with L the Cholesky factor of V.  The backward is the
    model's own rule for V: with a = L^-T g and U = L^-T phi(L^T tril(-a y^T)),
    dV = sym(L^-1 U^T) (the derivative of y would be sym(U L^-1))."""

    @staticmethod
    def forward(ctx, V, x):
        L = torch.linalg.cholesky(V)
        y = torch.linalg.solve_triangular(L, x[..., None], upper=False)[..., 0]
        ctx.save_for_backward(L, y)
        return y

    @staticmethod
    def backward(ctx, g):
        L, y = ctx.saved_tensors
        Lt = L.transpose(-1, -2)
        a = torch.linalg.solve_triangular(Lt, g[..., None], upper=True)[..., 0]
        S = (Lt @ (-(a[..., :, None] * y[..., None, :])).tril()).tril()
        S = S - 0.5 * torch.diag_embed(torch.diagonal(S, dim1=-2, dim2=-1))
        U = torch.linalg.solve_triangular(Lt, S, upper=True)
        G = torch.linalg.solve_triangular(L, U.transpose(-1, -2), upper=False)
        return 0.5 * (G + G.transpose(-1, -2)), a


def _project64(p, cam, near=0.01, far=1e10, shown=None):
    """One view's primitives in 64 bits: means2d, conics, opacities, betas,
    colours, depths of the visible ones, front to back, and their indices."""
    vm, K, w, h, time = cam
    vm, K = vm.cuda().double(), K.cuda().double()
    dim = p["scale"].shape[1]
    k = dim - 3
    s, b = F.softplus(p["scale"], threshold=1e9), 4.0 * torch.exp(p["beta"])
    n = s.shape[0]
    R, t = vm[:3, :3], vm[:3, 3]
    with torch.no_grad():
        q = p["xyz"] - (-(R.t() @ t))
        q = q / q.norm(dim=1, keepdim=True)
        if k == 4:
            q = torch.cat([q, q.new_full((n, 1), time)], 1)
    lt = p["l_triangle"]
    one, a01, a02, a12 = torch.ones_like(lt[:, 0]), lt[:, 0], lt[:, 1], lt[:, 2]
    rot = torch.stack([one, a01, a02, -a01, one, a12, -a02, -a12, one], 1).view(n, 3, 3)
    rows = [torch.cat([rot * s[:, None, :3], s.new_zeros(n, 3, k)], 2)]
    at = 3
    for r in range(3, dim):
        rows.append(torch.cat([lt[:, at:at + r], s[:, r:r + 1], s.new_zeros(n, dim - r - 1)], 1)[:, None])
        at += r
    Lf = torch.cat(rows, 1)
    V = Lf @ Lf.transpose(1, 2)
    x = q - p["mean"]
    adj = (b[:, 1:] / 4).clamp(max=1.0)
    reg = (V[:, :3, 3:] @ torch.linalg.inv(V[:, 3:, 3:])) * adj[:, None]
    m = p["xyz"] + (reg @ x[..., None])[..., 0]
    C = V[:, :3, :3] - reg @ V[:, 3:, :3]
    y = _Whiten.apply(V[:, 3:, 3:], x)
    fall = (1 - torch.tanh(y * y).clamp(0, 1 - 2.0 ** -23)) ** b[:, 1:]
    o = torch.sigmoid(p["opacity"].reshape(-1)) * fall.prod(1)
    up = C.triu()
    C = up + up.transpose(1, 2) - torch.diag_embed(torch.diagonal(C, dim1=1, dim2=2))
    pc = m @ R.t() + t
    C = R @ C @ R.t()
    fx, fy, cx, cy = K[0, 0], K[1, 1], K[0, 2], K[1, 2]
    z = pc[:, 2]
    ok = (z >= near) & (z <= far)
    z = torch.where(ok, z, torch.ones_like(z))
    lx, ly = 0.15 * w / fx, 0.15 * h / fy
    tx = z * torch.minimum((w - cx) / fx + lx, torch.maximum(-(cx / fx + lx), pc[:, 0] / z))
    ty = z * torch.minimum((h - cy) / fy + ly, torch.maximum(-(cy / fy + ly), pc[:, 1] / z))
    zero = torch.zeros_like(z)
    J = torch.stack([fx / z, zero, -fx * tx / z ** 2, zero, fy / z, -fy * ty / z ** 2], 1).view(n, 2, 3)
    c2 = J @ C @ J.transpose(1, 2)
    u = torch.stack([fx * pc[:, 0] / z + cx, fy * pc[:, 1] / z + cy], 1)
    A, B, D = c2[:, 0, 0] + EPS2D, c2[:, 1, 0], c2[:, 1, 1] + EPS2D
    det = A * D - B * c2[:, 0, 1]
    with torch.no_grad():
        half = 0.5 * (A + D)
        rad = torch.ceil(torch.sqrt(half + torch.sqrt((half * half - det).clamp(min=0.01))))
        ok = ok & (det > 0) & (rad > 0) & (u[:, 0] + rad > 0) & (u[:, 0] - rad < w) & \
            (u[:, 1] + rad > 0) & (u[:, 1] - rad < h)
        if shown is not None:
            ok = ok & shown
        idx = torch.nonzero(ok)[:, 0]
        idx = idx[torch.sort(z[idx].float(), stable=True).indices]
    conic = torch.stack([D / det, -B / det, A / det], 1)
    return u[idx], conic[idx], o[idx], b[idx, 0], p["rgb"][idx], z[idx], idx


def _blend64(u, conic, o, b, col, w, h, bg, v=None, budget=12_000_000):
    """Front-to-back blend in 64 bits over bands of rows: image [h, w, CH] and
    alpha [h, w]; with v = (v_image, v_alpha) also accumulates the gradients
    of the five leaves and returns them."""
    leaves = [t.detach().clone().requires_grad_(v is not None) for t in (u, conic, o, b, col)]
    u, conic, o, b, col = leaves
    with torch.no_grad():
        det = conic[:, 0] * conic[:, 2] - conic[:, 1] ** 2
        hx, hy = torch.sqrt(conic[:, 2] / det), torch.sqrt(conic[:, 0] / det)
        x0 = torch.ceil(u[:, 0] - hx - 0.5).clamp(0, w).long()
        x1 = (torch.floor(u[:, 0] + hx - 0.5) + 1).clamp(0, w).long()
        y0 = torch.ceil(u[:, 1] - hy - 0.5).clamp(0, h).long()
        y1 = (torch.floor(u[:, 1] + hy - 0.5) + 1).clamp(0, h).long()
        nx = (x1 - x0).clamp(min=0)
        per_row = torch.zeros(h + 1, dtype=torch.int64, device=u.device)
        per_row.index_add_(0, y0, nx * (y1 > y0))
        per_row.index_add_(0, torch.maximum(y0, y1), -nx * (y1 > y0))
        load = per_row.cumsum(0)[:h].cpu().numpy()
    img, alpha = u.new_zeros(h, w, col.shape[1]), u.new_zeros(h, w)
    top = 0
    while top < h:
        bot, total = top + 1, load[top]
        while bot < h and total + load[bot] <= budget:
            total += load[bot]
            bot += 1
        with torch.set_grad_enabled(v is not None):
            with torch.no_grad():
                ya, yb = y0.clamp(min=top), y1.clamp(max=bot)
                cnt = nx * (yb - ya).clamp(min=0)
                who = torch.repeat_interleave(torch.arange(cnt.numel(), device=u.device), cnt)
                k = torch.arange(who.numel(), device=u.device) - (cnt.cumsum(0) - cnt)[who]
                X, Y = x0[who] + k % nx[who], ya[who] + k // nx[who]
                dx, dy = u[who, 0] - X - 0.5, u[who, 1] - Y - 0.5
                s = conic[who, 0] * dx * dx + 2 * conic[who, 1] * dx * dy + conic[who, 2] * dy * dy
                keep = (s >= 0) & (s < 1)
                who, pix = who[keep], ((Y - top) * w + X)[keep]
                pix, order = torch.sort(pix, stable=True)
                who = who[order]
                X, Y = pix % w, pix // w + top
                del k, dx, dy, s, keep, order
            g = [t[who] for t in leaves]
            dx, dy = g[0][:, 0] - X - 0.5, g[0][:, 1] - Y - 0.5
            s = g[1][:, 0] * dx * dx + 2 * g[1][:, 1] * dx * dy + g[1][:, 2] * dy * dy
            a = (g[2] * (1 - s) ** g[3]).clamp(max=0.999)
            la = torch.log1p(-a)
            run = la.cumsum(0)
            with torch.no_grad():
                first = torch.ones_like(pix, dtype=torch.bool)
                first[1:] = pix[1:] != pix[:-1]
                at = torch.cummax(torch.where(first, torch.arange(pix.numel(), device=u.device), 0), 0).values
            before = run - la
            T = torch.exp(before - before[at])
            wt = torch.where(T * (1 - a) > 1e-4, a * T, 0.0)
            cols = torch.zeros((bot - top) * w, col.shape[1], dtype=u.dtype, device=u.device)
            cols = cols.index_add(0, pix, wt[:, None] * g[4])
            acc = torch.zeros((bot - top) * w, dtype=u.dtype, device=u.device).index_add(0, pix, wt)
            if bg is not None:
                cols = cols + (1 - acc)[:, None] * bg
            img[top:bot], alpha[top:bot] = cols.detach().view(bot - top, w, -1), acc.detach().view(bot - top, w)
            if v is not None and who.numel():
                tot = (cols.view(bot - top, w, -1) * v[0][top:bot]).sum()
                if v[1] is not None:
                    tot = tot + (acc.view(bot - top, w) * v[1][top:bot]).sum()
                tot.backward()
        top = bot
    return (img, alpha) if v is None else [torch.zeros_like(t) if t.grad is None else t.grad for t in leaves]


def _ssim64(x, y):
    d = torch.arange(11, dtype=torch.float64, device=x.device) - 5
    g = torch.exp(-d * d / 4.5)
    g = g / g.sum()
    win = (g[:, None] * g[None]).expand(x.shape[1], 1, 11, 11).contiguous()

    def conv(t):
        return F.conv2d(t, win, padding=5, groups=x.shape[1])

    mx, my = conv(x), conv(y)
    sx, sy, sxy = conv(x * x) - mx ** 2, conv(y * y) - my ** 2, conv(x * y) - mx * my
    m = (2 * mx * my + 1e-4) * (2 * sxy + 9e-4) / ((mx ** 2 + my ** 2 + 1e-4) * (sx + sy + 9e-4))
    return m.mean()


def _train_loss64(x, y):
    return 0.8 * (x - y).abs().mean() + 0.2 * (1 - _ssim64(x, y))


def exact(case, seed):
    kind = case["kind"]
    if kind == "mcmc" or case.get("n", 0) * len(_sizes(case)) > 6_000_000:
        return None  # the draws are the library's own; and too long in 64 bits
    if kind == "loss":
        img, gt = (t.double() for t in _loss_images(case, seed))
        img.requires_grad_(True)
        loss = _train_loss64(img, gt)
        loss.backward()
        return {"loss": loss.detach(), "grad": img.grad}
    if kind == "features":
        return _exact_features(case, seed)
    raw = _scene(case, seed)
    cams = _cameras(case, seed)
    grad = kind in ("train", "iterate") or case.get("grad", False)
    p = {k: v.double().requires_grad_(grad) for k, v in raw.items()}
    bg = _background(case, seed).double() if kind != "viewer" else torch.ones(1, 3, device="cuda").double()
    shown, near, far = None, 0.01, 1e10
    if kind == "viewer":
        shown, near, far = torch.ones(case["n"], dtype=torch.bool, device="cuda"), 1e-3, 1e3
        for t in (raw["beta"][:, 0], raw["beta"][:, 1:4].mean(1)):
            lo, hi = (torch.quantile(t, q) for q in (0.05, 0.95))
            shown &= (t >= lo) & (t <= hi)
    with torch.no_grad():
        views = [_project64(p, c, near, far, shown) for c in cams]
        mode = case.get("mode", "RGB")
        imgs = []
        for q, c, back in zip(views, cams, bg):
            col = torch.cat([q[4], q[5][:, None]], 1) if mode == "RGB+D" else q[4]
            back = torch.cat([back, back.new_zeros(1)]) if mode == "RGB+D" else back
            imgs.append(_blend64(*q[:4], col, c[2], c[3], back))
    w, h = cams[0][2], cams[0][3]
    if kind == "request":
        return {"image": imgs[0][0].view(-1, 3), "alpha": imgs[0][1].view(-1)}
    if kind == "viewer":
        return {"image": imgs[0][0]}
    out = {}
    if kind == "dropin":
        img, alpha = imgs[0]
        out = {"image": img.permute(2, 0, 1), "alpha": alpha[None, ..., None], "radii": None,
               "tiles": None, "offsets": None}
        if not grad:
            return out
    flat = torch.cat([i.reshape(-1, i.shape[-1])[:, :3] for i, _ in imgs]).requires_grad_(True)
    target = _images(case, seed).double()
    if kind == "iterate":
        loss = _train_loss64(flat.view(1, h, w, 3).permute(0, 3, 1, 2), target.view(1, h, w, 3).permute(0, 3, 1, 2))
    else:
        loss = (flat - target).abs().mean()
    loss.backward()
    at = 0
    for c, back in zip(cams, bg):
        v = flat.grad[at:at + c[2] * c[3]].view(c[3], c[2], 3)
        at += c[2] * c[3]
        q = _project64(p, c)
        torch.autograd.backward(q[:5], _blend64(*q[:5], c[2], c[3], back, (v, None)))
        del q
    out["loss"] = loss.detach()
    out["grads"] = {k: t.grad for k, t in p.items()}
    if kind == "iterate":
        out["image"] = flat.detach()
        m0 = _model(case, seed)
        out["params"], out["m"] = {}, {}
        for k, t in p.items():
            st = m0.optimizer.state[m0.params[k]]
            m = 0.9 * st["exp_avg"].double() + 0.1 * t.grad
            v2 = 0.999 * st["exp_avg_sq"].double() + 0.001 * t.grad ** 2
            T = ADAM_T + 1
            den = torch.sqrt(v2) / math.sqrt(1 - 0.999 ** T) + 1e-15
            out["params"][k] = t.detach() - LRS[k] / (1 - 0.9 ** T) * m / den
            out["m"][k] = m
    return out


def _exact_features(case, seed):
    p = _projected(case, seed)
    (w, h), = _sizes(case)
    order = torch.sort(p["depths"][0], stable=True).indices
    keys = ("means2d", "conics", "opacities", "betas", "colors")
    q = [p[k][0].double()[order] for k in keys]
    img, alpha = _blend64(*q, w, h, None)
    v = torch.randn(1, h, w, case["channels"], generator=_gen(seed, 6), device="cuda").double()[0]
    grads = dict(zip(keys, _blend64(*q, w, h, None, (v, None))))
    for k in keys:
        g = torch.zeros_like(grads[k])
        g[order] = grads[k]
        grads[k] = g[None]
    return {"image": img[None], "alpha": alpha[None, ..., None], "tiles": None, "offsets": None,
            "grads": [grads[k] for k in ("means2d", "conics", "colors", "opacities", "betas")]}
