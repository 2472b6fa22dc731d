"""The work a user of this framework has it do, as measurable cases.

Each case is one pass through a public entry point: a render, a batch of render
requests, a training step (plain, prior-guided, batched over views), the differentiable
render with its backward, densification, the kNN initialisation and the evaluation
metrics. Scenes follow the distributions of msplat_street_b200.scenes (a ball scene in
[-1, 1]^3 seen from a sphere around it, a 20 x 4 x 20 m street seen from cameras on a
line inside it); they are drawn on the GPU from the case's seed.

``exact`` evaluates the same pass in 64-bit torch: projection, tile lists, compositing,
the loss, every gradient (by autograd over chunks of tiles) and the Adam update.
"""
import math

import numpy as np
import torch

from msplat_street_b200 import autograd, scenes
from msplat_street_b200.backend import AdamState, BatchItem, Context, GaussianParams, PriorStep
from msplat_street_b200.camera import look_at, prepare_cam
from msplat_street_b200.workloads import BACKGROUND, BATCH_RESOLUTIONS

DEV = "cuda"
LRS = (1.6e-4, 5e-3, 1e-3, 2.5e-3, 1.25e-4, 0.05)  # the trainer's learning rates
SERVE_RESOLUTIONS = ((512, 512), (1280, 720), (1920, 1080))


def listed():
    return [
        # an interactive preview: few Gaussians, a small frame; the latency of one call
        {"name": "render_small", "kind": "render", "scene": "ball", "n": 10_000, "w": 256, "h": 256, "dtu": 3},
        # a viewer (or the targets of a synthetic run) inside a trained street scene
        {"name": "render_street", "kind": "render", "scene": "street", "n": 500_000, "w": 1024, "h": 512, "dtu": 3},
        # a render server's worker: eight requests over four resident scenes, three sizes
        {"name": "serve_mixed", "kind": "serve", "n": 3_000_000, "scenes": 4, "requests": 8},
        # the smallest training run: launches and host time count
        {"name": "train_small", "kind": "train", "scene": "ball", "n": 10_000, "w": 256, "h": 256, "dtu": 3},
        # street training early in the schedule (SH degree 0 in use)
        {"name": "train_street", "kind": "train", "scene": "street_init", "n": 100_000, "w": 1024, "h": 512,
         "dtu": 0},
        # street training after densification: a large model, all SH bands, a ragged size
        {"name": "train_large", "kind": "train", "scene": "street", "n": 1_000_000, "w": 1600, "h": 1060, "dtu": 3},
        # prior-guided street training: sky, depth prior, exposure, needle cap
        {"name": "train_prior", "kind": "prior", "scene": "street_init", "n": 100_000, "w": 1000, "h": 500, "dtu": 1},
        # several views of uneven sizes in one graph-replayed step
        {"name": "train_batch", "kind": "batch", "scene": "street_init", "n": 100_000, "views": 8, "dtu": 0},
        # the splatting path inside a torch program: render, loss, backward
        {"name": "autograd", "kind": "autograd", "scene": "ball", "n": 200_000, "w": 1024, "h": 768, "dtu": 3},
        # a refinement step of the schedule
        {"name": "densify", "kind": "densify", "n": 300_000},
        # a training run's start from a point cloud
        {"name": "init_points", "kind": "init", "n": 400_000},
        # evaluation of a rendered view
        {"name": "evaluate", "kind": "metrics", "w": 1297, "h": 840},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "serve", "train", "train", "train", "prior", "batch", "autograd",
                       "densify", "init", "metrics"])
    w = _log(rng, 200, 1920)
    h = max(120, min(1080, int(w * rng.uniform(0.45, 1.0))))
    if kind == "render":
        return {"kind": kind, "scene": rng.choice(["ball", "street"]), "n": _log(rng, 8_000, 1_500_000), "w": w, "h": h,
                "dtu": rng.randrange(4)}
    if kind == "serve":
        return {"kind": kind, "n": _log(rng, 100_000, 2_500_000), "scenes": rng.randrange(1, 5),
                "requests": rng.randrange(1, 9)}
    if kind in ("train", "prior", "autograd"):
        w = min(w, 1600)
        return {"kind": kind, "scene": rng.choice(["ball", "street", "street_init"]) if kind == "train" else
                ("street_init" if kind == "prior" else "ball"),
                "n": _log(rng, 8_000, 600_000 if kind == "train" else 200_000), "w": w, "h": min(h, 1060),
                "dtu": rng.randrange(4)}
    if kind == "batch":
        return {"kind": kind, "scene": "street_init", "n": _log(rng, 10_000, 150_000), "views": rng.randrange(2, 9),
                "dtu": rng.randrange(4)}
    if kind == "densify":
        return {"kind": kind, "n": _log(rng, 10_000, 300_000)}
    if kind == "init":
        return {"kind": kind, "n": _log(rng, 1_000, 800_000)}
    return {"kind": "metrics", "w": w, "h": h}


# --- inputs -------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _scene(kind, n, seed):
    """A scene drawn from the distributions of msplat_street_b200.scenes, on the GPU.
    "street_init": a street some steps into its training -- scales from the point
    spacing (not yet isotropic copies of one number), low opacities."""
    g = _gen(seed)
    if kind == "ball":
        lo, hi, ls, lv, om, ov = (-1.0, -1.0, -1.0), (1.0, 1.0, 1.0), -4.0, 0.5, 0.0, 1.0
    else:
        lo, hi, ls, lv, om, ov = scenes.STREET_LO, scenes.STREET_HI, -4.0, 0.5, 0.0, 1.0
        if kind == "street_init":
            ls, lv, om, ov = math.log(0.6 * (1600.0 / n) ** (1.0 / 3.0)), 0.3, -1.5, 1.0
    lo, hi = (torch.tensor(v, device=DEV) for v in (lo, hi))
    means = lo + (hi - lo) * torch.rand((n, 3), generator=g, device=DEV)
    scales = ls + lv * torch.randn((n, 3), generator=g, device=DEV)
    quats = torch.nn.functional.normalize(torch.randn((n, 4), generator=g, device=DEV), dim=1)
    opac = om + ov * torch.randn((n, 1), generator=g, device=DEV)
    dc = 0.3 * torch.randn((n, 3), generator=g, device=DEV)
    rest = 0.05 * torch.randn((n, 15, 3), generator=g, device=DEV)
    return GaussianParams(means, scales, quats, dc, rest, opac)


def _cameras(kind, w, h, count, seed):
    rng = np.random.default_rng(seed)
    if kind == "ball":
        return [scenes.sphere_camera(rng, w, h, 3.0 if w <= 512 else 5.0) for _ in range(count)]
    out = []
    for _ in range(count):
        eye = np.array([rng.uniform(-1, 1), 1.5, rng.uniform(-5, 5)])
        yaw = math.radians(rng.uniform(-30, 30))
        out.append(prepare_cam(look_at(eye, eye + np.array([math.sin(yaw), 0.0, math.cos(yaw)])), w, h, 0.5 * w,
                               0.5 * w, w / 2.0, h / 2.0))
    return out


_CONTEXTS = {}


def _context(user="main"):
    """One context for the program's renders and steps, as a viewer or trainer holds, and
    one for a render server's worker, which sets its own block shape."""
    if user not in _CONTEXTS:
        _CONTEXTS[user] = Context()
        if user == "server":
            _CONTEXTS[user].set_raster_shape(1)
    return _CONTEXTS[user]


def _targets(kind, n, cams, seed):
    """Targets: renders of another scene of the same distribution."""
    src = "street" if kind == "street_init" else kind
    gt = _scene(src, 3 * n if kind == "street_init" else n, seed + 7919)
    out = [_context().render(gt, c, BACKGROUND).clone() for c in cams]
    return out


def _serve_views(case, seed):
    rng = np.random.default_rng(seed)
    sizes = [int(case["n"])] + [int(math.exp(rng.uniform(math.log(50_000), math.log(case["n"]))))
                                for _ in range(case["scenes"] - 1)]
    views = []
    for r in range(case["requests"]):
        w, h = SERVE_RESOLUTIONS[r % 3]
        views.append((r % len(sizes), scenes.sphere_camera(rng, w, h)))
    return sizes, views


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "k": 0}
    if kind == "render":
        s["p"] = _scene(case["scene"], case["n"], seed)
        s["cam"] = _cameras(case["scene"], case["w"], case["h"], 1, seed)[0]
        s["ctx"] = _context()
    elif kind == "serve":
        sizes, views = _serve_views(case, seed)
        ps = [_scene("ball", n, seed * 16 + i) for i, n in enumerate(sizes)]
        s["items"] = [BatchItem(ps[i], c, BACKGROUND) for i, c in views]
        s["outs"] = [torch.empty((c.height, c.width, 3), device=DEV) for _, c in views]
        s["ctx"] = _context("server")
    elif kind in ("train", "prior", "batch"):
        s["p"] = _scene(case["scene"], case["n"], seed)
        s["adam"] = AdamState.zeros_like(s["p"], LRS)
        s["stats"] = [torch.zeros(case["n"], device=DEV) for _ in range(3)]
        if kind == "batch":
            rng = np.random.default_rng(seed)
            cams = []
            for i in range(case["views"]):
                w, h = BATCH_RESOLUTIONS[int(rng.integers(len(BATCH_RESOLUTIONS)))]
                cams += _cameras(case["scene"], w, h, 1, seed * 64 + i)
            s["ctx"] = Context()  # a trainer's own: it keeps the captured step
            s["ctx"].set_graph(True)
        else:
            cams = _cameras(case["scene"], case["w"], case["h"], 4, seed)
            s["ctx"] = _context()
        gts = _targets(case["scene"], case["n"], cams, seed)
        s["views"] = list(zip(cams, gts))
        if kind == "prior":
            s["prior"] = _prior(case, seed)
    elif kind == "autograd":
        s["p"] = _scene(case["scene"], case["n"], seed)
        for t in s["p"].tensors():
            t.requires_grad_(True)
        cams = _cameras(case["scene"], case["w"], case["h"], 1, seed)
        s["views"] = list(zip(cams, _targets(case["scene"], case["n"], cams, seed)))
    elif kind == "densify":
        n, cap = case["n"], 4 * case["n"]
        g = _gen(seed + 1)
        p = _scene("street", n, seed)
        # a sixth is split, an eighth cloned, a tenth pruned
        mixed = torch.randperm(n, generator=g, device=DEV)
        split, clone, prune = mixed[:n // 6], mixed[n // 6:n // 6 + n // 8], mixed[-(n // 10):]
        p.scales.clamp_(max=-4.0)
        p.scales[split, 0] = -3.0 + 0.2 * torch.rand(len(split), generator=g, device=DEV)
        p.opacities.clamp_(min=-1.0)
        p.opacities[prune] = -3.0
        steps = 1 + torch.randint(0, 30, (n,), generator=g, device=DEV).float()
        grad = 2e-7 * torch.rand(n, generator=g, device=DEV)
        grad[split] += 1e-6
        grad[clone] += 1e-6

        def grow(t, r=None):
            b = torch.zeros((cap,) + tuple(t.shape[1:]), device=DEV)
            b[:n] = t if r is None else r * torch.randn(t.shape, generator=g, device=DEV)
            return b
        s["buf"] = [grow(t) for t in p.tensors()]
        s["m1"] = [grow(t, 1e-3) for t in p.tensors()]
        s["m2"] = [grow(t, 1e-3).square_() for t in p.tensors()]
        s["vis"], s["gn"] = steps, steps * grad
        s["ms"] = 0.04 * torch.rand(n, generator=g, device=DEV)
        s["ctx"] = _context()
    elif kind == "init":
        n = case["n"]
        g = _gen(seed)
        # surfaces and clutter, as a structure-from-motion cloud has them
        p = _scene("street", n, seed).means
        flat = torch.rand(n, generator=g, device=DEV) < 0.6
        p[flat, 1] = 0.05 * torch.randn(int(flat.sum()), generator=g, device=DEV)
        s["pts"] = p.contiguous()
        s["rgb"] = torch.randint(0, 256, (n, 3), generator=g, device=DEV, dtype=torch.uint8)
        s["ctx"] = _context()
    else:
        s["gt"], s["img"] = _pictures(case, seed)
        s["ctx"] = _context()
    return s


def _pictures(case, seed):
    g = _gen(seed)
    small = torch.rand((1, 3, case["h"] // 8 + 1, case["w"] // 8 + 1), generator=g, device=DEV)
    gt = torch.nn.functional.interpolate(small, (case["h"], case["w"]), mode="bilinear")[0].permute(1, 2, 0)
    img = (gt + 0.05 * torch.randn(gt.shape, generator=g, device=DEV)).clamp(0, 1)
    return gt.contiguous(), img.contiguous()


def _prior(case, seed):
    g = _gen(seed + 2)
    pw, ph = case["w"] // 2 + 3, case["h"] // 2 + 1
    depth = 2.0 + 8.0 * torch.rand((ph // 8 + 1, pw // 8 + 1), generator=g, device=DEV)
    depth = depth.repeat_interleave(8, 0).repeat_interleave(8, 1)[:ph, :pw].contiguous()
    depth[torch.rand((ph, pw), generator=g, device=DEV) < 0.08] = 0.0
    aux = torch.randint(0, 256, (ph, pw, 4), generator=g, device=DEV, dtype=torch.uint8)
    aux[..., 1] = torch.where(torch.rand((ph, pw), generator=g, device=DEV) < 0.2, 200, 30).to(torch.uint8)
    aux[..., 2] = torch.where(torch.rand((ph, pw), generator=g, device=DEV) < 0.1, 0, 255).to(torch.uint8)
    tex = torch.rand((128, 256, 3), generator=g, device=DEV)
    expo = torch.eye(3, device=DEV).reshape(-1)
    expo = torch.cat([expo, torch.zeros(3, device=DEV)]).repeat(4, 1)
    expo += 0.02 * torch.randn(expo.shape, generator=g, device=DEV)
    return PriorStep(
        aux=True, sky=True, sky_tex=tex, sky_grad=torch.zeros_like(tex), sky_exp_avg=torch.zeros_like(tex),
        sky_exp_avg_sq=torch.zeros_like(tex), sky_frame=(0, -1, 0, 1, 0, 0, 0, 0, -1), sky_step_size=1e-3,
        sky_bc2_sqrt=1.0, prior_depth=depth, prior_aux=aux, has_depth=True, has_sky_mask=True, depth_weight=0.05,
        sky_weight=0.02, fill_weight=0.01, loss_terms=torch.zeros(4, device=DEV), exposure=True, cam_index=1,
        expo_params=expo.contiguous(), expo_exp_avg=torch.zeros_like(expo), expo_exp_avg_sq=torch.zeros_like(expo),
        expo_grad=torch.zeros(12, device=DEV), expo_step_size=1e-3, expo_bc2_sqrt=1.0, expo_reg=1e-2,
        log_max_scale_ratio=math.log(8.0))


# --- one pass -------------------------------------------------------------------------

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "render":
        return s["ctx"].render(s["p"], s["cam"], BACKGROUND, degrees_to_use=case["dtu"])
    if kind == "serve":
        return s["ctx"].render_batch(s["items"], s["outs"])
    if kind in ("train", "prior"):
        cam, gt = s["views"][s["k"] % len(s["views"])]
        s["k"] += 1
        ctx = s["ctx"]
        ctx.set_prior(s.get("prior"))
        ctx.train_step(s["p"], s["adam"], cam, BACKGROUND, gt, s["stats"], degrees_to_use=case["dtu"])
        out = {"params": s["p"].tensors(), "exp_avg": s["adam"].exp_avg, "exp_avg_sq": s["adam"].exp_avg_sq,
               "stats": s["stats"], "loss": ctx.loss_tensor()}
        if kind == "prior":
            ctx.set_prior(None)
            pr = s["prior"]
            out["sky"] = [pr.sky_tex, pr.sky_exp_avg]
            out["expo"] = [pr.expo_params, pr.expo_exp_avg]
            out["terms"] = pr.loss_terms
        return out
    if kind == "batch":
        losses = s["ctx"].train_batch(s["p"], s["adam"], s["views"], BACKGROUND, s["stats"],
                                      degrees_to_use=case["dtu"])
        return {"params": s["p"].tensors(), "exp_avg": s["adam"].exp_avg, "exp_avg_sq": s["adam"].exp_avg_sq,
                "stats": s["stats"], "loss": losses}
    if kind == "autograd":
        cam, gt = s["views"][0]
        p = s["p"]
        for t in p.tensors():
            t.grad = None
        img = autograd.render(p, cam, BACKGROUND, degrees_to_use=case["dtu"])
        loss = autograd.ssim_l1_loss(img, gt)
        loss.backward()
        return {"image": img.detach(), "loss": loss.detach(), "grads": [t.grad for t in p.tensors()]}
    if kind == "densify":
        n = s["ctx"].densify(case["n"], s["buf"], s["m1"], s["m2"], s["gn"], s["vis"], s["ms"], 512.0, seed=7,
                             size_thresh=0.03)
        return {"count": n, "params": [b[:n] for b in s["buf"]], "exp_avg": [b[:n] for b in s["m1"]],
                "exp_avg_sq": [b[:n] for b in s["m2"]]}
    if kind == "init":
        return s["ctx"].init_gaussians(s["pts"], s["rgb"]).tensors()
    return list(s["ctx"].image_metrics(s["img"], s["gt"]))


# --- the least a pass moves and computes ------------------------------------------------

def _views(case):
    if case["kind"] == "batch":  # the mean size of the resolutions drawn from
        return case["views"], case["views"] * sum(w * h for w, h in BATCH_RESOLUTIONS) / len(BATCH_RESOLUTIONS)
    return 1, case["w"] * case["h"]


def work(case):
    kind = case["kind"]
    n = case.get("n", 0)
    used = 14 + 3 * (case.get("dtu", 3) + 1) ** 2 - 3  # floats of a Gaussian that a frame reads
    if kind == "render":
        return {"bytes": n * used * 4 + 12 * case["w"] * case["h"], "flops": n * 300 + 100 * case["w"] * case["h"]}
    if kind == "serve":
        sizes, views = _serve_views(case, 0)
        pix = sum(c.width * c.height for _, c in views)
        return {"bytes": sum(sizes[i] for i, _ in views) * 236 + 12 * pix,
                "flops": sum(sizes[i] for i, _ in views) * 300 + 100 * pix}
    if kind in ("train", "prior", "batch"):
        v, pix = _views(case)
        # parameters and two moments read and written once, statistics, targets
        return {"bytes": n * (used * 24 + 24) + 12 * pix, "flops": n * (700 * v + used * 15) + 2200 * pix}
    if kind == "autograd":
        _, pix = _views(case)
        return {"bytes": n * used * 8 + 28 * pix, "flops": n * 1000 + 2200 * pix}
    if kind == "densify":  # every row read once, about 1.2 times as many written
        return {"bytes": n * 59 * 12 * 2.2 + 12 * n, "flops": n * 40}
    if kind == "init":
        return {"bytes": n * (15 + 236), "flops": n * 400}
    return {"bytes": 24 * case["w"] * case["h"], "flops": 1100 * case["w"] * case["h"]}


# --- the same passes in 64 bits ---------------------------------------------------------

_C1, _C0 = 0.4886025119029199, 0.28209479177387814
_C2 = (1.0925484305920792, -1.0925484305920792, 0.31539156525252005, -1.0925484305920792, 0.5462742152960396)
_C3 = (-0.5900435899266435, 2.890611442640554, -0.4570457994644658, 0.3731763325901154, -0.4570457994644658,
       1.445305721320277, -0.5900435899266435)
_MOST_PAIRS = 3e9  # (pixel, Gaussian) pairs worth evaluating in 64 bits


def _project64(p, cam, dtu):
    """(xy, conic, colour, opacity, depth, radius, tile rectangle, index) of the visible
    Gaussians; p: six float64 tensors."""
    means, scales, quats, dc, rest, opac = p
    V = torch.tensor(np.asarray(cam.viewmat, np.float64), device=DEV)
    P = torch.tensor(np.asarray(cam.projmat, np.float64), device=DEV)
    near = ((means @ V[2, :3] + V[2, 3]) > 0.01).nonzero()[:, 0]
    m = means[near]
    pv = m @ V[:3, :3].T + V[:3, 3]
    q = torch.nn.functional.normalize(quats[near], dim=1)
    w, x, y, z = q.unbind(1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z),
                     1 - 2 * (x * x + z * z), 2 * (y * z - w * x), 2 * (x * z - w * y), 2 * (y * z + w * x),
                     1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)
    M = R * scales[near].exp()[:, None, :]
    cov = M @ M.transpose(1, 2)
    tz = pv[:, 2]
    t = []
    for c, size, f in ((0, cam.width, cam.fx), (1, cam.height, cam.fy)):
        lim = 1.3 * 0.5 * size / f
        clamped = tz * (pv[:, c] / tz).clamp(-lim, lim)
        t.append(pv[:, c] + (clamped - pv[:, c]).detach())  # the clamp passes gradients through
    zero = torch.zeros_like(tz)
    J = torch.stack([cam.fx / tz, zero, -cam.fx * t[0] / tz ** 2, zero, cam.fy / tz, -cam.fy * t[1] / tz ** 2],
                    1).reshape(-1, 2, 3)
    T = J @ V[:3, :3]
    c2 = T @ cov @ T.transpose(1, 2)
    a, b, c = c2[:, 0, 0] + 0.3, c2[:, 0, 1], c2[:, 1, 1] + 0.3
    det = a * c - b * b
    conic = torch.stack([c / det, -b / det, a / det], 1)
    half = 0.5 * (a + c)
    radius = (3 * (half + (half * half - det).clamp_min(0.1).sqrt()).sqrt()).ceil().detach()
    hom = m @ P[:, :3].T + P[:, 3]
    rw = 1 / (hom[:, 3] + 1e-6)
    xy = torch.stack([0.5 * cam.width * hom[:, 0] * rw + cam.cx - 0.5, 0.5 * cam.height * hom[:, 1] * rw + cam.cy - 0.5], 1)
    ext = torch.stack([(3 * a.sqrt()).ceil(), (3 * c.sqrt()).ceil()], 1).detach()
    cen = xy.detach() / 16
    lim = torch.tensor([cam.tiles_x, cam.tiles_y], device=DEV)
    lo = (cen - ext / 16).to(torch.int64).clamp_min(0).minimum(lim)
    hi = (cen + ext / 16 + 1).to(torch.int64).clamp_min(0).minimum(lim)
    keep = ((hi - lo).prod(1) > 0).nonzero()[:, 0]
    near, xy, conic, lo, hi, tz, radius = (v[keep] for v in (near, xy, conic, lo, hi, tz, radius))
    d = means[near].detach() - torch.tensor(np.asarray(cam.cam_pos, np.float64), device=DEV)
    x, y, z = torch.nn.functional.normalize(d, dim=1).unbind(1)
    basis = [-_C1 * y, _C1 * z, -_C1 * x, _C2[0] * x * y, _C2[1] * y * z, _C2[2] * (2 * z * z - x * x - y * y),
             _C2[3] * x * z, _C2[4] * (x * x - y * y), _C3[0] * y * (3 * x * x - y * y), _C3[1] * x * y * z,
             _C3[2] * y * (4 * z * z - x * x - y * y), _C3[3] * z * (2 * z * z - 3 * x * x - 3 * y * y),
             _C3[4] * x * (4 * z * z - x * x - y * y), _C3[5] * z * (x * x - y * y), _C3[6] * x * (x * x - 3 * y * y)]
    used = (dtu + 1) ** 2 - 1
    col = _C0 * dc[near]
    if used:
        col = col + (torch.stack(basis[:used], 1)[:, :, None] * rest[near][:, :used]).sum(1)
    return xy, conic, (col + 0.5).clamp_min(0), torch.sigmoid(opac[near][:, 0]), tz.detach(), radius, lo, hi, near


def _lists64(cam, depth, lo, hi):
    """Per tile: first entry and length in the list of Gaussians ordered by (tile, depth)."""
    order = torch.argsort(depth, stable=True)
    lo, hi = lo[order], hi[order]
    wide = hi[:, 0] - lo[:, 0]
    cnt = wide * (hi[:, 1] - lo[:, 1])
    src = torch.repeat_interleave(torch.arange(len(cnt), device=DEV), cnt)
    k = torch.arange(len(src), device=DEV) - (cnt.cumsum(0) - cnt)[src]
    tile = (lo[src, 1] + k // wide[src]) * cam.tiles_x + lo[src, 0] + k % wide[src]
    by = torch.argsort(tile, stable=True)
    length = torch.bincount(tile, minlength=cam.tiles_x * cam.tiles_y)
    return order[src[by]], length.cumsum(0) - length, length


def _chunks64(cam, ids, first, length):
    """Tiles in groups of similar list lengths: (pixel x, pixel y, list, is an entry)."""
    lx = torch.arange(16, device=DEV)
    for tiles in torch.argsort(length).split(256):
        longest = max(1, int(length[tiles].max()))
        for part in tiles.split(max(1, int(3e7 // (256 * longest)))):
            most = max(1, int(length[part].max()))
            k = torch.arange(most, device=DEV)
            real = k < length[part][:, None]
            ent = ids[(first[part][:, None] + k).clamp_max(max(len(ids) - 1, 0))] if len(ids) else torch.zeros_like(
                real, dtype=torch.int64)
            px = ((part % cam.tiles_x) * 16)[:, None, None] + lx[None, None, :].expand(1, 16, 16)
            py = ((part // cam.tiles_x) * 16)[:, None, None] + lx[None, :, None].expand(1, 16, 16)
            yield px.reshape(-1, 256), py.reshape(-1, 256), ent, real


def _composite64(px, py, ent, real, xy, conic, col, op, bg):
    """Colours (tiles, 256, 3) of one group of tiles."""
    g, cn = xy[ent], conic[ent]
    dx, dy = g[..., 0, None] - px[:, None, :], g[..., 1, None] - py[:, None, :]
    sigma = 0.5 * (cn[..., 0, None] * dx * dx + cn[..., 2, None] * dy * dy) + cn[..., 1, None] * dx * dy
    alpha = (op[ent][..., None] * torch.exp(-sigma)).clamp_max(0.999)
    ok = real[..., None] & (sigma >= 0) & (sigma < 5.55) & (alpha >= 1 / 255)
    alpha = torch.where(ok, alpha, torch.zeros_like(alpha))
    logs = torch.log1p(-alpha)
    after = logs.cumsum(1)
    alive = (after > math.log(1e-4)).to(alpha.dtype)  # the entry that would end the pixel takes no part
    weight = alpha * torch.exp(after - logs) * alive
    last = torch.exp((logs * alive).sum(1))
    out = torch.einsum("tlp,tlc->tpc", weight, col[ent]) + last[..., None] * bg
    return out.clamp(0, 1) if not torch.is_grad_enabled() else out


def _frame64(p, cam, dtu, v_of=None):
    """The image in 64 bits (or None where it would take too long); with v_of (image ->
    its gradient and more), also what v_of returned, the gradients of the six parameters,
    of the pixel centres, and the visible Gaussians' indices and radii."""
    p = [t.detach().double().requires_grad_(v_of is not None) for t in p]
    bg = torch.tensor(np.asarray(BACKGROUND, np.float64), device=DEV)
    xy, conic, col, op, depth, radius, lo, hi, vis = _project64(p, cam, dtu)
    ids, first, length = _lists64(cam, depth, lo, hi)
    if float(length.sum()) * 256 > _MOST_PAIRS:
        return None
    img = torch.zeros((cam.tiles_y * 16, cam.tiles_x * 16, 3), dtype=torch.float64, device=DEV)
    with torch.no_grad():
        for px, py, ent, real in _chunks64(cam, ids, first, length):
            img[py, px] = _composite64(px, py, ent, real, xy, conic, col, op, bg)
    img = img[:cam.height, :cam.width]
    if v_of is None:
        return img
    v, more = v_of(img)
    pad = torch.zeros((cam.tiles_y * 16, cam.tiles_x * 16, 3), dtype=torch.float64, device=DEV)
    pad[:cam.height, :cam.width] = v
    leaf = [t.detach().requires_grad_(True) for t in (xy, conic, col, op)]
    for px, py, ent, real in _chunks64(cam, ids, first, length):
        (_composite64(px, py, ent, real, *leaf, bg) * pad[py, px]).sum().backward()
    torch.autograd.backward([xy, conic, col, op], [t.grad for t in leaf])
    grads = [t.grad if t.grad is not None else torch.zeros_like(t) for t in p]
    return img, more, grads, leaf[0].grad, vis, radius


def _window64():
    g = [math.exp(-(i - 5) ** 2 / 4.5) for i in range(11)]
    return torch.tensor([v / sum(g) for v in g], dtype=torch.float64, device=DEV)


def _blur64(x, edge):
    """11-tap separable Gaussian of (channels, H, W), zero-padded or clamped to the edge."""
    k = _window64()
    pad = torch.nn.functional.pad(x[:, None], (5, 5, 5, 5), mode="replicate" if edge else "constant")
    return torch.nn.functional.conv2d(torch.nn.functional.conv2d(pad, k.view(1, 1, 1, 11)), k.view(1, 1, 11, 1))[:, 0]


def _ssim64(a, b, edge=False):
    a, b = a.permute(2, 0, 1), b.permute(2, 0, 1)
    ma, mb = _blur64(a, edge), _blur64(b, edge)
    va, vb, ab = _blur64(a * a, edge) - ma * ma, _blur64(b * b, edge) - mb * mb, _blur64(a * b, edge) - ma * mb
    return ((2 * ma * mb + 1e-4) * (2 * ab + 9e-4) / ((ma * ma + mb * mb + 1e-4) * (va + vb + 9e-4))).mean()


def _loss64(gt):
    gt = gt.double()

    def v_of(img):
        x = img.detach().requires_grad_(True)
        with torch.enable_grad():
            loss = 0.2 * (1 - _ssim64(gt, x)) + 0.8 * (x - gt).abs().mean()
            loss.backward()
        return x.grad, loss.detach()
    return v_of


def _step64(p, views, dtu):
    """The outputs of the first Adam step from zero moments and statistics."""
    total, losses, stats = None, [], None
    for cam, gt in views:
        got = _frame64(p, cam, dtu, _loss64(gt))
        if got is None:
            return None
        _, loss, grads, vxy, vis, radius = got
        losses.append(loss)
        total = grads if total is None else [a + b for a, b in zip(total, grads)]
        if stats is None:
            stats = [torch.zeros(len(p[0]), dtype=torch.float64, device=DEV) for _ in range(3)]
        stats[0][vis] += 1
        stats[1][vis] += vxy.norm(dim=1)
        stats[2][vis] = stats[2][vis].maximum(radius / max(cam.width, cam.height))
    m1, m2, new = [], [], []
    for t, g, lr in zip(p, total, LRS):
        m1.append(0.1 * g)
        m2.append(0.001 * g * g)
        new.append(t.double() - lr * g / (g.abs() + 1e-8))
    return {"params": new, "exp_avg": m1, "exp_avg_sq": m2, "stats": stats, "loss": losses}


def _three64(pts):
    """Mean distance to the three nearest other points: points sorted along x, each block
    of queries against the window of x that can hold them."""
    n = len(pts)
    p = pts.double()
    p = p[torch.argsort(p[:, 0])]
    back = torch.argsort(torch.argsort(pts.double()[:, 0]))
    out = torch.empty(n, dtype=torch.float64, device=DEV)
    reach = 8.0 * (1600.0 / n) ** (1.0 / 3.0)
    step = 1024
    for i in range(0, n, step):
        q = p[i:i + step]
        r = reach
        while True:
            lo = int(torch.searchsorted(p[:, 0].contiguous(), q[0, 0] - r))
            hi = int(torch.searchsorted(p[:, 0].contiguous(), q[-1, 0] + r))
            d = sum((q[:, None, c] - p[None, lo:hi, c]) ** 2 for c in range(3))
            best = d.topk(min(4, hi - lo), largest=False).values.sqrt()
            if best.shape[1] == min(4, n) and (hi - lo == n or float(best[:, -1].max()) <= r):
                break
            r *= 3
        out[i:i + step] = best[:, 1:].mean(1) if best.shape[1] > 1 else 1.0
    return out[back]


def exact(case, seed):
    kind = case["kind"]
    if kind == "densify" or kind == "prior":
        return None  # copies of rows and counter-based random offsets; the prior terms' own definitions
    if kind == "render":
        s = prepare(case, seed)
        with torch.no_grad():
            return _frame64(s["p"].tensors(), s["cam"], case["dtu"])
    if kind == "serve":
        s = prepare(case, seed)
        with torch.no_grad():
            return [_frame64(i.params.tensors(), i.camera, 3) for i in s["items"]]
    if kind == "train":
        s = prepare(case, seed)
        got = _step64(s["p"].tensors(), s["views"][:1], case["dtu"])
        return got and {**got, "loss": got["loss"][0]}
    if kind == "batch":
        s = prepare(case, seed)
        got = _step64(s["p"].tensors(), s["views"], case["dtu"])
        return got and {**got, "loss": torch.stack(got["loss"])}
    if kind == "autograd":
        s = prepare(case, seed)
        cam, gt = s["views"][0]
        got = _frame64(s["p"].tensors(), cam, case["dtu"], _loss64(gt))
        return got and {"image": got[0], "loss": got[1], "grads": got[2]}
    if kind == "init":
        s = prepare(case, seed)
        scales = _three64(s["pts"]).clamp_min(1e-7).log()[:, None].expand(-1, 3)
        colours = (s["rgb"].double() / 255 - 0.5) / _C0
        return [s["pts"].double(), scales, None, colours, None, None]
    gt, img = (t.double() for t in _pictures(case, seed))
    psnr = -10 * torch.log10((gt - img).square().mean())
    return [psnr, _ssim64(img, gt, edge=True), (gt - img).abs().mean()]
