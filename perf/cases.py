"""Performance cases of the framework: what a program that uses it has it do,
through the public entry points, with inputs made on the GPU from a seed.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same
kinds and ranges; ``prepare`` / ``run`` make a case's inputs and take one pass
over it, ``work`` states what the pass cannot do without, and ``exact`` gives
the pass's results in 64-bit arithmetic from plain torch expressions.

Kinds (``case["kind"]``):
  render   decode of one Gaussian set through the drop-in API, no gradients
  train    one LIG training iteration through the drop-in API under autograd:
           project, rasterize, clamp, L2, backward
  fit      one iteration of the fit engine for one level (LevelFit)
  batch    one iteration of the batched fit engine (BatchedFit)
  gatrain  one training iteration with the gradient-aware render and upscale
  handover the gradient-aware render of a fitted level and its upscale to the
           next level's size, no gradients
  views    a server's batch of region decodes of a resident set
  levels   the residual target of the next level and the compose of a decode
"""
from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from lig_b200 import gsplat2d
from lig_b200.batch import BatchedFit
from lig_b200.fit import LevelFit
from lig_b200.levels import compose, residual_target
from lig_b200.serve import GaussianSet, render_views

DEV = "cuda"
LOG_255 = math.log(255.0)


def listed():
    return [
        # a thumbnail: latency of the launches and of the host path counts
        {"name": "render_64x80", "kind": "render", "h": 64, "w": 80, "n": 400, "block": 16,
         "d0": 0.5, "d1": 4.0, "opac": True, "cov": False},
        # LIG's own loop (train_iter) on a plain single-level 512^2 fit
        {"name": "train_512", "kind": "train", "h": 512, "w": 512, "n": 50_000, "block": 16,
         "d0": 0.5, "d1": 4.0, "opac": False, "cov": False},
        # the same loop on an odd-sized photo, covariance parameters and
        # learned opacities
        {"name": "train_767x1023_opac", "kind": "train", "h": 767, "w": 1023, "n": 150_000,
         "block": 16, "d0": 0.5, "d1": 4.0, "opac": True, "cov": True},
        # the fit engine's iteration at the three level sizes of the fit
        # configurations: a small level, the dense first level of a two-level
        # fit and its full-resolution second level (8-bit target)
        {"name": "fit_512", "kind": "fit", "h": 512, "w": 512, "n": 50_000, "block": 16,
         "d0": 0.5, "d1": 4.0, "u8": False},
        {"name": "fit_2048", "kind": "fit", "h": 2048, "w": 2048, "n": 1_000_000, "block": 16,
         "d0": 0.5, "d1": 6.0, "u8": False},
        {"name": "fit_8192", "kind": "fit", "h": 8192, "w": 8192, "n": 2_000_000, "block": 16,
         "d0": 0.5, "d1": 6.0, "u8": True},
        # many uneven images fitted together
        {"name": "batch_16", "kind": "batch", "images": 16, "lo": 256, "hi": 1024,
         "density": 0.2, "block": 16, "d0": 0.5, "d1": 4.0},
        # the upscale trainer: opacities, gradient-aware render, 2x upscale
        {"name": "gatrain_512_opac", "kind": "gatrain", "h": 512, "w": 512, "n": 50_000,
         "block": 16, "d0": 0.5, "d1": 4.0, "opac": True, "up_h": 1024, "up_w": 1024},
        # gradients of project + rasterize + upscale at the density of the
        # full-scale differentiation check, on an odd size
        {"name": "gatrain_2047x1535", "kind": "gatrain", "h": 2047, "w": 1535, "n": 190_000,
         "block": 16, "d0": 0.5, "d1": 8.0, "opac": False, "up_h": 3070, "up_w": 2302},
        # a two-level fit's hand-over: the first level's gradient-aware render
        # and its 4x upscale
        {"name": "handover_2048", "kind": "handover", "h": 2048, "w": 2048, "n": 1_000_000,
         "block": 16, "d0": 0.5, "d1": 6.0, "up_h": 8192, "up_w": 8192},
        # eight queued region decodes of a resident set, crops of mixed sides
        # and scales
        {"name": "views_8", "kind": "views", "views": 8, "n": 500_000, "side": 2048,
         "lo": 256, "hi": 1536, "block": 16, "d0": 0.5, "d1": 6.0},
        # the residual target of a full-resolution level and the compose of
        # its decode, odd sizes
        {"name": "levels_4095x4093", "kind": "levels", "h": 4095, "w": 4093, "ph": 2047,
         "pw": 2046},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "train", "fit", "batch", "gatrain", "handover", "views",
                       "levels"])
    block = rng.choice([16, 16, 16, 8])
    d1 = rng.choice([4.0, 6.0, 8.0])
    if kind == "levels":
        h, w = _log_uniform(rng, 256, 4096), _log_uniform(rng, 256, 4096)
        return {"kind": kind, "h": h, "w": w, "ph": (h + 1) // 2, "pw": (w + 1) // 2}
    if kind == "batch":
        return {"kind": kind, "images": rng.randint(2, 24), "lo": 256,
                "hi": _log_uniform(rng, 400, 1024), "density": rng.uniform(0.05, 0.25),
                "block": block, "d0": 0.5, "d1": 4.0}
    if kind == "views":
        return {"kind": kind, "views": rng.randint(1, 12), "n": _log_uniform(rng, 20_000, 600_000),
                "side": 2048, "lo": 256, "hi": _log_uniform(rng, 400, 1536), "block": block,
                "d0": 0.5, "d1": d1}
    # one image: sides over the whole range, density of the configurations
    most = {"render": 4096, "train": 4096, "fit": 8192, "gatrain": 2048, "handover": 2048}[kind]
    h = _log_uniform(rng, 64, most)
    w = min(max(int(round(h * rng.uniform(0.5, 2.0))), 48), most)
    n = max(64, min(int(h * w * math.exp(rng.uniform(math.log(0.03), math.log(0.24)))), 1_200_000))
    c = {"kind": kind, "h": h, "w": w, "n": n, "block": block, "d0": 0.5, "d1": d1}
    if kind in ("render", "train"):
        c["opac"] = rng.random() < 0.4
        c["cov"] = rng.random() < 0.4
    elif kind == "fit":
        c["u8"] = rng.random() < 0.5
    else:
        s = rng.uniform(1.25, 4.0)
        c["up_h"], c["up_w"] = int(round(h * s)), int(round(w * s))
        if kind == "gatrain":
            c["opac"] = rng.random() < 0.5
    return c


# ------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV, dtype=torch.float32)


def _gaussians(g, n, h, w, d0, d1, cov=False, opac=False):
    """Gaussians of the fit configurations: means uniform over the image,
    Cholesky diagonals U[d0, d1], off-diagonal N(0, 0.5); opacities
    (sigmoid-parameterised in the trainers) U[0.05, 0.98].  Colours U(0, 1)
    over the mean overlap, so that the render lies in [0, 1] as a fit's does
    from its first iterations on."""
    p = {"means": _rand(g, n, 2) * torch.tensor([float(w), float(h)], device=DEV)}
    l = torch.stack([d0 + (d1 - d0) * _rand(g, n),
                     0.5 * torch.randn(n, generator=g, device=DEV),
                     d0 + (d1 - d0) * _rand(g, n)], 1)
    if cov:
        l = torch.stack([l[:, 0] * l[:, 0], l[:, 0] * l[:, 1],
                         l[:, 1] * l[:, 1] + l[:, 2] * l[:, 2]], 1)
    p["shape"] = l.contiguous()
    overlap = n / (h * w) * 2 * math.pi * (0.5 * (d0 + d1)) ** 2
    p["colors"] = _rand(g, n, 3) / max(1.0, overlap)
    p["opac"] = (0.05 + 0.93 * _rand(g, n)) if opac else None
    return p


def _image(g, h, w):
    """Smooth image plus noise, [h, w, 3] in [0, 1]."""
    low = _rand(g, 1, 3, max(h // 16, 2), max(w // 16, 2))
    img = F.interpolate(low, size=(h, w), mode="bicubic", align_corners=False)[0]
    img = img.permute(1, 2, 0) + 0.02 * torch.randn(h, w, 3, generator=g, device=DEV)
    return img.clamp(0, 1).contiguous()


def _target(case, g):
    img = _image(g, case["h"], case["w"])
    return (img * 255).round().to(torch.uint8) if case.get("u8") else img


def _sides(case, g, count):
    """`count` uneven (h, w): sides log-uniform in [lo, hi]."""
    u = _rand(g, count, 2).double().cpu()
    lo, hi = math.log(case["lo"]), math.log(case["hi"])
    return [(int(round(math.exp(lo + (hi - lo) * float(a)))),
             int(round(math.exp(lo + (hi - lo) * float(b))))) for a, b in u]


def _shape_seed(case):
    """Sizes inside a case are the same for every seed of it."""
    return 77 + case.get("images", 0) + 31 * case.get("views", 0)


def _batch_inputs(case, seed):
    g = _gen(seed)
    targets, init = [], []
    for h, w in _sides(case, _gen(_shape_seed(case)), case["images"]):
        n = max(1, int(round(case["density"] * h * w)))
        targets.append(_image(g, h, w))
        init.append(_gaussians(g, n, h, w, case["d0"], case["d1"]))
    return targets, init


def _view_inputs(case, seed):
    side = case["side"]
    p = _gaussians(_gen(seed), case["n"], side, side, case["d0"], case["d1"])
    sg = _gen(_shape_seed(case))
    views = []
    for (h, w), u in zip(_sides(case, sg, case["views"]), _rand(sg, case["views"], 3).cpu()):
        s = float(0.25 * 8.0 ** float(u[2]))  # scale log-uniform in [0.25, 2]
        ox = float(u[0]) * max(side - w / s, 0.0)
        oy = float(u[1]) * max(side - h / s, 0.0)
        views.append((h, w, (ox, oy), (s, s)))
    return p, views


def _level_inputs(case, seed):
    g = _gen(seed)
    gt = _image(g, case["h"], case["w"])
    up = (gt + 0.05 * torch.randn(gt.shape, generator=g, device=DEV)).clamp(0, 1).contiguous()
    return gt, up, _image(g, case["ph"], case["pw"]), _image(g, case["h"], case["w"])


def _train_inputs(case, seed):
    g = _gen(seed)
    p = _gaussians(g, case["n"], case["h"], case["w"], case["d0"], case["d1"],
                   case.get("cov", False), case.get("opac", False))
    if case["kind"] in ("train", "fit"):
        return p, _target(case, g)
    if case["kind"] == "gatrain":
        return p, _image(g, case["up_h"], case["up_w"])
    return p, None


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        targets, init = _batch_inputs(case, seed)
        init = [(p["means"], p["shape"], p["colors"]) for p in init]
        fit = BatchedFit(targets, [i[0].shape[0] for i in init], block=case["block"], init=init)
        return {"case": case, "fit": fit}
    if kind == "views":
        p, views = _view_inputs(case, seed)
        gs = GaussianSet(p["means"], p["shape"], p["colors"], case["side"], case["side"])
        return {"case": case, "views": [(gs, *v) for v in views]}
    if kind == "levels":
        return {"case": case, "in": _level_inputs(case, seed)}
    p, target = _train_inputs(case, seed)
    if kind == "fit":
        fit = LevelFit(case["n"], case["h"], case["w"], device=DEV, block=case["block"],
                       diag=(case["d0"], case["d1"]))
        with torch.no_grad():
            fit.means.copy_(p["means"])
            fit.chol.copy_(p["shape"])
            fit.rgbs.copy_(p["colors"])
        return {"case": case, "fit": fit, "target": target}
    if kind in ("train", "gatrain"):
        for k, t in p.items():
            if t is not None:
                p[k] = t.requires_grad_()
    return {"case": case, "p": p, "target": target}


# ---------------------------------------------------------------------- run
def _rasterize(case, p, grad_aware=False):
    project = (gsplat2d.project_gaussians if case.get("cov")
               else gsplat2d.project_gaussians_cholesky)
    h, w, b = case["h"], case["w"], case["block"]
    xys, ext, con, cnt = project(p["shape"], p["means"], h, w, b, p["opac"])
    return gsplat2d.rasterize_gaussians(xys, ext, con, cnt, p["colors"], p["opac"], h, w, b,
                                        compute_upscale_gradients=grad_aware)


def _gradients(loss, p):
    params = {k: t for k, t in p.items() if t is not None}
    for t in params.values():
        t.grad = None
    loss.backward()
    return {"loss": loss.detach(), **{k: t.grad for k, t in params.items()}}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "render":
        with torch.no_grad():
            img, wsum = _rasterize(case, state["p"])[:2]
        return {"img": img, "wsum": wsum}
    if kind == "train":
        p = state["p"]
        img = torch.clamp(_rasterize(case, p)[0], 0, 1)
        return _gradients(F.mse_loss(img, state["target"]), p)
    if kind == "gatrain":
        p = state["p"]
        img, _, dx, dy, dxy = _rasterize(case, p, grad_aware=True)
        up = gsplat2d.gradient_aware_upscale(img, dx, dy, dxy, case["up_h"], case["up_w"])
        return _gradients(F.mse_loss(up, state["target"]), p)
    if kind == "handover":
        with torch.no_grad():
            img, wsum, dx, dy, dxy = _rasterize(case, state["p"], grad_aware=True)
            up = gsplat2d.gradient_aware_upscale(img, dx, dy, dxy, case["up_h"], case["up_w"])
        return {"img": img, "wsum": wsum, "dx": dx, "dy": dy, "dxy": dxy, "up": up}
    if kind == "fit":
        fit = state["fit"]
        loss = fit.step(state["target"])
        return {"loss": loss, "means": fit.means, "shape": fit.chol, "colors": fit.rgbs}
    if kind == "batch":
        fit = state["fit"]
        fit.step_checked()
        return {"loss": fit.loss, "per_image": fit.per_image, "grad": fit.grad, "flat": fit.flat}
    if kind == "views":
        return render_views(state["views"], block=case["block"])
    gt, up, prev, render = state["in"]
    target, lo, hi = residual_target(gt, up)
    return {"target": target, "lo": lo, "hi": hi, "out": compose(prev, render, lo, hi, True)}


# --------------------------------------------------------------------- work
def _pixels_reached(case, scale2=1.0):
    """Mean pixels of a Gaussian's alpha >= 1/255 ellipse, opacity 1 or
    averaged over the opacities' range: pi t sqrt(det cov)."""
    m = 0.5 * (case["d0"] + case["d1"])
    t = 2 * LOG_255
    if case.get("opac"):
        t = 2 * (LOG_255 - 0.72)
    return math.pi * t * m * m * scale2


def work(case):
    """Bytes: parameters, targets and results once each (fp32 unless the case
    says otherwise).  Flops: the per-pixel expressions of the forward (20, or
    49 gradient-aware) and the backward (40 / 110) over the pixels that each
    Gaussian reaches."""
    kind = case["kind"]
    if kind == "levels":
        px, prev = case["h"] * case["w"] * 3, case["ph"] * case["pw"] * 3
        return {"bytes": 4 * (2 * px + px + prev + px + px), "flops": 20 * px}
    if kind == "batch":
        px = sum(h * w for h, w in _sides(case, _gen(_shape_seed(case)), case["images"]))
        n = case["density"] * px
        return {"bytes": 4 * (n * 8 * 7 + px * 3), "flops": 60 * n * _pixels_reached(case)}
    if kind == "views":
        px, flops = 0, 0.0
        for h, w, _, (s, _) in _view_inputs(dict(case, n=1), 0)[1]:
            px += h * w
            inside = min(1.0, h / s / case["side"]) * min(1.0, w / s / case["side"])
            flops += 20 * case["n"] * inside * _pixels_reached(case, s * s)
        return {"bytes": 4 * (case["n"] * 8 * case["views"] + px * 3), "flops": flops}
    px, n = case["h"] * case["w"], case["n"]
    per = 8 + (1 if case.get("opac") else 0)
    pairs = n * _pixels_reached(case)
    if kind == "render":
        return {"bytes": 4 * (n * per + px * 4), "flops": 20 * pairs}
    if kind == "train":
        return {"bytes": 4 * (n * per * 2 + px * 3), "flops": 60 * pairs}
    if kind == "fit":
        # parameters and both moments read and written
        return {"bytes": 4 * n * 8 * 6 + px * 3 * (1 if case["u8"] else 4), "flops": 60 * pairs}
    up = case["up_h"] * case["up_w"]
    if kind == "gatrain":
        return {"bytes": 4 * (n * per * 2 + up * 3), "flops": 159 * pairs + 2 * 100 * up}
    return {"bytes": 4 * (n * per + px * 13 + up * 3), "flops": 49 * pairs + 100 * up}


# -------------------------------------------------------------------- exact
def _conics64(p):
    """(a, b, c) of the inverse covariance, and the covariance's diagonal."""
    s = p["shape"]
    if p.get("is_cov"):
        cx, cy, cz = s[:, 0], s[:, 1], s[:, 2]
    else:
        cx, cy = s[:, 0] * s[:, 0], s[:, 0] * s[:, 1]
        cz = s[:, 1] * s[:, 1] + s[:, 2] * s[:, 2]
    det = cx * cz - cy * cy
    return cz / det, -cy / det, cx / det, cx, cz


def _splat64(p, h, w, clamp, grad_aware, chunk):
    """Yields, per chunk of Gaussians, (pixel indices, list of [K, D, C]
    contributions to each plane) of every pixel whose alpha is at least
    1/255; chunks are grouped by window size."""
    with torch.no_grad():
        _, _, _, cx, cz = _conics64(p)
        o = p["opac"] if p["opac"] is not None else torch.ones_like(cx)
        t = 2 * torch.log(255 * o).clamp_min(0)
        r = torch.maximum((t * cx).sqrt(), (t * cz).sqrt()).ceil().long() + 1
        order = torch.argsort(r)
        rs = r[order].cpu()
    n, i0 = order.numel(), 0
    while i0 < n:
        k = max(1, min(n - i0, chunk // int(2 * rs[i0] + 1) ** 2))
        rad = int(rs[i0 + k - 1])
        if k * (2 * rad + 1) ** 2 > 2 * chunk and k > 1:
            k = max(1, k // 2)
            rad = int(rs[i0 + k - 1])
        sel = order[i0:i0 + k]
        i0 += k
        q = {key: (v[sel] if torch.is_tensor(v) else v) for key, v in p.items()}
        a, b, c, _, _ = _conics64(q)
        mx, my = q["means"][:, 0], q["means"][:, 1]
        d = torch.arange(-rad, rad + 1, device=DEV)
        gx = mx.detach().floor().long()[:, None, None] + d[None, None, :]
        gy = my.detach().floor().long()[:, None, None] + d[None, :, None]
        dx = gx.double() + 0.5 - mx[:, None, None]
        dy = gy.double() + 0.5 - my[:, None, None]
        a, b, c = (v[:, None, None] for v in (a, b, c))
        sigma = 0.5 * (a * dx * dx + c * dy * dy) + b * dx * dy
        alpha = torch.exp(-sigma)
        if q["opac"] is not None:
            alpha = q["opac"][:, None, None] * alpha
        with torch.no_grad():
            keep = (alpha >= 1.0 / 255) & (gx >= 0) & (gx < w) & (gy >= 0) & (gy < h)
            # the clamp scales alpha without a derivative of its own
            ratio = torch.where(keep, (clamp / alpha).clamp(max=1.0), 0.0)
            pix = (gy.clamp(0, h - 1) * w + gx.clamp(0, w - 1)).reshape(-1)
        alpha = alpha * ratio
        planes = [alpha]
        if grad_aware:
            sx, sy = a * dx + b * dy, b * dx + c * dy
            planes += [-alpha * sx, -alpha * sy, alpha * (sx * sy - b)]
        yield q["colors"], pix, [v.reshape(k, -1) for v in planes]


def _render64(p, h, w, grad_aware=False, chunk=6_000_000):
    """[img, (dx, dy, dxy)], wsum in 64 bits."""
    outs = [torch.zeros(h * w, 3, dtype=torch.float64, device=DEV)
            for _ in range(4 if grad_aware else 1)]
    wsum = torch.zeros(h * w, dtype=torch.float64, device=DEV)
    with torch.no_grad():
        for colors, pix, planes in _splat64(p, h, w, 0.999, grad_aware, chunk):
            wsum.index_add_(0, pix, planes[0].reshape(-1))
            for out, v in zip(outs, planes):
                out.index_add_(0, pix, (v[:, :, None] * colors[:, None, :]).reshape(-1, 3))
    return [o.view(h, w, 3) for o in outs], wsum.view(h, w)


def _backward64(p, h, w, cots, clamp, chunk=3_000_000):
    """Gradients of sum(plane * cotangent) over the planes for every
    parameter (the render is a sum over Gaussians, so chunks add up)."""
    leaves = {k: v.detach().clone().requires_grad_() for k, v in p.items() if torch.is_tensor(v)}
    q = {**p, **leaves}
    flat = [c.reshape(-1, 3) for c in cots]
    for colors, pix, planes in _splat64(q, h, w, clamp, len(cots) > 1, chunk):
        total = 0.0
        for v, c in zip(planes, flat):
            cot = c[pix].view(v.shape[0], v.shape[1], 3)
            total = total + (v * torch.einsum("kc,kdc->kd", colors, cot)).sum()
        total.backward()
    return {k: v.grad for k, v in leaves.items()}


def _double(p, case):
    q = {k: (None if t is None else t.double()) for k, t in p.items()}
    q["is_cov"] = bool(case.get("cov"))
    return q


def _l2_64(img, target):
    """Loss and its cotangent for mean((clamp(img) - target)^2)."""
    d = img.clamp(0, 1) - target
    cot = torch.where((img >= 0) & (img <= 1), d, 0.0) * (2.0 / d.numel())
    return (d * d).mean(), cot


def _upscale64(planes, up_h, up_w):
    """Half-pixel Hermite bicubic of the four planes [h, w, 3]."""
    def axis(dst, src):
        s = (torch.arange(dst, device=DEV, dtype=torch.float64) + 0.5) * src / dst - 0.5
        f = s.floor()
        t = s - f
        i0 = f.long().clamp(0, src - 1)
        i1 = (f.long() + 1).clamp(0, src - 1)
        t2, t3 = t * t, t * t * t
        return i0, i1, (1 - 3 * t2 + 2 * t3, 3 * t2 - 2 * t3, t - 2 * t2 + t3, t3 - t2)

    img, dx, dy, dxy = planes
    y0, y1, wy = axis(up_h, img.shape[0])
    x0, x1, wx = axis(up_w, img.shape[1])
    wy = [v.view(-1, 1, 1) for v in wy]
    wx = [v.view(1, -1, 1) for v in wx]
    val = img[y0] * wy[0] + img[y1] * wy[1] + dy[y0] * wy[2] + dy[y1] * wy[3]
    der = dx[y0] * wy[0] + dx[y1] * wy[1] + dxy[y0] * wy[2] + dxy[y1] * wy[3]
    return val[:, x0] * wx[0] + val[:, x1] * wx[1] + der[:, x0] * wx[2] + der[:, x1] * wx[3]


def _adam64(param, grad, lr=1e-3, b1=0.9, b2=0.999, eps=1e-8):
    """First Adam step from zero moments."""
    m, v = (1 - b1) * grad, (1 - b2) * grad * grad
    return param - lr * (m / (1 - b1)) / ((v / (1 - b2)).sqrt() + eps)


def _fit_step64(p, target, h, w):
    img = _render64(p, h, w)[0][0]
    t = target.double() / 255 if target.dtype == torch.uint8 else target.double()
    loss, cot = _l2_64(img, t)
    # the sum backward clamps alpha at 0.99 (its forward at 0.999)
    return loss, _backward64(p, h, w, [cot], 0.99)


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        targets, init = _batch_inputs(case, seed)
        losses, grads, flats = [], [], []
        for t, p in zip(targets, init):
            p = _double(p, case)
            loss, g = _fit_step64(p, t, t.shape[0], t.shape[1])
            losses.append(loss)
            grads.append(g)
            flats.append({k: _adam64(p[k], g[k]) for k in g})
        cat = lambda ds: torch.cat([d[k].reshape(-1) for k in ("means", "shape", "colors")  # noqa: E731
                                    for d in ds])
        return {"loss": sum(losses), "per_image": torch.stack(losses), "grad": cat(grads),
                "flat": cat(flats)}
    if kind == "views":
        p, views = _view_inputs(case, seed)
        outs = []
        for h, w, (ox, oy), (s, _) in views:
            q = _double(p, case)
            q["means"] = (q["means"] - torch.tensor([ox, oy], device=DEV, dtype=torch.float64)) * s
            q["shape"] = q["shape"] * s
            m, reach = q["means"], 4.0 * q["shape"].abs().sum(1) + 4
            near = ((m[:, 0] > -reach) & (m[:, 0] < w + reach) & (m[:, 1] > -reach)
                    & (m[:, 1] < h + reach))
            q = {k: (v[near] if torch.is_tensor(v) else v) for k, v in q.items()}
            outs.append(_render64(q, h, w)[0][0])
        return outs
    if kind == "levels":
        gt, up, prev, render = (t.double() for t in _level_inputs(case, seed))
        r = gt - up + 0.5
        lo, hi = r.min(), r.max()
        base = F.interpolate(prev.permute(2, 0, 1)[None], size=(case["h"], case["w"]),
                             mode="bilinear", align_corners=False)[0].permute(1, 2, 0)
        out = base + (render.clamp(0, 1) * (hi - lo) - 0.5 + lo)
        return {"target": (r - lo) / (hi - lo), "lo": lo, "hi": hi, "out": out.clamp(0, 1)}
    p, target = _train_inputs(case, seed)
    p = _double(p, case)
    h, w = case["h"], case["w"]
    if kind == "render":
        planes, wsum = _render64(p, h, w)
        return {"img": planes[0], "wsum": wsum}
    if kind == "train":
        loss, g = _fit_step64(p, target, h, w)
        return {"loss": loss, **g}
    if kind == "fit":
        loss, g = _fit_step64(p, target, h, w)
        return {"loss": loss, **{k: _adam64(p[k], g[k]) for k in g}}
    planes, wsum = _render64(p, h, w, grad_aware=True)
    if kind == "handover":
        return {"img": planes[0], "wsum": wsum, "dx": planes[1], "dy": planes[2],
                "dxy": planes[3], "up": _upscale64(planes, case["up_h"], case["up_w"])}
    planes = [t.requires_grad_() for t in planes]
    loss = F.mse_loss(_upscale64(planes, case["up_h"], case["up_w"]), target.double())
    loss.backward()
    g = _backward64(p, h, w, [t.grad for t in planes], 0.999)
    # the gradient-aware backward's opacity gradient leaves out the derivative
    # planes (the reference's own rule): no 64-bit value is stated for it
    g = {k: (None if k == "opac" else v) for k, v in g.items()}
    return {"loss": loss.detach(), **g}
