"""Workloads of the splatting framework, through its public entry points.

Kinds of case:
  step      one training iteration as the trainer runs it: forward, fused
            L1 + SSIM loss, backward with the fused structure Adam and the
            quantized SH Adam (Rasterizer.forward / fused_l1_ssim /
            Rasterizer.backward); optimiser state of a run in progress
  grads     the differentiable render (rasterize_gaussians) and its gradients,
            for a caller with an optimiser of its own
  render    inference: one view, no backward state
  geometry  training forward with the median-depth and normal channels and the
            backward of colour, alpha, depth and normal gradients
  batch     many views of uneven resolution, forward and backward replayed
            from one captured graph (BatchRasterizer)
  loss      compute_training_loss with every term
  prune     Speedy-Splat pruning scores of one view

Scenes have the distributions of photara-studio_b200/scenes.py (means uniform
in a box in front of the camera, log-scales N(-3.5, 0.5), normalised
quaternions, opacity logits N(0, 1), SH with DC N(0, 0.3) and the rest
N(0, 0.05)), drawn on the GPU from the seed.

`exact` restates the paths in float64 torch: projection, SH colour and the
blend of every block of pixels, differentiated by autograd.
"""
from __future__ import annotations

import importlib
import math

import numpy as np
import torch

gsb = importlib.import_module("photara-studio_b200")
batch = importlib.import_module("photara-studio_b200.batch")

STEP = 500  # iteration the optimiser state belongs to (bias corrections)
BETA1, BETA2 = float(np.float32(0.9)), float(np.float32(0.999))
ADAM_EPS, SH_EPS, CODEC_EPS = 1e-15, 1e-8, 1e-15
LRS = dict(means_lr=1.6e-4, scales_lr=5e-3, quaternions_lr=1e-3, opacities_lr=5e-2)
SH_LR, SH_REST_LR = 5e-3, 1.25e-4
LOSS_OPTIONS = dict(photometric_weight=0.8, ssim_weight=0.3, depth_weight=0.3, normal_weight=0.2,
                    depth_normal_weight=0.05, alpha_mode="transparent", ai_prior=True)


# ------------------------------------------------------------------ cases --
def _case(name, kind, n, w, h, f, half, z_lo, z_hi, degree=3, kernel=0.0, views=1):
    c = {"kind": kind, "n": n, "w": w, "h": h, "f": float(f), "half": float(half),
         "z_lo": float(z_lo), "z_hi": float(z_hi), "degree": degree, "kernel": kernel,
         "views": views}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a small capture or an interactive preview being trained: latency and launches
        _case("step_16k_256", "step", 16384, 256, 256, 256, 1, 2, 6),
        # the early phase of a run, before densification has grown the model
        _case("step_131k_640x480", "step", 131072, 640, 480, 500, 4, 2, 12),
        # the ordinary training step at full HD: the framework's headline workload
        _case("step_1m_1080p", "step", 1048576, 1920, 1080, 1500, 4, 2, 12),
        # a large scene at 4K
        _case("step_8m_2160p", "step", 8388608, 3840, 2160, 3000, 8, 2, 30),
        # own optimiser, sizes that divide by nothing, SH degree 1 while colours warm up
        _case("grads_20k_odd", "grads", 20011, 319, 243, 301, 1, 2, 6, degree=1, kernel=0.1),
        # own optimiser at an ordinary odd size, SH degree 2
        _case("grads_300k_odd", "grads", 300007, 1237, 823, 1001, 4, 2, 12, degree=2),
        # viewer frame: the size of the reference's published render timings
        _case("render_213k_1000", "render", 213003, 1000, 1000, 900, 4, 2, 12),
        # evaluation renders of a trained model at full HD
        _case("render_1m_1080p", "render", 1048576, 1920, 1080, 1500, 4, 2, 12),
        # geometry-regularised training of a surface model
        _case("geometry_500k_720p", "geometry", 500000, 1280, 720, 1000, 4, 2, 12),
        # multi-view step: eight ring views of uneven resolution over one model
        _case("batch_8x500k", "batch", 500000, 1920, 1080, 0.5, 2, 0, 0, views=8),
        # the training loss of one full-HD view
        _case("loss_1080p", "loss", 1, 1920, 1080, 1700, 1, 1, 2),
        # pruning pass over one training view
        _case("prune_500k_720p", "prune", 500000, 1280, 720, 1000, 4, 2, 12),
    ]


def draw(rng):
    kind = rng.choices(["step", "grads", "render", "geometry", "batch", "loss", "prune"],
                       [5, 2, 2, 1, 1, 1, 1])[0]
    log_uniform = lambda a, b: int(math.exp(rng.uniform(math.log(a), math.log(b))))
    top_w, top_n = {"step": (1920, 1500000), "grads": (1920, 800000), "render": (1920, 1500000),
                    "geometry": (1280, 300000), "batch": (1280, 300000), "loss": (1920, 2),
                    "prune": (1280, 500000)}[kind]
    w = log_uniform(64, top_w)
    h = max(48, int(w * rng.uniform(0.5, 1.0)))
    n = log_uniform(1 if kind == "loss" else 500, top_n)
    half, z_lo, z_hi = (1, 2, 6) if n < 65536 else (4, 2, 12)
    degree = rng.choice([3, 3, 3, 2, 1, 0]) if kind in ("grads", "render") else 3
    kernel = rng.choice([0.0, 0.0, 0.1]) if kind != "loss" else 0.0
    if kind == "batch":
        return _case(None, kind, n, w, h, rng.uniform(0.4, 0.6), 2, 0, 0, degree=degree,
                     kernel=kernel, views=rng.randint(2, 6))
    return _case(None, kind, n, w, h, w * rng.uniform(0.7, 1.1), half, z_lo, z_hi, degree=degree,
                 kernel=kernel)


# ----------------------------------------------------------------- inputs --
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _model(case, g):
    n = case["n"]
    u = lambda *s: torch.rand(s, device="cuda", generator=g)
    r = lambda *s: torch.randn(s, device="cuda", generator=g)
    if case["kind"] == "batch":
        means = (2 * u(n, 3) - 1) * case["half"]
    else:
        means = torch.cat([(2 * u(n, 2) - 1) * case["half"],
                           case["z_lo"] + (case["z_hi"] - case["z_lo"]) * u(n, 1)], dim=1)
    q = r(n, 4)
    sh = 0.05 * r(n, 16, 3)
    sh[:, 0] = 0.3 * r(n, 3)
    return gsb.GaussianModel(means.contiguous(), -3.5 + 0.5 * r(n, 3),
                             (q / q.norm(dim=1, keepdim=True)).contiguous(), r(n, 1), sh, 3)


def _cameras(case):
    if case["kind"] != "batch":
        identity = [1.0, 0, 0, 0, 0, 1.0, 0, 0, 0, 0, 1.0, 0, 0, 0, 0, 1.0]
        return [gsb.Camera(identity, [0.0, 0.0, 0.0], case["f"], case["f"], case["w"] / 2,
                           case["h"] / 2, case["w"], case["h"])]
    cams = []
    for k in range(case["views"]):  # four resolutions in turn, down to a third of the largest
        w = max(64, case["w"] * (6 - k % 4 - (k % 4 > 1)) // 6)
        h = max(48, case["h"] * (6 - k % 4 - (k % 4 > 1)) // 6)
        a = 2 * math.pi * k / case["views"]
        cams.append(gsb.look_at_camera((6 * math.cos(a), 0.5, 6 * math.sin(a)), (0, 0, 0),
                                       (0, 1, 0), w, h, case["f"] * w))
    return cams


def _options(case, **kw):
    return gsb.RasterizeOptions(active_sh_degree=case["degree"], kernel_size=case["kernel"],
                                background=(0.1, 0.2, 0.3), **kw)


def _photo(case, g):
    """A photograph-like target: smooth colour, fine texture."""
    h, w = case["h"], case["w"]
    coarse = torch.rand((1, 3, h // 24 + 2, w // 24 + 2), device="cuda", generator=g)
    img = torch.nn.functional.interpolate(coarse, (h, w), mode="bilinear", align_corners=False)[0]
    return (img + 0.05 * torch.randn((3, h, w), device="cuda", generator=g)).clamp(0, 1)


def _adam(model, g):
    """Moments of a run in progress: updates of about a third of a step."""
    def pair(p, scale):
        second = scale * scale * torch.exp(torch.randn(p.shape, device="cuda", generator=g))
        first = 0.3 * second.sqrt() * torch.randn(p.shape, device="cuda", generator=g)
        return first, second
    s = {}
    for name, p, scale in (("means", model.means, 1e-6), ("scales", model.log_scales, 1e-7),
                           ("rotations", model.quaternions, 1e-7),
                           ("opacity", model.opacity_logits, 1e-7)):
        s[name + "_first"], s[name + "_second"] = pair(p, scale)
    n = model.size()
    lo = 18 + torch.rand((n, 2), device="cuda", generator=g)  # log(sqrt(v) / 1e-15)
    hi = lo + 2 * torch.rand((n, 2), device="cuda", generator=g) + 0.1
    sh = dict(first=(0.3 * torch.randn((n, 16, 3), device="cuda", generator=g)).half(),
              packed=torch.randint(0, 256, (n, 16, 3), device="cuda", generator=g,
                                   dtype=torch.uint8),
              bounds=torch.stack([lo[:, 0], hi[:, 0], lo[:, 1], hi[:, 1]], 1).contiguous())
    return s, sh


def _loss_images(case, g):
    h, w = case["h"], case["w"]
    u = lambda *s: torch.rand(s, device="cuda", generator=g)
    r = lambda *s: torch.randn(s, device="cuda", generator=g)
    yy, xx = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"),
                            indexing="ij")
    depth = 2.0 + 0.01 * xx + 0.02 * yy + 0.05 * u(h, w)
    depth[u(h, w) < 0.03] = 0.0
    normal = r(3, h, w)
    target_normal = r(3, h, w)
    target_normal[:, u(h, w) < 0.2] = 0.0
    target = _photo(case, g)
    return dict(color=(target + 0.05 * r(3, h, w)).clamp(0, 1), target_color=target,
                alpha=0.01 + 0.98 * u(h, w), median_depth=depth,
                normal=(normal / normal.norm(dim=0, keepdim=True)).contiguous(),
                target_depth=torch.where(u(h, w) < 0.85, depth + 0.1 * r(h, w),
                                         0.0).contiguous(),
                target_normal=target_normal, mask=(u(h, w) > 0.25).float())


def _image_grads(case, cams, g):
    """Gradients of the size a mean loss gives, with respect to every channel."""
    r = lambda *s: 1e-3 * torch.randn(s, device="cuda", generator=g)
    if case["kind"] == "batch":
        pixels = sum(c.width * c.height for c in cams)
        return dict(color=r(3 * pixels))
    h, w = case["h"], case["w"]
    out = dict(color=r(3, h, w), alpha=r(h, w))
    if case["kind"] == "geometry":
        out.update(depth=r(h, w), normal=r(3, h, w))
    return out


def prepare(case, seed):
    g = _gen(seed)
    kind = case["kind"]
    if kind == "loss":
        return {"case": case, "images": _loss_images(case, g), "camera": _cameras(case)[0],
                "options": gsb.TrainingLossOptions(**LOSS_OPTIONS)}
    model, cams = _model(case, g), _cameras(case)
    s = {"case": case, "model": model, "camera": cams[0], "rasterizer": gsb.Rasterizer()}
    if kind == "step":
        s["target"] = _photo(case, g)
        s["structure"], s["sh"] = _adam(model, g)
        s["step"] = STEP
        s["options"] = _options(case)
    elif kind == "grads":
        s["grads"] = _image_grads(case, cams, g)
        s["params"] = [p.requires_grad_() for p in (model.means, model.log_scales,
                                                    model.quaternions, model.opacity_logits,
                                                    model.sh)]
        s["options"] = _options(case)
    elif kind == "render":
        s["options"] = _options(case, record_backward_state=False)
    elif kind == "geometry":
        s["grads"] = _image_grads(case, cams, g)
        s["options"] = _options(case, require_depth=True)
    elif kind == "prune":
        s["options"] = _options(case)
    elif kind == "batch":
        s["grads"] = _image_grads(case, cams, g)
        br = batch.BatchRasterizer()
        br.plan(model, cams, _options(case), batch.BatchSchedule(16, 32, 4, "heavy_first"))
        br.capture(s["grads"]["color"])
        s["batch"] = br
    return s


def _corrections(step):
    return 1 - 0.9 ** step, 1 - 0.999 ** step


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "loss":
        im = s["images"]
        g = gsb.compute_training_loss(im["color"], im["target_color"], alpha=im["alpha"],
                                      median_depth=im["median_depth"], normal=im["normal"],
                                      target_depth=im["target_depth"],
                                      target_normal=im["target_normal"], mask=im["mask"],
                                      camera=s["camera"], options=s["options"],
                                      need_geometry_gradients=True)
        return {"color": g.color, "alpha": g.alpha, "depth": g.depth, "normal": g.normal,
                "terms": g.terms}
    model, cam, rast = s["model"], s["camera"], s["rasterizer"]
    if kind == "step":
        s["step"] += 1
        c1, c2 = _corrections(s["step"])
        r = rast.forward(model, cam, s["options"])
        loss, grad = gsb.fused_l1_ssim(r.color, s["target"])
        sa = gsb.StructureAdamUpdate(**s["structure"], **LRS, correction1=c1, correction2=c2)
        sh = gsb.SHAdamUpdate(**s["sh"], lr=SH_LR, rest_lr=SH_REST_LR, correction1=c1,
                              correction2=c2)
        grads = rast.backward(model, r, grad, None, sh_adam=sh, structure_adam=sa)
        return {"color": r.color, "alpha": r.alpha, "radii": r.radii,
                "visibility": r.visibility, "loss": loss,
                "means": model.means, "log_scales": model.log_scales,
                "quaternions": model.quaternions, "opacity_logits": model.opacity_logits,
                "sh": model.sh, **s["structure"], "sh_first": s["sh"]["first"],
                "sh_packed": s["sh"]["packed"], "sh_bounds": s["sh"]["bounds"],
                "refine_weight": grads.refine_weight}
    if kind == "grads":
        color, alpha, radii = gsb.rasterize_gaussians(*s["params"], cam, s["options"])
        g = torch.autograd.grad([color, alpha], s["params"],
                                [s["grads"]["color"], s["grads"]["alpha"]])
        return {"color": color.detach(), "alpha": alpha.detach(), "radii": radii, "means": g[0],
                "log_scales": g[1], "quaternions": g[2], "opacity_logits": g[3], "sh": g[4]}
    if kind == "render":
        r = rast.forward(model, cam, s["options"])
        return {"color": r.color, "alpha": r.alpha, "radii": r.radii, "visibility": r.visibility}
    if kind == "geometry":
        r = rast.forward(model, cam, s["options"])
        gi = s["grads"]
        g = rast.backward(model, r, gi["color"], gi["alpha"], grad_depth=gi["depth"],
                          grad_normal=gi["normal"])
        return {"color": r.color, "alpha": r.alpha, "median_depth": r.median_depth,
                "normal": r.normal, "radii": r.radii, "means": g.means,
                "log_scales": g.log_scales, "quaternions": g.quaternions,
                "opacity_logits": g.opacity_logits, "sh": g.sh,
                "refine_weight": g.refine_weight}
    if kind == "prune":
        return {"scores": rast.pruning_scores(model, cam, s["options"])}
    res = s["batch"].replay()
    g = s["batch"].grads
    return {"color": res.color, "alpha": res.alpha, "radii": res.radii, "means": g.means,
            "log_scales": g.log_scales, "quaternions": g.quaternions,
            "opacity_logits": g.opacity_logits, "sh": g.sh, "refine_weight": g.refine_weight}


# ------------------------------------------------------------------- work --
def _pairs(case):
    """Expected (Gaussian, pixel) pairs that are blended in one view: mean
    overlap of the visible footprints per pixel, at most the hundred or so
    that saturate a pixel of these scenes."""
    if case["kind"] == "batch":
        z, f = 6.0, case["f"] * case["w"]
        seen = case["n"]
    else:
        z, f = 0.5 * (case["z_lo"] + case["z_hi"]), case["f"]
        reach = min(1.0, 0.5 * case["w"] * z / f / case["half"]) * \
            min(1.0, 0.5 * case["h"] * z / f / case["half"])
        seen = case["n"] * reach
    area = math.pi * 6.0 * (f * math.exp(-3.5) / z) ** 2
    pixels = case["w"] * case["h"]
    return pixels * min(100.0, seen * area / pixels), seen


def work(case):
    px = case["w"] * case["h"]
    n, kind = case["n"], case["kind"]
    if kind == "loss":
        # 13 image planes in, 8 gradient planes out; two 11-tap separable passes
        # over the moments and over the derivative maps of each channel
        return {"bytes": 4.0 * px * (13 + 8), "flops": 3.0 * px * (4 * 11 * 5 + 4 * 11 * 3 + 60)}
    pairs, seen = _pairs(case)
    sh_floats = 3 * (case["degree"] + 1) ** 2
    params = 11 * 4 * n + 4 * sh_floats * seen
    images = 16.0 * px
    forward_flops = 20.0 * pairs + 400.0 * seen
    if kind == "render":
        return {"bytes": params + images + 8.0 * n, "flops": forward_flops}
    if kind == "prune":
        return {"bytes": params + 4.0 * n, "flops": forward_flops + 25.0 * pairs}
    if kind == "step":
        state = n * 2 * (59 * 4 + 88 + 96 + 48 + 16)  # parameters, moments, codec: in and out
        return {"bytes": state + images + 12.0 * px + 12.0 * n,
                "flops": 80.0 * pairs + 2000.0 * n + 3.0 * px * (4 * 11 * 5 + 4 * 11 * 3)}
    if kind == "batch":
        # mean pixels per view of the four resolutions
        share = [((6 - k % 4 - (k % 4 > 1)) / 6.0) ** 2 for k in range(case["views"])]
        scale = sum(share)
        return {"bytes": params + 2 * 59 * 4 * n + 4.0 * n * case["views"] + 28.0 * px * scale,
                "flops": (80.0 * pairs * scale + 1000.0 * seen * case["views"])}
    grads = 4.0 * n * 59
    if kind == "grads":
        return {"bytes": params + grads + images + 16.0 * px + 4.0 * n,
                "flops": 80.0 * pairs + 1000.0 * seen}
    # geometry: five bisection walks and the slope walk beside the two colour walks
    return {"bytes": params + grads + 32.0 * px + 32.0 * px + 8.0 * n,
            "flops": (80.0 + 6 * 25.0 + 60.0) * pairs + 1500.0 * seen}


def tolerance(case):
    """About four times the distance to `exact` over listed and drawn cases. A
    rounding that moves an opacity across 1/255 or a transmittance across 1e-4
    changes that pixel's blend: colours 2e-5 off in all, gradients (many terms
    that cancel) 2e-4 to 4e-4, first moments 1.5e-4 after one step. Moment
    codes are rounded: one in a million flips when gradients are summed in
    another order (one of the 24,000 codes of the smallest drawn model)."""
    kind = case["kind"]
    if kind in ("render", "prune"):
        return {"rel": 1e-4}
    if kind == "loss":
        return {"rel": 5e-5}
    return {"rel": 1e-3, "differ": 1e-4}


# ---------------------------------------------------------- 64-bit restatement --
SH_C = (0.28209479177387814, 0.4886025119029199,
        (1.0925484305920792, -1.0925484305920792, 0.31539156525252005, -1.0925484305920792,
         0.5462742152960396),
        (-0.5900435899266435, 2.890611442640554, -0.4570457994644658, 0.3731763325901154,
         -0.4570457994644658, 1.445305721320277, -0.5900435899266435))


def _sh_basis(d, degree):
    x, y, z = d.unbind(1)
    b = [torch.full_like(x, SH_C[0])]
    if degree > 0:
        b += [-SH_C[1] * y, SH_C[1] * z, -SH_C[1] * x]
    if degree > 1:
        q = (x * y, y * z, 2 * z * z - x * x - y * y, x * z, x * x - y * y)
        b += [c * v for c, v in zip(SH_C[2], q)]
    if degree > 2:
        xx, yy, zz = x * x, y * y, z * z
        q = (y * (3 * xx - yy), x * y * z, y * (4 * zz - xx - yy),
             z * (2 * zz - 3 * xx - 3 * yy), x * (4 * zz - xx - yy), z * (xx - yy),
             x * (xx - 3 * yy))
        b += [c * v for c, v in zip(SH_C[3], q)]
    return torch.stack(b, 1)


def _project(p, cam, case):
    """Screen-space Gaussians of float64 parameters (differentiable)."""
    means, log_scales, quats, logits, sh = p
    dev = means.device
    V = torch.tensor(cam.world_to_camera, dtype=torch.float32, device=dev).double().view(4, 4).T
    eye = torch.tensor(cam.position, dtype=torch.float32, device=dev).double()
    f32 = lambda v: float(np.float32(v))
    fx, fy, cx, cy = f32(cam.fx), f32(cam.fy), f32(cam.cx), f32(cam.cy)
    t = means @ V[:3, :3].T + V[:3, 3]
    front = t[:, 2] > f32(0.2)
    z = torch.where(front, t[:, 2], torch.ones_like(t[:, 2]))
    lx, ly = 1.3 * cam.width / (2 * fx), 1.3 * cam.height / (2 * fy)
    tx, ty = (t[:, 0] / z).clamp(-lx, lx) * z, (t[:, 1] / z).clamp(-ly, ly) * z
    zero = torch.zeros_like(z)
    J = torch.stack([torch.stack([fx / z, zero, -fx * tx / (z * z)], 1),
                     torch.stack([zero, fy / z, -fy * ty / (z * z)], 1)], 1)
    r, x, y, w = (quats / quats.norm(dim=1, keepdim=True)).unbind(1)
    # rows of the rotation in the layout S R: world covariance (S R)^T (S R)
    R = torch.stack([torch.stack([1 - 2 * (y * y + w * w), 2 * (x * y + r * w),
                                  2 * (x * w - r * y)], 1),
                     torch.stack([2 * (x * y - r * w), 1 - 2 * (x * x + w * w),
                                  2 * (y * w + r * x)], 1),
                     torch.stack([2 * (x * w + r * y), 2 * (y * w - r * x),
                                  1 - 2 * (x * x + y * y)], 1)], 1)
    M = torch.exp(log_scales)[:, :, None] * R @ V[:3, :3].T @ J.transpose(1, 2)
    cov = M.transpose(1, 2) @ M
    k = f32(case["kernel"])
    a, b, c = cov[:, 0, 0] + k, cov[:, 0, 1], cov[:, 1, 1] + k
    det0 = (cov[:, 0, 0] * cov[:, 1, 1] - b * b).clamp_min(1e-6)
    coef = torch.sqrt(det0 / (a * c - b * b).clamp_min(1e-6)).detach()
    # the largest screen variance is capped at min(1024, W, H)^2 / 8
    radius = torch.sqrt((0.5 * (a - c)) ** 2 + b * b + 1e-300)
    lam = 0.5 * (a + c) + radius
    cap = 0.125 * min(1024.0, cam.width, cam.height) ** 2
    q = torch.where(lam > cap, cap / lam, torch.ones_like(lam))
    a, b, c = a * q, b * q, c * q
    det = a * c - b * b
    opac = torch.sigmoid(logits.reshape(-1)) * coef
    d = means - eye
    d = d / d.norm(dim=1, keepdim=True)
    basis = _sh_basis(d, case["degree"])
    rgb = (torch.einsum("nk,nkc->nc", basis, sh[:, :basis.shape[1]]) + 0.5).clamp_min(0)
    reach = 2 * torch.log((opac * 255).clamp_min(1e-30))
    seen = front & (reach >= 0) & (det > 0)
    px, py = t[:, 0] / z * fx + cx, t[:, 1] / z * fy + cy
    ex, ey = torch.sqrt((reach * a).clamp_min(0)), torch.sqrt((reach * c).clamp_min(0))
    seen = seen & (px + ex > -1) & (px - ex < cam.width) & (py + ey > -1) & (py - ey < cam.height)
    flat = torch.stack([px, py, c / det, -b / det, a / det, opac], 1)
    flat = torch.cat([flat, rgb], 1)  # [N, 9]
    with torch.no_grad():
        order = torch.nonzero(seen).flatten()
        order = order[torch.sort(t[order].norm(dim=1), stable=True).indices]
        box = torch.stack([px - ex, px + ex, py - ey, py + ey], 1)[order]
    return flat, order, box


def _blend(q, xs, ys, clip=float(np.float32(0.99))):
    """Blend of the depth-ordered Gaussians q [K,9] at pixels (xs, ys): weights
    [P,K], final transmittance [P], alphas and transmittances in front."""
    dx, dy = q[None, :, 0] - xs[:, None], q[None, :, 1] - ys[:, None]
    power = -0.5 * (q[:, 2] * dx * dx + q[:, 4] * dy * dy) - q[:, 3] * dx * dy
    raw = q[:, 5] * torch.exp(power.clamp_max(0))
    alpha = raw + (raw.clamp_max(clip) - raw).detach()  # the clip passes gradients through
    alpha = torch.where((power > 0) | (alpha < 1 / 255), torch.zeros_like(alpha), alpha)
    after = torch.cumprod(1 - alpha, 1)
    alpha = torch.where(after >= 1e-4, alpha, torch.zeros_like(alpha))
    after = torch.cumprod(1 - alpha, 1)
    before = torch.cat([torch.ones_like(after[:, :1]), after[:, :-1]], 1)
    return alpha * before, after[:, -1], alpha, before


def _blocks(cam, order, box, side=32):
    """(pixel ids, x, y, rows of the depth order reaching the block)."""
    dev = box.device
    for y0 in range(0, cam.height, side):
        y1 = min(cam.height, y0 + side)
        row = torch.nonzero((box[:, 2] <= y1) & (box[:, 3] >= y0 - 1)).flatten()
        bx = box[row]
        for x0 in range(0, cam.width, side):
            x1 = min(cam.width, x0 + side)
            hit = row[(bx[:, 0] <= x1) & (bx[:, 1] >= x0 - 1)]
            ys, xs = torch.meshgrid(torch.arange(y0, y1, device=dev),
                                    torch.arange(x0, x1, device=dev), indexing="ij")
            ys, xs = ys.flatten(), xs.flatten()
            yield ys * cam.width + xs, xs.double(), ys.double(), order[hit]


def _background(dev):
    return torch.tensor([0.1, 0.2, 0.3], dtype=torch.float32, device=dev).double()


def _image64(flat, order, box, cam):
    bg = _background(flat.device)
    color = bg[:, None].repeat(1, cam.width * cam.height)
    alpha = torch.zeros(cam.width * cam.height, dtype=torch.float64, device=flat.device)
    with torch.no_grad():
        for pid, xs, ys, ids in _blocks(cam, order, box):
            if ids.numel() == 0:
                continue
            q = flat[ids]
            w, T, _, _ = _blend(q, xs, ys)
            color[:, pid] = (w @ q[:, 6:] + T[:, None] * bg).T
            alpha[pid] = 1 - T
    return color.view(3, cam.height, cam.width), alpha.view(cam.height, cam.width)


def _flat_grads(flat, order, box, cam, g_color, g_alpha):
    bg = _background(flat.device)
    out = torch.zeros_like(flat)
    gc = g_color.double().reshape(3, -1)
    ga = None if g_alpha is None else g_alpha.double().reshape(-1)
    for pid, xs, ys, ids in _blocks(cam, order, box):
        if ids.numel() == 0:
            continue
        q = flat[ids].detach().requires_grad_()
        w, T, _, _ = _blend(q, xs, ys)
        total = ((w @ q[:, 6:] + T[:, None] * bg) * gc[:, pid].T).sum()
        if ga is not None:
            total = total + ((1 - T) * ga[pid]).sum()
        out.index_add_(0, ids, torch.autograd.grad(total, q)[0])
    return out


def _params64(model):
    return [p.detach().double().requires_grad_() for p in
            (model.means, model.log_scales, model.quaternions, model.opacity_logits, model.sh)]


def _window64(dev):
    # the 11 float32 taps of a normalised Gaussian of sigma 1.5
    t = np.exp(-0.5 * (np.arange(-5, 6) / 1.5) ** 2)
    return torch.tensor((t / t.sum()).astype(np.float32), device=dev).double()


def _ssim_loss(a, b, mask, ssim_weight, photometric_weight):
    """w / (3 (W-10)(H-10)) sum over the valid window of lambda (1 - SSIM) +
    (1 - lambda) |a - b| (both images times the mask)."""
    if mask is not None:
        a, b = a * mask, b * mask
    k = _window64(a.device)

    def blur(x):
        x = torch.nn.functional.conv2d(x[:, None], k.view(1, 1, 1, 11), padding=(0, 5))
        return torch.nn.functional.conv2d(x, k.view(1, 1, 11, 1), padding=(5, 0))[:, 0]

    m1, m2 = blur(a), blur(b)
    s11, s22, s12 = blur(a * a) - m1 * m1, blur(b * b) - m2 * m2, blur(a * b) - m1 * m2
    c1, c2 = 0.01 ** 2, 0.03 ** 2
    ssim = ((2 * m1 * m2 + c1) * (2 * s12 + c2)) / ((m1 * m1 + m2 * m2 + c1) * (s11 + s22 + c2))
    per = ssim_weight * (1 - ssim) + (1 - ssim_weight) * (a - b).abs()
    _, h, w = a.shape
    return photometric_weight * per[:, 5:h - 5, 5:w - 5].sum() / (3 * (h - 10) * (w - 10))


def _exact_loss(case, g):
    im = {k: v.double() for k, v in _loss_images(case, g).items()}
    o = gsb.TrainingLossOptions(**LOSS_OPTIONS)
    h, w = case["h"], case["w"]
    inv = 1.0 / (h * w)
    color, alpha, depth, normal = [im[k].requires_grad_() for k in
                                   ("color", "alpha", "median_depth", "normal")]
    mask = im["mask"]
    rgb = _ssim_loss(color, im["target_color"], mask, o.ssim_weight, o.photometric_weight)
    td = im["target_depth"]
    has = (td > 0) & (depth > 0) & (mask > 0)
    rel = (depth - td) / td.clamp_min(1e-4)
    t_depth = (torch.where(has, torch.sqrt(rel * rel + o.geometry_epsilon ** 2),
                           torch.zeros_like(rel)) * mask).sum() * o.depth_weight * inv
    tn = im["target_normal"]
    l2 = (tn * tn).sum(0)
    has = (l2 > 0.25) & (mask > 0)
    unit = tn / torch.sqrt(l2.clamp_min(1e-30))
    t_normal = (torch.where(has, 1 - (normal * unit).sum(0), torch.zeros_like(l2)) *
                mask).sum() * o.normal_weight * inv
    lo, hi = float(np.float32(1e-7)), float(np.float32(1) - np.float32(1e-7))
    pr = alpha.clamp(lo, hi)
    t_alpha = -o.match_alpha_weight * inv * (mask * torch.log(pr) +
                                             (1 - mask) * torch.log(1 - pr)).sum()
    f, cx, cy = case["f"], w / 2, h / 2
    yy, xx = torch.meshgrid(torch.arange(h, device="cuda").double(),
                            torch.arange(w, device="cuda").double(), indexing="ij")
    pts = torch.stack([(xx - cx) / f, (yy - cy) / f, torch.ones_like(xx)]) * depth
    dy, dx = pts[:, 2:, 1:-1] - pts[:, :-2, 1:-1], pts[:, 1:-1, 2:] - pts[:, 1:-1, :-2]
    ok = ((depth[1:-1, 1:-1] > 0) & (depth[:-2, 1:-1] > 0) & (depth[2:, 1:-1] > 0) &
          (depth[1:-1, :-2] > 0) & (depth[1:-1, 2:] > 0))
    cr = torch.linalg.cross(dy, dx, dim=0)
    n2 = (cr * cr).sum(0)
    ok = ok & (n2 > 1e-20)
    unit = cr / torch.sqrt(torch.where(ok, n2, torch.ones_like(n2)))
    t_normal = t_normal + o.depth_normal_weight * inv * torch.where(
        ok, 1 - (normal[:, 1:-1, 1:-1] * unit).sum(0), torch.zeros_like(n2)).sum()
    gc, ga, gd, gn = torch.autograd.grad(rgb + t_depth + t_normal + t_alpha,
                                         [color, alpha, depth, normal])
    terms = torch.stack([rgb, t_depth, t_normal, t_alpha]).detach()
    return {"color": gc, "alpha": ga, "depth": gd, "normal": gn, "terms": terms}


def _adam64(p, grad, first, second, lr, c1, c2, lo=-math.inf, hi=math.inf):
    first = BETA1 * first.double() + (1 - BETA1) * grad
    second = BETA2 * second.double() + (1 - BETA2) * grad * grad
    new = p.double() - lr * (first / c1) / (torch.sqrt(second / c2) + ADAM_EPS)
    return new.clamp(lo, hi), first, second


def _sh_adam64(sh, grad, state, c1, c2):
    """The quantized SH Adam: log-second codes decoded, one update, new bounds."""
    n = sh.shape[0]
    b = state["bounds"].double()
    dc = (torch.arange(16, device=sh.device) == 0)[None, :, None]
    lo = torch.where(dc, b[:, 0, None, None], b[:, 2, None, None])
    hi = torch.where(dc, b[:, 1, None, None], b[:, 3, None, None])
    s = CODEC_EPS * (torch.exp(lo + (hi - lo) * state["packed"].double() / 255) - 1)
    pc1, pc2 = (c1 - (1 - BETA1)) / BETA1, (c2 - (1 - BETA2)) / BETA2
    m = BETA1 * state["first"].double() * (s / math.sqrt(pc2) + SH_EPS) * pc1 + (1 - BETA1) * grad
    v = BETA2 * s * s + (1 - BETA2) * grad * grad
    norm = (m / c1) / (torch.sqrt(v / c2) + SH_EPS)
    new = sh.double() - torch.where(dc, SH_LR, SH_REST_LR) * norm
    log_s = torch.log(1 + torch.sqrt(v) / CODEC_EPS)
    d, r = log_s[:, :1].reshape(n, -1), log_s[:, 1:].reshape(n, -1)
    bounds = torch.stack([d.amin(1), d.amax(1), r.amin(1), r.amax(1)], 1)
    return new, norm, bounds


def _exact_step(case, g):
    model, cam = _model(case, g), _cameras(case)[0]
    target = _photo(case, g).double()
    st, sh = _adam(model, g)
    c1, c2 = (float(np.float32(c)) for c in _corrections(STEP + 1))
    p = _params64(model)
    flat, order, box = _project(p, cam, case)
    fd = flat.detach()
    color, alpha = _image64(fd, order, box, cam)
    pred = color.clone().requires_grad_()
    loss = _ssim_loss(pred, target, None, 0.2, 1.0)
    gc = torch.autograd.grad(loss, pred)[0]
    gp = torch.autograd.grad(flat, p, _flat_grads(fd, order, box, cam, gc, None))
    out = {"color": color, "alpha": alpha, "radii": None, "visibility": None,
           "loss": loss.detach().reshape(1)}
    names = (("means", "means"), ("log_scales", "scales"), ("quaternions", "rotations"),
             ("opacity_logits", "opacity"))
    moments = {}
    for k, (field, m) in enumerate(names):
        lr = list(LRS.values())[k]
        clamp = 12.0 if m == "opacity" else math.inf
        out[field], moments[m + "_first"], moments[m + "_second"] = _adam64(
            getattr(model, field), gp[k], st[m + "_first"], st[m + "_second"], lr, c1, c2,
            -clamp, clamp)
    out["sh"], first, bounds = _sh_adam64(model.sh, gp[4], sh, c1, c2)
    out.update({k: moments[k] for k in st})
    out.update(sh_first=first, sh_packed=None, sh_bounds=bounds, refine_weight=None)
    return out


def _exact_prune(case, g):
    model, cam = _model(case, g), _cameras(case)[0]
    with torch.no_grad():
        flat, order, box = _project(_params64(model), cam, case)
        bg = _background(flat.device).sum()
        scores = torch.zeros(case["n"], dtype=torch.float64, device="cuda")
        for _, xs, ys, ids in _blocks(cam, order, box):
            if ids.numel() == 0:
                continue
            q = flat[ids]
            w, T, alpha, before = _blend(q, xs, ys)
            c = q[:, 6:].sum(1)
            part = torch.cumsum(w * c, 1)
            behind = part[:, -1:] + (T * bg)[:, None] - part
            d = q[:, 5] * (before * c - behind / (1 - alpha))
            scores.index_add_(0, ids, torch.where(alpha > 0, d * d, torch.zeros_like(d)).sum(0))
    return {"scores": scores}


def exact(case, seed):
    kind = case["kind"]
    views = _cameras(case)
    pixels = sum(c.width * c.height for c in views)
    if case["n"] * len(views) > 1200000 or pixels > 2200000:
        return None  # the blend of every pixel in 64 bits takes too long
    g = _gen(seed)
    if kind == "loss":
        return _exact_loss(case, g)
    if kind == "step":
        return _exact_step(case, g)
    if kind == "prune":
        return _exact_prune(case, g)
    model = _model(case, g)
    p = _params64(model)
    if kind == "render":
        with torch.no_grad():
            flat, order, box = _project(p, views[0], case)
        color, alpha = _image64(flat, order, box, views[0])
        return {"color": color, "alpha": alpha, "radii": None, "visibility": None}
    grads = _image_grads(case, views, g)
    if kind == "geometry":
        with torch.no_grad():
            flat, order, box = _project(p, views[0], case)
        color, alpha = _image64(flat, order, box, views[0])
        out = dict.fromkeys(("color", "alpha", "median_depth", "normal", "radii", "means",
                             "log_scales", "quaternions", "opacity_logits", "sh",
                             "refine_weight"))
        out.update(color=color, alpha=alpha)
        return out
    total, colors, alphas, off = None, [], [], 0
    for cam in views:
        size = cam.width * cam.height
        gc = grads["color"].flatten()[3 * off:3 * (off + size)] if kind == "batch" \
            else grads["color"]
        flat, order, box = _project(p, cam, case)
        fd = flat.detach()
        color, alpha = _image64(fd, order, box, cam)
        gp = torch.autograd.grad(flat, p, _flat_grads(fd, order, box, cam, gc,
                                                      grads.get("alpha")))
        total = list(gp) if total is None else [a + b for a, b in zip(total, gp)]
        colors.append(color)
        alphas.append(alpha)
        off += size
    out = {"color": colors[0], "alpha": alphas[0], "radii": None, "means": total[0],
           "log_scales": total[1], "quaternions": total[2], "opacity_logits": total[3],
           "sh": total[4]}
    if kind == "batch":
        out["color"] = torch.cat([c.flatten() for c in colors])
        out["alpha"] = torch.cat([a.flatten() for a in alphas])
        out["refine_weight"] = None
    return out
