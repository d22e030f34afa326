"""The geometry channels' adjoint (median depth, normals, colour, alpha)
against central differences of the rendered channels, on few wide overlapping
Gaussians: every weighted pixel keeps its blends, its order and its median
bracket under the steps taken, so the channels are smooth there. Both strip
shapes (up to 1,000 tiles, and above), and lists with more Gaussians around the
median than a pixel keeps (96), whose forward is also held to the CPU oracle.

Bound: 3e-3 of the gradients' size along a step, for the third-order term of the
differences and the adjoint's own rounding (a wrong or missing term is of the
size itself), and four deviations of the channels' float32 rounding: an ulp
(2^-23 of values around 1 to 3) a weighted value, at random, over the
differences' 4e-3."""
import importlib

import numpy as np
import pytest
import torch

from helpers import camera_of, clone_model, device_model, gsb

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

cpu = pytest.importorskip("oracle.cpu")
scenes = importlib.import_module("photara-studio_b200.scenes")

PARAMS = ("means", "log_scales", "quaternions", "opacity_logits")


def _scene(n, w, h, opacity, seed):
    """n flat Gaussians about 0.27 of the image wide (below the covariance cap),
    a little tilted, one behind the other around z = 3.15: thin enough for every
    median to lie within the window around its seed."""
    rng = np.random.default_rng(seed)
    means = np.column_stack([rng.uniform(-0.25, 0.25, (n, 2)), np.linspace(3.0, 3.3, n)])
    q = np.column_stack([np.ones(n), 0.05 * rng.normal(size=(n, 3))])
    axes = np.log([0.9, 0.9, 0.08])
    f32 = lambda a: np.ascontiguousarray(a, np.float32)
    sh = 0.3 * rng.normal(size=(n, 16, 3))
    return scenes.SceneArrays(
        f32(means), f32(axes + 0.1 * rng.normal(size=(n, 3))),
        f32(q / np.linalg.norm(q, axis=1, keepdims=True)),
        f32(np.full((n, 1), np.log(opacity / (1 - opacity)))), f32(sh), w, h, float(w), float(w),
        w / 2.0, h / 2.0, list(scenes.IDENTITY16), [0.0, 0.0, 0.0])


def _forward(model, cam):
    return gsb.Rasterizer().forward(model, cam, gsb.RasterizeOptions(
        active_sh_degree=3, require_depth=True, background=(0.1, 0.2, 0.3)))


@pytest.mark.parametrize("n,w,h,opacity,channels", [
    (12, 24, 24, 0.3, ("depth",)),
    (12, 24, 24, 0.3, ("normal",)),
    (12, 24, 24, 0.3, ("color", "alpha", "depth", "normal")),
    (12, 512, 530, 0.3, ("color", "alpha", "depth", "normal")),  # 1,088 tiles
    (150, 24, 24, 0.03, ("depth", "alpha")),                     # more than a pixel keeps
    (150, 512, 530, 0.03, ("depth", "alpha")),
])
def test_gradients_match_central_differences(n, w, h, opacity, channels):
    scene = _scene(n, w, h, opacity, seed=n + w)
    model, cam = device_model(scene), camera_of(scene)
    r = _forward(model, cam)
    g = torch.Generator("cuda").manual_seed(n + h)
    yy, xx = torch.meshgrid(torch.arange(h, device="cuda"), torch.arange(w, device="cuda"),
                            indexing="ij")
    disc = ((xx - w / 2) ** 2 + (yy - h / 2) ** 2) < (0.33 * w) ** 2
    assert float(r.alpha[disc].min()) > 0.6 and float(r.alpha.max()) < 1 - 2e-4
    assert bool((r.median_depth[disc] > 0).all())
    waves = lambda: torch.cos(2 * xx / w + 3 * yy / h + 6 * float(torch.rand(
        (), device="cuda", generator=g))) * disc
    weight = {c: torch.stack([waves() for _ in range(k)]).view(*([3] if k == 3 else []), h, w) *
              (c in channels) for c, k in (("color", 3), ("alpha", 1), ("depth", 1),
                                           ("normal", 3))}
    weight = {c: v.float().contiguous() for c, v in weight.items()}
    grads = gsb.Rasterizer().backward(model, r, weight["color"], weight["alpha"],
                                      grad_depth=weight["depth"], grad_normal=weight["normal"])

    def value(name, step):
        m = clone_model(model)
        getattr(m, name).add_(step)
        q = _forward(m, cam)
        assert bool((q.median_depth[disc] > 0).all())
        out = {"color": q.color, "alpha": q.alpha, "depth": q.median_depth, "normal": q.normal}
        return sum(float((weight[c].double() * out[c].double()).sum()) for c in channels)

    values = sum(int((v != 0).sum()) for v in weight.values())
    for name in PARAMS:
        grad = getattr(grads, name).double()
        size = float(grad.norm())
        assert size > 0
        steps = [grad / grad.abs().max()]  # all at once, single Gaussians, at random
        for k in (0, n // 2, n - 1):
            one = torch.zeros_like(grad)
            one[k] = grad[k] / grad[k].abs().max()
            steps.append(one)
        steps += [torch.randn(grad.shape, device="cuda", generator=g).double().clamp(-1, 1)
                  for _ in range(3)]
        for d in steps:
            eps = 2e-3
            diff = (value(name, (eps * d).float()) - value(name, (-eps * d).float())) / (2 * eps)
            along = float((grad * d).sum())
            scale = float((grad * (d != 0)).norm() * d.norm())
            noise = 4 * values ** 0.5 * 2.0 ** -23 / (2 * eps)
            assert abs(diff - along) <= 3e-3 * scale + noise, (name, diff, along, scale, noise)


@pytest.mark.parametrize("n,opacity", [(60, 0.08), (96, 0.05), (97, 0.05), (300, 0.015)])
def test_median_depth_of_long_lists_matches_oracle(n, opacity):
    """Every pixel's Gaussians are all around its median: up to the 96 it keeps,
    and above (the tolerance of test_gpu_geometry.py against the oracle)."""
    scene = _scene(n, 40, 36, opacity, seed=n)
    r = _forward(device_model(scene), camera_of(scene))
    o = cpu.render(scene, use_double=False, background=(0.1, 0.2, 0.3))
    expect = cpu.geometry(scene, o)["median_depth"]
    got = r.median_depth.cpu().numpy()
    assert (got > 0).mean() > 0.3
    assert (np.abs(got - expect) <= 1e-3).mean() >= 0.995
    assert np.abs(got - expect)[(got > 0) & (expect > 0)].max() <= 1e-3
