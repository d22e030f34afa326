"""Infinities and NaN reach only the pixels and Gaussians they are blended
into: a Gaussian or pixel that does not take part keeps its value (images bit
for bit; gradients to the order of float atomics, 1e-5 of the largest)."""
import dataclasses
import importlib

import pytest
import torch

from helpers import camera_of, device_model, gsb

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

batch = importlib.import_module("photara-studio_b200.batch")

NAMES = ("means", "log_scales", "quaternions", "opacity_logits", "refine_weight")


class _Case:
    """Precomputed colours over one view, with the blend weights of one
    Gaussian per pixel, or of every Gaussian over a set of pixels."""

    def __init__(self, ppt, seed, **options):
        scene = gsb.make_scene("tiny", seed=seed)
        if ppt == "690 tiles":  # the automatic schedule's two pixels, in segments
            scene, ppt = dataclasses.replace(scene, width=480, height=368, cx=240.0, cy=184.0,
                                             fx=400.0, fy=400.0), None
        self.model, self.cam = device_model(scene), camera_of(scene)
        self.rast, self.options = gsb.Rasterizer(pixels_per_thread=ppt), options
        self.n = self.model.size()
        g = torch.Generator("cuda").manual_seed(seed)
        self.colors = torch.rand((self.n, 3), device="cuda", generator=g)
        self.grad = torch.randn((3, self.cam.height, self.cam.width), device="cuda", generator=g)

    def render(self, colors):
        return self.rast.forward(self.model, self.cam, gsb.RasterizeOptions(
            colors_precomp=colors, **self.options))

    def weights_of(self, k):
        one = torch.zeros_like(self.colors)
        one[k] = 1.0
        return self.render(one).color[0]

    def weights_over(self, pixels):
        dl = torch.zeros_like(self.grad)
        dl[0] = pixels.float()
        return self.rast.backward(self.model, self.render(self.colors), dl).colors_precomp[:, 0]

    def middle(self):
        """A Gaussian blended into a fair number of pixels."""
        r = self.render(self.colors)
        order = torch.argsort((r.radii - 12).abs())
        return next(int(k) for k in order[:50] if int((self.weights_of(int(k)) > 0).sum()) > 20)


def _same(a, b, rows, names):
    assert int(rows.sum()) > 20
    for name in names:
        x, y = getattr(a, name), getattr(b, name)
        assert float((x[rows] - y[rows]).abs().max()) <= 1e-5 * float(y.abs().max()), name


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("ppt", [1, 2, 4, 8, None, "690 tiles"])
def test_colour_that_is_not_finite(ppt, value):
    c = _Case(ppt, 5)
    k = c.middle()
    inside = c.weights_of(k) > 0
    bad = c.colors.clone()
    bad[k] = value
    good, r = c.render(c.colors), c.render(bad)
    assert torch.equal(r.color[:, ~inside], good.color[:, ~inside])
    assert not bool(torch.isfinite(r.color[:, inside]).any())
    assert torch.equal(r.alpha, good.alpha) and torch.equal(r.visibility, good.visibility)
    again = c.rast.forward_colors(c.render(c.colors), bad)
    assert torch.equal(again.color[:, ~inside], good.color[:, ~inside])
    assert not bool(torch.isfinite(again.color[:, inside]).any())
    back = c.rast.forward_colors(again, c.colors)
    assert torch.equal(back.color, good.color)
    away = c.weights_over(inside) == 0
    _same(c.rast.backward(c.model, r, c.grad), c.rast.backward(c.model, good, c.grad), away,
          NAMES + ("colors_precomp",))


@pytest.mark.parametrize("geometry", [False, True])
@pytest.mark.parametrize("ppt", [1, 2, 4, 8, None, "690 tiles"])
def test_pixel_gradient_that_is_not_finite(ppt, geometry):
    c = _Case(ppt, 6, require_depth=geometry)
    r = c.render(c.colors)
    full = r.alpha > 0.5
    y, x = [int(v) for v in full.nonzero()[int(full.sum()) // 2]]
    pixel = torch.zeros_like(r.alpha)
    pixel[y, x] = 1.0
    dl = c.grad.clone()
    dl[1, y, x] = float("nan")
    extra = dict(grad_depth=torch.zeros_like(r.alpha), grad_normal=torch.zeros_like(r.color)) \
        if geometry else {}
    ones = torch.ones_like(r.alpha)
    away = c.weights_over(pixel) == 0
    plain = c.rast.backward(c.model, r, c.grad, densify_map=ones, **extra)
    _same(c.rast.backward(c.model, r, dl, **extra), plain, away, NAMES + ("colors_precomp",))
    ones[y, x] = float("inf")
    _same(c.rast.backward(c.model, r, c.grad, densify_map=ones, **extra), plain, away,
          NAMES + ("colors_precomp", "densify_weight", "densify_weight_den"))


@pytest.mark.parametrize("gaussian_pop", [False, True])
def test_pruning_scores_of_an_infinite_colour(gaussian_pop):
    """The scores of the Gaussians that share no pixel with the infinite one."""
    c = _Case(None, 7)
    k = c.middle()
    away = c.weights_over(c.weights_of(k) > 0) == 0
    scores = [c.rast.pruning_scores(c.model, c.cam, gaussian_pop=gaussian_pop)]
    c.model.sh[k] = float("inf")
    scores.append(c.rast.pruning_scores(c.model, c.cam, gaussian_pop=gaussian_pop))
    assert not bool(torch.isfinite(scores[1]).all())
    assert int(away.sum()) > 20
    assert float((scores[0][away] - scores[1][away]).abs().max()) <= 1e-5 * float(scores[0].max())


@pytest.mark.parametrize("tw,th,ppt,schedule", [
    (8, 8, 1, "dynamic"), (8, 8, 2, "static"), (16, 16, 4, "heavy_first"),
    (16, 32, 2, "dynamic")])
def test_batched_colour_that_is_not_finite(tw, th, ppt, schedule):
    """Both views show it; the batch planned before the colour turns infinite."""
    c = _Case(1, 9)
    k = c.middle()
    inside = c.weights_of(k) > 0
    br = batch.BatchRasterizer().plan(c.model, [c.cam, c.cam], gsb.RasterizeOptions(
        active_sh_degree=0), batch.BatchSchedule(tw, th, ppt, schedule))
    good = br.forward().color.clone()
    c.model.sh[k, 0, 1] = float("inf")
    br.forward()
    for v in range(2):
        got, was = br.result.view_color(v), good.view(2, *c.grad.shape)[v]
        assert torch.equal(got[:, ~inside], was[:, ~inside])
        assert torch.equal(got[::2], was[::2])
        assert not bool(torch.isfinite(got[1, inside]).any())
    c.model.sh[k, 0, 1] = 0.0
    br.forward()
    torch.cuda.synchronize()
    assert bool(torch.isfinite(br.result.color).all())


@pytest.mark.parametrize("tw,th,ppt", [(8, 8, 1), (16, 16, 4), (16, 32, 2)])
def test_batched_pixel_gradient_that_is_not_finite(tw, th, ppt):
    c = _Case(None, 8)
    br = batch.BatchRasterizer().plan(c.model, [c.cam, c.cam], gsb.RasterizeOptions(
        active_sh_degree=3), batch.BatchSchedule(tw, th, ppt))
    res = br.forward()
    y, x = 20, 30
    pixel = torch.zeros_like(res.view_alpha(0))
    pixel[y, x] = 1.0
    away = c.weights_over(pixel) == 0
    flat = torch.randn(res.color.numel(), device="cuda",
                       generator=torch.Generator("cuda").manual_seed(8))
    plain = br.backward(flat)
    flat = flat.clone()
    flat[y * c.cam.width + x] = float("nan")
    got = br.backward(flat)
    torch.cuda.synchronize()
    assert not bool(torch.isfinite(got.means).all())
    _same(got, plain, away, NAMES + ("sh",))
