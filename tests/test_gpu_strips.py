"""Strip compositing kernels at every pixels-per-thread count on sizes where
strips, bands, batches of 32 Gaussians and gathers of four end unevenly: images
narrower or lower than a strip, last tiles partly outside, lists of 1 to a few
hundred entries, empty tiles. Forward and adjoint (with the densify sums)
against the CPU oracle: images 2e-5 absolute, gradients 1e-3 relative L2 (the
tolerances of test_gpu_oracle_parity.py; a lone Gaussian's few terms obey them
too)."""
import dataclasses

import numpy as np
import pytest
import torch

from helpers import camera_of, device_model, gsb

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

cpu = pytest.importorskip("oracle.cpu")


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64).ravel(), np.asarray(b, np.float64).ravel()
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30))


@pytest.mark.parametrize("ppt", [1, 2, 4, 8, None])
@pytest.mark.parametrize("w,h,n", [(5, 3, 1), (16, 16, 33), (17, 31, 300), (33, 18, 5),
                                   (47, 65, 700)])
def test_uneven_strips_match_oracle(ppt, w, h, n):
    """ppt None: the automatic schedule, whose adjoint of so few tiles walks
    the list segments in parallel."""
    scene = dataclasses.replace(gsb.make_scene("tiny", seed=n + w, count=n), width=w, height=h,
                                cx=w / 2.0, cy=h / 2.0, fx=40.0, fy=40.0)
    model, cam = device_model(scene), camera_of(scene)
    rast = gsb.Rasterizer(pixels_per_thread=ppt)
    bg = (0.3, 0.1, 0.2)
    r = rast.forward(model, cam, gsb.RasterizeOptions(active_sh_degree=3, background=bg))
    o = cpu.render(scene, background=bg)
    assert np.abs(r.color.cpu().numpy() - o["color"]).max() <= 2e-5
    assert np.abs(r.alpha.cpu().numpy() - o["alpha"]).max() <= 2e-5
    rng = np.random.default_rng(n)
    gc = rng.normal(size=(3, h, w)).astype(np.float32)
    ga = rng.normal(size=(h, w)).astype(np.float32)
    t = lambda a: torch.from_numpy(a).cuda()
    plain = rast.backward(model, r, t(gc), t(ga))
    weighted = rast.backward(model, r, t(gc), t(ga), densify_map=torch.ones((h, w), device="cuda"))
    og = cpu.backward(scene, o, gc, ga)
    for g in (plain, weighted):  # the adjoint may run twice on one forward
        for name, ref in (("means", "means"), ("log_scales", "scales"),
                          ("quaternions", "rotations"), ("opacity_logits", "opacities"),
                          ("sh", "sh"), ("refine_weight", "refine_weight")):
            assert rel_l2(getattr(g, name).cpu().numpy(), og[ref]) <= 1e-3, name
    # with a map of ones both densify sums are the blend weights, whose total
    # is the rendered alpha (float32 sums of at most w h n terms). Their atomics
    # add equal values, one a strip (at most 8 of each of 15 tiles), in two
    # orders: 119 additions of 2^-24 of the sum each
    den = weighted.densify_weight_den
    assert bool(((weighted.densify_weight - den).abs() <= 2 * 119 * 2.0 ** -24 * den).all())
    assert abs(float(weighted.densify_weight_den.sum()) - float(r.alpha.sum())) <= \
        1e-4 * max(float(r.alpha.sum()), 1.0)


@pytest.mark.parametrize("count,logit", [(64, 0.0), (65, -3.0), (1024, -5.0), (1500, -5.2)])
def test_long_lists_in_segments_match_whole_lists(count, logit):
    """Every Gaussian over the whole of a small image, lists of one segment to
    more than the sixteen checkpoint levels hold: the segment-parallel adjoint
    against the whole-list one and, for one more colour set, after
    forward_colors. Tolerance (relative L2): the whole-list walk recovers the
    transmittance by one rounded multiplication per entry (an ulp, 2^-23, each),
    the segments restart it from the forward's, so the two may part by
    count * 2^-23 of a term; 1e-5 for the other sums, 1e-4 for the opacities,
    whose terms cancel."""
    drift = count * 2.0 ** -23
    scene = dataclasses.replace(gsb.make_scene("tiny", seed=count, count=count), width=20,
                                height=18, cx=10.0, cy=9.0, fx=20.0, fy=20.0)
    model, cam = device_model(scene), camera_of(scene)
    model.means = (model.means * torch.tensor([0.1, 0.1, 1.0], device="cuda")).contiguous()
    # unequal axes: an isotropic Gaussian's quaternion gradient is zero, and the
    # relative difference of two roundings of zero has no bound
    model.log_scales = (1.0 + 0.5 * (model.log_scales + 3.5)).contiguous()
    model.opacity_logits = torch.full_like(model.opacity_logits, logit)
    g = torch.Generator("cuda").manual_seed(count)
    colors = [torch.rand((count, 3), device="cuda", generator=g) for _ in range(2)]
    gc = torch.randn((3, 18, 20), device="cuda", generator=g)
    ga = torch.randn((18, 20), device="cuda", generator=g)
    out = []
    for ppt in (1, None):
        rast = gsb.Rasterizer(pixels_per_thread=ppt)
        r = rast.forward(model, cam, gsb.RasterizeOptions(colors_precomp=colors[0],
                                                          background=(0.1, 0.2, 0.3)))
        first = rast.backward(model, r, gc, ga)
        again = rast.forward_colors(r, colors[1])
        second = rast.backward(model, again, gc, ga)
        out.append((r.color, again.color, first, second))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    for a, b in zip(out[0][2:], out[1][2:]):
        for name in ("means", "log_scales", "quaternions", "opacity_logits", "colors_precomp",
                     "refine_weight"):
            x, y = getattr(a, name).cpu().numpy(), getattr(b, name).cpu().numpy()
            assert rel_l2(y, x) <= drift + (1e-4 if name == "opacity_logits" else 1e-5), name


@pytest.mark.parametrize("w,h", [(400, 300), (512, 530)])  # 475 and 1,088 tiles
@pytest.mark.parametrize("minor,aspect", [(0.05, 3000), (0.02, 5000), (0.3, 1000), (0.3, 300),
                                          (0.5, 70)])
def test_needles_lose_no_blend(w, h, minor, aspect):
    """Thin tilted Gaussians (minor axis in pixels), whose 32-bit ellipse has
    lost its digits: every strip shape blends what the forward of the geometry
    channels blends, which tests each pixel against the whole list, and both
    adjoints walk all of it (with a map of ones the densify weights add up to
    the rendered alpha: float32 terms of 1e-8 to 1, so 1e-6 of the sum)."""
    n, z, f = 400, 4.0, 500.0
    g = torch.Generator("cuda").manual_seed(aspect)
    u = lambda *s: torch.rand(s, device="cuda", generator=g)
    s = minor * z / f
    scales = torch.tensor([s * aspect, s, s], device="cuda").log().expand(n, 3).contiguous()
    q = torch.randn((n, 4), device="cuda", generator=g)
    half = torch.tensor([0.45 * w * z / f, 0.45 * h * z / f, 0.25], device="cuda")
    means = ((2 * u(n, 3) - 1) * half + torch.tensor([0.0, 0.0, z], device="cuda")).contiguous()
    model = gsb.GaussianModel(means, scales, (q / q.norm(dim=1, keepdim=True)).contiguous(),
                              torch.randn((n, 1), device="cuda", generator=g),
                              0.3 * torch.randn((n, 16, 3), device="cuda", generator=g), 3)
    identity = [1.0, 0, 0, 0, 0, 1.0, 0, 0, 0, 0, 1.0, 0, 0, 0, 0, 1.0]
    cam = gsb.Camera(identity, [0.0, 0.0, 0.0], f, f, w / 2, h / 2, w, h)
    ones = torch.ones((h, w), device="cuda")

    def weights_add_up(rast, r, **grads):
        got = rast.backward(model, r, torch.zeros_like(r.color), densify_map=ones, **grads)
        total = float(r.alpha.double().sum())
        assert abs(float(got.densify_weight_den.double().sum()) - total) <= 1e-6 * total

    rast = gsb.Rasterizer()
    whole = rast.forward(model, cam, gsb.RasterizeOptions(active_sh_degree=3, require_depth=True))
    assert float(whole.alpha.max()) > 0.5
    weights_add_up(rast, whole, grad_depth=torch.zeros_like(ones),
                   grad_normal=torch.zeros_like(whole.color))
    for ppt in (1, 2, 4, 8, None):
        rast = gsb.Rasterizer(pixels_per_thread=ppt)
        r = rast.forward(model, cam, gsb.RasterizeOptions(active_sh_degree=3))
        assert torch.equal(r.color, whole.color) and torch.equal(r.alpha, whole.alpha), ppt
        weights_add_up(rast, r)


@pytest.mark.parametrize("ppt", [1, 2, 4, 8, None])
def test_a_clip_below_the_blend_threshold_blends_and_adjoins_nothing(ppt):
    """Every opacity is clipped to 0.003 < 1/255: no Gaussian is blended, so
    none has a last contributor or a gradient."""
    scene = gsb.make_scene("tiny", seed=3)
    model, cam = device_model(scene), camera_of(scene)
    rast = gsb.Rasterizer(pixels_per_thread=ppt)
    r = rast.forward(model, cam, gsb.RasterizeOptions(
        active_sh_degree=3, rasterization=gsb.RasterizationPolicy(alpha_clip=0.003)))
    assert r.rendered_instances > 0 and not bool(r.alpha.any()) and not bool(r.visibility.any())
    g = rast.backward(model, r, torch.ones_like(r.color), torch.ones_like(r.alpha))
    for name in ("means", "log_scales", "quaternions", "opacity_logits", "sh", "refine_weight"):
        assert not bool(getattr(g, name).any()), name
