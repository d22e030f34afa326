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


@pytest.mark.parametrize("ppt", [1, 2, 4, 8])
@pytest.mark.parametrize("w,h,n", [(5, 3, 1), (16, 16, 33), (17, 31, 300), (33, 18, 5),
                                   (47, 65, 700)])
def test_uneven_strips_match_oracle(ppt, w, h, n):
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
    # is the rendered alpha (float32 sums of at most w h n terms)
    assert torch.equal(weighted.densify_weight, weighted.densify_weight_den)
    assert abs(float(weighted.densify_weight_den.sum()) - float(r.alpha.sum())) <= \
        1e-4 * max(float(r.alpha.sum()), 1.0)
