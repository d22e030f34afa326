"""Several batched plans alive at once on one device (tolerances of
test_gpu_batch.py)."""
import importlib

import numpy as np
import pytest
import torch

from helpers import gsb

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

batch = importlib.import_module("photara-studio_b200.batch")
scenes = importlib.import_module("photara-studio_b200.scenes")

NAMES = ("means", "log_scales", "quaternions", "opacity_logits", "sh", "refine_weight")


def rel_l2(a, b):
    a, b = a.double().flatten(), b.double().flatten()
    return float((a - b).norm() / b.norm().clamp_min(1e-30))


def _setup(n, views, sizes, seed):
    arrays, ring = scenes.make_ring_batch(n, views=views, sizes=sizes, radius=6.0, half=2.0,
                                          seed=seed)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()
    model = gsb.GaussianModel(t(arrays.means), t(arrays.log_scales), t(arrays.quaternions),
                              t(arrays.opacity_logits), t(arrays.sh), 3)
    shapes = [sizes[k % len(sizes)] for k in range(views)]
    return model, [gsb.look_at_camera(v.eye, (0, 0, 0), (0, 1, 0), w, h, 0.5 * w)
                   for v, (w, h) in zip(ring, shapes)]


@pytest.mark.parametrize("sh_bases", [16, 9])  # rows staged by 16-byte copies, and the others
def test_a_later_plan_of_fewer_views_leaves_an_earlier_one_usable(sh_bases):
    model, cams = _setup(3000, 5, ((96, 72), (64, 48)), 1)
    if sh_bases == 9:
        model.sh, model.sh_degree = model.sh[:, :9].contiguous(), 2
    opts = gsb.RasterizeOptions(active_sh_degree=model.sh_degree)
    first = batch.BatchRasterizer().plan(model, cams, opts)
    color = first.forward().color.clone()
    flat = torch.randn(color.numel(), device="cuda",
                       generator=torch.Generator("cuda").manual_seed(1))
    before = first.backward(flat)
    second = batch.BatchRasterizer().plan(model, cams[:2], opts)
    second.backward(torch.ones_like(second.forward().color))
    assert torch.equal(first.forward().color, color)
    after = first.backward(flat)
    first.capture(flat)
    first.replay()
    torch.cuda.synchronize()
    for name in NAMES:
        assert rel_l2(getattr(after, name), getattr(before, name)) <= 2e-5, name
        assert rel_l2(getattr(first.grads, name), getattr(before, name)) <= 2e-5, name
