"""Batched rendering where plans meet: several plans alive at once, and views
of enough tiles (above 4,800 of 16x16) that four pixels per thread run as
eight, against the single-view path (tolerances of test_gpu_batch.py)."""
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


@pytest.mark.parametrize("tw,th,sched,capacity", [
    (16, 16, "dynamic", 0), (16, 32, "static", 0),
    (16, 16, "heavy_first", 0),        # the order lists in a buffer of their own
    (16, 32, "heavy_first", 1 << 21),  # the order lists in the sort's spare keys
])
def test_eight_pixels_per_thread_match_single_views(tw, th, sched, capacity):
    sizes = ((701, 903), (803, 717), (333, 211))
    model, cams = _setup(4000, 6, sizes, 4)
    tiles16 = sum(-(-c.width // 16) * -(-c.height // 16) for c in cams)
    tiles = sum(-(-c.width // tw) * -(-c.height // th) for c in cams)
    assert tiles * tw * th // 256 > 4800 and tiles16 > 4800
    opts = gsb.RasterizeOptions(active_sh_degree=3)
    br = batch.BatchRasterizer().plan(model, cams, opts, batch.BatchSchedule(tw, th, 4, sched),
                                      instance_capacity=capacity)
    res = br.forward()
    g = torch.Generator("cuda").manual_seed(2)
    flat = torch.randn(res.color.numel(), device="cuda", generator=g) * 1e-3
    grads = br.backward(flat)
    info = br.info()
    assert info["overflow"] == 0 and info["device_error"] == 0
    # counts and lists of both orders: 64 classes of the tiles and of the strips
    strips = th // 16 * tiles
    assert sched != "heavy_first" or \
        (64 * (tiles + strips) <= info["instance_capacity"]) == (capacity > 0)
    rast, total = gsb.Rasterizer(), {}
    for k, cam in enumerate(cams):
        r = rast.forward(model, cam, opts)
        assert float((res.view_color(k) - r.color).abs().max()) <= 1e-6
        assert float((res.view_alpha(k) - r.alpha).abs().max()) <= 1e-6
        w, h, off = res.views[k]
        one = rast.backward(model, r, flat[3 * off:3 * (off + w * h)].view(3, h, w).contiguous())
        for name in NAMES:
            total[name] = total.get(name, 0) + getattr(one, name)
    for name in NAMES:
        assert rel_l2(getattr(grads, name), total[name]) <= 2e-5, name
