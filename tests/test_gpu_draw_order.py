"""The draw list's order over the digit plans of its two sorts (depth bits and
tile bits cut into digits of up to 9 bits) and around the 3,072-key sort tiles:
(tile, depth bits, Gaussian index) ascending, every instance once, tile ranges
matching. Integer work: exact."""
import dataclasses

import pytest
import torch

from helpers import camera_of, device_model, gsb

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]


@pytest.mark.parametrize("n,w,h,depths", [
    (1, 16, 16, None),          # one key, one tile bit
    (3071, 64, 64, "equal"),    # one depth: ties by index; 5 tile bits
    (3072, 352, 336, None),     # a full sort tile; 9 tile bits in one pass
    (3073, 368, 368, "two"),    # 10 tile bits in 5 + 5
    (6145, 1000, 900, None),    # 12 tile bits
    (70000, 4100, 2100, "far"), # 16 tile bits in 8 + 8; 27 or more depth bits
])
def test_draw_list_is_sorted_and_complete(n, w, h, depths):
    f = 0.8 * w
    scene = dataclasses.replace(gsb.make_scene("small", seed=n, count=n), width=w, height=h,
                                cx=w / 2.0, cy=h / 2.0, fx=f, fy=f)
    model = device_model(scene)
    if depths == "far":  # depths from 0.3 to 3e4
        g = torch.Generator("cuda").manual_seed(n)
        scale = torch.exp(torch.rand((n, 1), device="cuda", generator=g) * 11.5) * 0.1
        model.means = (model.means * scale).contiguous()
    elif depths:  # radial depths on one or two exact values
        model.means = torch.zeros_like(model.means)
        model.means[:, 2] = 4.0
        if depths == "two":
            model.means[1::3, 2] = 5.0
    r = gsb.Rasterizer().forward(model, camera_of(scene), gsb.RasterizeOptions(active_sh_degree=3))
    keys, vals, ranges = gsb.draw_list(r)
    count = keys.numel()
    assert count == r.rendered_instances > 0
    step = keys[1:] - keys[:-1]
    assert bool((step >= 0).all())
    assert bool((vals[1:] > vals[:-1])[step == 0].all())  # equal keys by index, no repeats
    tiles = keys >> 32
    present, counts = torch.unique_consecutive(tiles, return_counts=True)
    starts = torch.cumsum(counts, 0) - counts
    assert torch.equal(ranges[present, 0].long(), starts)
    assert torch.equal(ranges[present, 1].long(), starts + counts)
    empty = torch.ones(ranges.shape[0], dtype=torch.bool, device="cuda")
    empty[present] = False
    assert bool((ranges[empty, 0] == ranges[empty, 1]).all())
    depth = torch.linalg.vector_norm(model.means[vals.long()].double(), dim=1)
    stored = (keys & 0xffffffff).int().view(torch.float32).double()
    assert bool(((stored - depth).abs() <= 1e-6 * depth).all())
