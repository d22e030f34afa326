"""The two layouts of the fused quantized SH Adam on degree-3 rows, a thread
per row (16-byte aligned state) and a half-warp per row (any alignment), on
row counts around the CTA size. Both evaluate the same expressions, but their
multiply-adds may round differently and the image gradients are summed by
float atomics: parameters within 1e-6, log bounds within 1e-5 (an ulp at 23 is
2e-6), first moments within one fp16 step at their size, codes within one
unit."""
import pytest
import torch

from helpers import camera_of, clone_model, device_model, gsb

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]


def unaligned(t):
    """A copy of t one element past an aligned address."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    out = flat[1:].view(t.shape)
    out.copy_(t)
    return out


@pytest.mark.parametrize("n", [1, 31, 127, 128, 129, 300])
def test_thread_rows_match_half_warp_rows(n):
    model = device_model(gsb.make_scene("tiny", seed=n, count=n))
    cam = camera_of(gsb.make_scene("tiny", seed=n, count=n))
    g = torch.Generator("cuda").manual_seed(n)
    first = (0.3 * torch.randn((n, 16, 3), device="cuda", generator=g)).half()
    packed = torch.randint(0, 256, (n, 16, 3), device="cuda", generator=g, dtype=torch.uint8)
    lo = 18 + torch.rand((n, 2), device="cuda", generator=g)
    bounds = torch.stack([lo[:, 0], lo[:, 0] + 2, lo[:, 1], lo[:, 1] + 3], 1).contiguous()
    grad = torch.randn((3, cam.height, cam.width), device="cuda", generator=g) * 1e-3
    out = []
    for move in (lambda t: t.clone(), unaligned):
        m = clone_model(model)
        m.sh = move(model.sh)
        st = dict(first=move(first), packed=move(packed), bounds=bounds.clone())
        rast = gsb.Rasterizer()
        r = rast.forward(m, cam, gsb.RasterizeOptions(active_sh_degree=3))
        rast.backward(m, r, grad, None,
                      sh_adam=gsb.SHAdamUpdate(**st, lr=5e-3, rest_lr=1e-3, correction1=0.8,
                                               correction2=0.3, regularization_weight=0.1))
        out.append((m.sh, st["first"].float(), st["packed"].int(), st["bounds"]))
    assert r.rendered_instances > 0
    (p0, f0, c0, b0), (p1, f1, c1, b1) = out
    assert float((p0 - p1).abs().max()) <= 1e-6
    assert float((b0 - b1).abs().max()) <= 1e-5
    assert bool(((f0 - f1).abs() <= 1e-3 * f0.abs() + 1e-7).all())
    assert int((c0 - c1).abs().max()) <= 1
    assert not torch.equal(p0, model.sh)


@pytest.mark.parametrize("move", [lambda t: t.clone(), unaligned])
def test_a_negative_regularization_factor_is_no_term(monkeypatch, move):
    """In both layouts; the C ABI takes the factor as it is (the Python layer
    passes none below 0)."""
    n = 200
    scene = gsb.make_scene("tiny", seed=4, count=n)
    cam = camera_of(scene)
    g = torch.Generator("cuda").manual_seed(4)
    state = dict(first=(0.3 * torch.randn((n, 16, 3), device="cuda", generator=g)).half(),
                 packed=torch.randint(0, 256, (n, 16, 3), device="cuda", generator=g,
                                      dtype=torch.uint8),
                 bounds=torch.tensor([18.0, 20.0, 18.0, 21.0], device="cuda").repeat(n, 1))
    grad = torch.randn((3, cam.height, cam.width), device="cuda", generator=g) * 1e-3

    class Negative(gsb._lib.ShAdam):
        def __setattr__(self, name, value):
            super().__setattr__(name, -0.5 if name == "regularization_factor" else value)

    out = []
    for cls in (gsb._lib.ShAdam, Negative):
        monkeypatch.setattr(gsb._lib, "ShAdam", cls)
        m = device_model(scene)
        m.sh = move(m.sh)
        st = {k: move(v) if k != "bounds" else v.clone() for k, v in state.items()}
        rast = gsb.Rasterizer()
        r = rast.forward(m, cam, gsb.RasterizeOptions(active_sh_degree=3))
        rast.backward(m, r, grad, None, sh_adam=gsb.SHAdamUpdate(
            **st, lr=5e-3, rest_lr=1e-3, correction1=0.8, correction2=0.3))
        out.append((m.sh, st["bounds"]))
    assert float((out[0][0] - out[1][0]).abs().max()) <= 1e-6
    assert float((out[0][1] - out[1][1]).abs().max()) <= 1e-5
