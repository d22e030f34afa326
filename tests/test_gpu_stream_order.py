"""A native context that moves between streams: the next stream waits for the
work it was left with, and nothing of an old stream is touched any more."""
import pytest
import torch

from helpers import camera_of, device_model, gsb

pytestmark = [pytest.mark.gpu,
              pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

OPTIONS = gsb.RasterizeOptions(active_sh_degree=3)


@pytest.fixture
def one_context(monkeypatch):
    """Every pass of the test takes the same context."""
    index = torch.cuda.current_device()
    monkeypatch.setitem(gsb.rasterizer._POOLS, index, gsb.rasterizer._ContextPool(index))


def _scene(seed):
    scene = gsb.make_scene("small", seed=seed)
    return device_model(scene), camera_of(scene)


def test_next_stream_waits_for_a_backward_in_flight(one_context):
    (model, cam), (other, _) = _scene(0), _scene(1)
    rast = gsb.Rasterizer()
    r = rast.forward(model, cam, OPTIONS)
    gc = torch.full_like(r.color, 1e-3)
    expect = rast.backward(model, r, gc)
    native = r.context.ctx.ptr.value
    del r
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        r = rast.forward(model, cam, OPTIONS)
        torch.cuda._sleep(40_000_000)  # some 20 ms: the adjoint starts after it
        got = rast.backward(model, r, gc)
        del r
    with torch.cuda.stream(b):
        r = rast.forward(other, cam, OPTIONS)
        assert r.context.ctx.ptr.value == native
    torch.cuda.synchronize()
    for name in ("means", "log_scales", "quaternions", "opacity_logits", "sh", "refine_weight"):
        x, y = getattr(got, name), getattr(expect, name)
        assert float((x - y).abs().max()) <= 1e-4 * float(y.abs().max()), name


def test_render_beside_a_capture_on_the_last_stream(one_context):
    """The stream that used the context last is being captured; a render on
    another stream takes no part in the capture."""
    model, cam = _scene(2)
    rast = gsb.Rasterizer()
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        expect = rast.forward(model, cam, OPTIONS).color.clone()
    torch.cuda.synchronize()
    x = torch.zeros(64, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=a, capture_error_mode="relaxed"):
        x.add_(1)
        with torch.cuda.stream(b):
            got = rast.forward(model, cam, OPTIONS).color
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, expect)
    assert bool((x == 1).all())
