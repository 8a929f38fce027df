"""Readers of a framebuffer whose draws are still pending in the keys: pixels (aligned and unaligned
destinations) and the resolve give what they give after the draws were written to the layers first, on frames
that the scene covers in part, over a second draw, and for a depth-only view."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.helpers import GpuRenderer, TexturePair, default_lights, gpu_lights

pytestmark = pytest.mark.gpu
SIZES = [(4, 4), (12, 8), (260, 36), (324, 180)]


@pytest.fixture(scope="module")
def scene():
    sc = scenes.volume_scene(n=300, width=324, height=180, n_materials=2, extent=20.0, texture_size=64)
    texs = [TexturePair([sc.texture_pixels(i, 0), sc.texture_pixels(i, 1)], 64) for i in range(2)]
    return sc, GpuRenderer(sc.meshlets, sc.materials, [t.g for t in texs])


def _draw(sc, g, size, n, fb=None):
    v = scenes.make_view(*size, eye=(4.0, 3.0, -30.0), target=(0.0, 0.0, 0.0))
    return v, g.render(v.world_to_clip, *size, count=n, fb=fb, clear=(0xFF123456, 0.0))[0]


def _device(fb, layer, shift):
    import torch
    n = fb.width * fb.height
    buf = torch.full((n + 8,), -1, dtype=torch.int32, device="cuda")
    fb.get_pixels_device(layer, buf[shift:])
    out = buf.cpu().numpy()
    assert (out[:shift] == -1).all() and (out[n + shift:] == -1).all()
    return out[shift:n + shift].view(np.uint32).reshape(fb.height, fb.width)


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("shift", [0, 1, 4])
def test_pixels(scene, size, shift):
    sc, g = scene
    _, done = _draw(sc, g, size, 200)
    done.layer_data(0)  # writes the layers
    ids, depth = done.get_pixels(0), done.get_pixels(1)
    _, fb = _draw(sc, g, size, 200)
    for layer, want in ((1, depth), (0, ids), (1, depth)):
        assert np.array_equal(_device(fb, layer, shift), want)
        assert np.array_equal(fb.get_pixels(layer), want)
    _draw(sc, g, size, 300, fb=fb)  # over the pending draw
    _draw(sc, g, size, 300, fb=done)
    done.layer_data(0)
    assert np.array_equal(_device(fb, 0, shift), done.get_pixels(0))
    fb.layer_data(1)
    assert all(np.array_equal(_device(fb, k, shift), done.get_pixels(k)) for k in (0, 1))


@pytest.mark.parametrize("size", SIZES)
def test_resolve(scene, size):
    sc, g = scene
    api = g.api
    out = []
    for write in (False, True):
        v, fb = _draw(sc, g, size, 200)
        if write:
            fb.layer_data(0)
        ctx = api.ShadingContext(g.scene, v.world_to_clip, world_to_clip=v.world_to_clip, lights=gpu_lights(default_lights()),
                                 view_pos=(4.0, 3.0, -30.0))
        ctx.resolve(g.rast, fb)
        out.append((fb.get_pixels(0), fb.get_pixels(1)))
        _draw(sc, g, size, 300, fb=fb)  # from the depth layer
        out[-1] += (fb.get_pixels(0), fb.get_pixels(1))
    assert all(np.array_equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("depth_only", [False, True])
def test_batch_view(scene, depth_only):
    sc, g = scene
    api = g.api
    fbs = []
    for write in (False, True):
        fb = api.Framebuffer(324, 180)
        fb.clear(0xFF123456, 0.0)
        v = scenes.make_view(324, 180, eye=(4.0, 3.0, -30.0), target=(0.0, 0.0, 0.0))
        batch = api.Batch(g.rast, g.scene, [(fb, v.proj, v.view, np.eye(4, dtype=np.float32).ravel(), depth_only)])
        batch.render()
        if write:
            fb.layer_data(0)
        fbs.append((_device(fb, 0, 0), _device(fb, 1, 1), fb.get_pixels(0), fb.get_pixels(1)))
    assert all(np.array_equal(a, b) for a, b in zip(*fbs))
    assert (fbs[0][1] != 0).any()
