"""Draws of fewer meshlets than the GPU has warps, whose meshlets are shared by up to 32 warps each, and draws
of a little more: bit for bit the oracle's image and counters, for counts around every change of the share, with
cull bitmaps, alpha-tested materials, clipped triangles, a meshlet offset and draws after one another."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.helpers import GpuRenderer, TexturePair, assert_visbuffer_equal, render_oracle

pytestmark = pytest.mark.gpu
W, H = 252, 140


@pytest.fixture(scope="module")
def scene():
    sc = scenes.volume_scene(n=5000, width=W, height=H, n_materials=2, extent=14.0, texture_size=64, alpha_every=2)
    texs = [TexturePair([sc.texture_pixels(i, 0)], 64) for i in range(2)]
    view = scenes.make_view(W, H, eye=(0.0, 0.0, 0.0), target=(0.3, 0.1, 1.0))
    return sc, texs, GpuRenderer(sc.meshlets, sc.materials, [t.g for t in texs]), view


def _warps():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count * 32


def _bitmap(count, every, offset=0):
    bits = np.zeros((count + 31) // 32 * 32, dtype=np.uint8)
    bits[offset:count:every] = 1
    return np.packbits(bits, bitorder="little").view(np.uint16)


def _check(scene, count, bitmap=None, **kw):
    import torch
    sc, texs, g, view = scene
    dev = None if bitmap is None else torch.from_numpy(bitmap.view(np.int16).copy()).cuda()
    gfb, gc = g.render(view.world_to_clip, W, H, count=count, cull_bitmap=dev, **kw)
    ofb, oc = render_oracle(sc.meshlets, sc.materials, view.world_to_clip, W, H, count=count, cull_bitmap=bitmap,
                            textures=[t.o for t in texs], **kw)
    assert_visbuffer_equal(gfb, ofb)
    assert list(gc[:3]) == list(oc[:3])


@pytest.mark.parametrize("part", ["1", "2", "/32", "/32+1", "/16", "/8+1", "/4", "/2", "/2+1", "-1", "+0", "+1"])
@pytest.mark.parametrize("clipping", [True, False])
def test_counts(scene, part, clipping):
    n = _warps()
    count = int(part) if part in ("1", "2") else (n // int(part[1:].split("+")[0]) + (1 if part.endswith("+1") else 0)
                                                  if part[0] == "/" else n + int(part))
    _check(scene, min(count, 5000), clipping=clipping)


@pytest.mark.parametrize("count,offset", [(40, 3000), (700, 100), (4000, 1000), (5000, 0)])
@pytest.mark.parametrize("every", [1, 3, 50])
def test_bitmaps_and_offsets(scene, count, offset, every):
    _check(scene, count, _bitmap(count, every), meshlet_offset=offset)


def test_draws_after_one_another(scene):
    sc, texs, g, view = scene
    gfb = ofb = None
    for offset, count in ((0, 30), (30, 4900), (4930, 70)):
        gfb, _ = g.render(view.world_to_clip, W, H, count=count, meshlet_offset=offset, fb=gfb)
        ofb, _ = render_oracle(sc.meshlets, sc.materials, view.world_to_clip, W, H, count=count, meshlet_offset=offset, fb=ofb,
                               textures=[t.o for t in texs])
    assert_visbuffer_equal(gfb, ofb)


@pytest.mark.parametrize("capacity", [1, 2, 13])
def test_full_queue(scene, capacity):
    g = scene[2]
    g.rast.set_queue_capacity(capacity)
    try:
        _check(scene, 60)
    finally:
        g.rast.set_queue_capacity(0)
