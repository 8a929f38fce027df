"""Draws on both sides of the number of positions from which a pass's first groups are the warps' own (16 positions for
each of 32 warps a multiprocessor), with and without a cull bitmap: bit for bit against the oracle with the same
counters."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.helpers import GpuRenderer, assert_visbuffer_equal, render_oracle

pytestmark = pytest.mark.gpu
W, H, BASE = 64, 36, 4000


@pytest.fixture(scope="module")
def scene():
    import torch
    line = 16 * 32 * torch.cuda.get_device_properties(0).multi_processor_count
    sc = scenes.volume_scene(n=BASE, width=W, height=H, n_materials=1, extent=14.0, texture_size=64)
    raw = sc.meshlets.view(np.uint8).reshape(BASE, -1)
    m = np.ascontiguousarray(raw[np.arange(line + 100) % BASE]).view(scenes.MESHLET_DTYPE).ravel()
    view = scenes.make_view(W, H, eye=(0.0, 0.0, -18.0), target=(0.3, 0.1, 1.0))
    return sc, m, GpuRenderer(m, sc.materials), view, line


@pytest.mark.parametrize("offset", [-1, 0, 1, 65])
@pytest.mark.parametrize("bitmap", [False, True])
def test_line(scene, bitmap, offset):
    import torch
    sc, m, g, view, line = scene
    count = line + offset
    words = dev = None
    if bitmap:
        on = np.zeros((count + 31) // 32 * 32, dtype=np.uint8)
        on[:count] = np.random.default_rng(offset + 2).uniform(size=count) < 0.5
        words = np.packbits(on, bitorder="little").view(np.uint16)
        dev = torch.from_numpy(words.view(np.int16).copy()).cuda()
    gfb, gc = g.render(view.world_to_clip, W, H, count=count, cull_bitmap=dev)
    ofb, oc = render_oracle(m, sc.materials, view.world_to_clip, W, H, count=count, cull_bitmap=words)
    assert_visbuffer_equal(gfb, ofb)
    assert list(gc[:3]) == list(oc[:3])
