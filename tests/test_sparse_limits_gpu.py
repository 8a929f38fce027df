"""Sparse draws on both sides of each of the rule's limits: numbers of positions around 40 and 64 a warp and shares of
visible ones around 4, 12 and 32 in 1024, bit for bit against the oracle with the same counters."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.helpers import GpuRenderer, assert_visbuffer_equal, render_oracle

pytestmark = pytest.mark.gpu
W, H, BASE = 324, 180, 4000


@pytest.fixture(scope="module")
def scene():
    import torch
    warps = 32 * torch.cuda.get_device_properties(0).multi_processor_count
    n = 64 * warps + 1000
    sc = scenes.volume_scene(n=BASE, width=W, height=H, n_materials=1, extent=14.0, texture_size=64)
    raw = sc.meshlets.view(np.uint8).reshape(BASE, -1)
    m = np.ascontiguousarray(raw[np.arange(n) % BASE]).view(scenes.MESHLET_DTYPE).ravel()
    view = scenes.make_view(W, H, eye=(0.0, 0.0, -18.0), target=(0.3, 0.1, 1.0))
    return sc, m, GpuRenderer(m, sc.materials), view, warps


@pytest.mark.parametrize("share", [3, 5, 11, 13, 31, 34])
@pytest.mark.parametrize("per_warp", [8, 40, 64])
@pytest.mark.parametrize("more", [0, 1])
def test_limits(scene, per_warp, more, share):
    import torch
    sc, m, g, view, warps = scene
    count = per_warp * warps + more * 33
    on = np.zeros((count + 31) // 32 * 32, dtype=np.uint8)
    on[:count] = np.random.default_rng(count + share).uniform(size=count) < share / 1024
    words = np.packbits(on, bitorder="little").view(np.uint16)
    dev = torch.from_numpy(words.view(np.int16).copy()).cuda()
    gfb, gc = g.render(view.world_to_clip, W, H, count=count, cull_bitmap=dev)
    ofb, oc = render_oracle(m, sc.materials, view.world_to_clip, W, H, count=count, cull_bitmap=words)
    assert_visbuffer_equal(gfb, ofb)
    assert list(gc[:3]) == list(oc[:3])
