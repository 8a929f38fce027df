"""Draws of more positions than the GPU has warps whose cull bitmap holds few of them, and the change to dense
ones: bit for bit the oracle's image and counters for shares of visible meshlets around the sampled limit
(one in 32), none at all, and bitmaps whose visible meshlets the sample misses or alone meets."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.helpers import GpuRenderer, assert_visbuffer_equal, render_oracle

pytestmark = pytest.mark.gpu
W, H, N = 324, 180, 12_000


@pytest.fixture(scope="module")
def scene():
    sc = scenes.volume_scene(n=N, width=W, height=H, n_materials=1, extent=14.0, texture_size=64)
    view = scenes.make_view(W, H, eye=(0.0, 0.0, 0.0), target=(0.3, 0.1, 1.0))
    return sc, GpuRenderer(sc.meshlets, sc.materials), view


def _sampled(count):
    """The words of the bitmap that the draw samples."""
    return (np.arange(64, dtype=np.int64) * (count >> 4)) >> 6


@pytest.mark.parametrize("bits", ["none", "one", "1/1000", "1/33", "1/31", "1/8", "missed", "met"])
@pytest.mark.parametrize("count", [N, N - 7, 9999])
def test_shares(scene, bits, count):
    import torch
    sc, g, view = scene
    rng = np.random.default_rng(count)
    if bits in ("missed", "met"):
        words = np.zeros((count + 31) // 32 * 2, dtype=np.uint16)
        if bits == "missed":  # dense all over but where the sample looks
            words[: count >> 4] = 0x5555
            words[_sampled(count)] = 0
        else:
            words[_sampled(count)] = 0xFFFF
    else:
        share = {"none": 0.0, "one": 0.0, "1/1000": 1e-3, "1/33": 1 / 33, "1/31": 1 / 31, "1/8": 1 / 8}[bits]
        on = np.zeros((count + 31) // 32 * 32, dtype=np.uint8)
        on[:count] = rng.uniform(size=count) < share
        if bits == "one":
            on[count - 1] = 1
        words = np.packbits(on, bitorder="little").view(np.uint16)
    dev = torch.from_numpy(words.view(np.int16).copy()).cuda()
    gfb, gc = g.render(view.world_to_clip, W, H, count=count, cull_bitmap=dev)
    ofb, oc = render_oracle(sc.meshlets, sc.materials, view.world_to_clip, W, H, count=count, cull_bitmap=words)
    assert_visbuffer_equal(gfb, ofb)
    assert list(gc[:3]) == list(oc[:3])
