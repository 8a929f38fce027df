"""Meshlets passed between the warps of a block and shared alpha-tested ones, bit for bit against the oracle with the
same counters: dense and clustered bitmaps (groups of many visible meshlets, also where they overflow the
block's pool), many views in a batch up to and past the number a pool's word can name, and alpha passes of
fewer meshlets than warps, up to four times as many, and more."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.helpers import GpuRenderer, TexturePair, assert_visbuffer_equal, render_oracle

pytestmark = pytest.mark.gpu
W, H, N = 324, 180, 12_000


@pytest.fixture(scope="module")
def scene():
    sc = scenes.volume_scene(n=N, width=W, height=H, n_materials=1, extent=30.0, texture_size=64)
    view = scenes.make_view(W, H, eye=(0.0, 0.0, -20.0), target=(0.0, 0.0, 0.0))
    return sc, GpuRenderer(sc.meshlets, sc.materials), view


@pytest.mark.parametrize("bits", ["all", "half", "clusters", "most"])
def test_bitmaps(scene, bits):
    import torch
    sc, g, view = scene
    rng = np.random.default_rng(3)
    on = {"all": np.ones(N, bool), "half": rng.uniform(size=N) < 0.5, "most": rng.uniform(size=N) < 0.95,
          "clusters": (np.arange(N) // 500) % 3 == 0}[bits]
    padded = np.zeros((N + 31) // 32 * 32, dtype=np.uint8)
    padded[:N] = on
    words = np.packbits(padded, bitorder="little").view(np.uint16)
    dev = torch.from_numpy(words.view(np.int16).copy()).cuda()
    gfb, gc = g.render(view.world_to_clip, W, H, cull_bitmap=dev)
    ofb, oc = render_oracle(sc.meshlets, sc.materials, view.world_to_clip, W, H, cull_bitmap=words)
    assert_visbuffer_equal(gfb, ofb)
    assert list(gc[:3]) == list(oc[:3])


@pytest.mark.parametrize("views", [3, 2046, 2047, 2050])
def test_many_views(views):
    from glimpsw_gb300 import api
    api.load_library()
    count = 400 if views < 100 else 33
    sc = scenes.volume_scene(n=count, width=64, height=36, n_materials=1, extent=6.0, texture_size=64)
    g = GpuRenderer(sc.meshlets, sc.materials)
    size = (64, 36) if views < 100 else (8, 4)
    vs = [scenes.make_view(*size, eye=(np.sin(i) * 9.0, 1.0, -9.0 + np.cos(i)), target=(0.0, 0.0, 0.0)) for i in range(views)]
    fbs = [api.Framebuffer(*size) for _ in vs]
    for fb in fbs:
        fb.clear(0xFF000000, 0.0)
    ident = np.eye(4, dtype=np.float32).ravel()
    g.rast.EnableBinning = False  # as the single draws
    api.Batch(g.rast, g.scene, [(fb, v.proj, v.view, ident, False) for fb, v in zip(fbs, vs)], frustum_cull=False).render()
    for i in list(range(0, views, max(1, views // 20))) + [views - 1]:
        single, _ = g.render(vs[i].world_to_clip, *size)
        for layer in (0, 1):
            assert np.array_equal(fbs[i].get_pixels(layer), single.get_pixels(layer)), i


@pytest.mark.parametrize("n", [600, 9_000, 20_000, 44_000])
def test_alpha_counts(n):
    sc = scenes.volume_scene(n=n, width=W, height=H, n_materials=2, extent=40.0, texture_size=64, alpha_every=2)
    texs = [TexturePair([sc.texture_pixels(i, 0)], 64) for i in range(2)]
    g = GpuRenderer(sc.meshlets, sc.materials, [t.g for t in texs])
    v = scenes.make_view(W, H, eye=(0.0, 0.0, -25.0), target=(0.0, 0.0, 0.0))
    gfb, gc = g.render(v.world_to_clip, W, H)
    ofb, oc = render_oracle(sc.meshlets, sc.materials, v.world_to_clip, W, H, textures=[t.o for t in texs])
    assert_visbuffer_equal(gfb, ofb)
    assert list(gc[:3]) == list(oc[:3])
