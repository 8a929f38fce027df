"""Batches against the oracle, view by view bit for bit, and their processed, rasterized and clipped counters against the
sum over the views: dense views (their groups overflow the blocks' pools), culled ones, views up to and past the
number a pool's word can name, with and without clipping, and with alpha-tested materials."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.helpers import GpuRenderer, TexturePair, assert_visbuffer_equal, render_oracle

pytestmark = pytest.mark.gpu


def _batch(sc, texs, size, eyes, binning, cull, repeat=2):
    from glimpsw_gb300 import api
    from oracle import oracle as O
    api.load_library()
    g = GpuRenderer(sc.meshlets, sc.materials, [t.g for t in texs])
    n = len(sc.meshlets)
    vs = [scenes.make_view(*size, eye=e, target=(0.0, 0.0, 0.0)) for e in eyes]
    fbs = [api.Framebuffer(*size) for _ in vs]
    g.rast.EnableBinning = binning
    b = api.Batch(g.rast, g.scene, [(fb, v.proj, v.view, scenes.IDENTITY, False) for fb, v in zip(fbs, vs)], frustum_cull=cull)
    total = np.zeros(3, np.uint64)
    oracle = []
    for v in vs:
        bits = None
        if cull:
            bits, _ = O.cull_meshlets(sc.meshlets, n, v.proj, v.view, scenes.IDENTITY, v.view, *size, None)
        ofb, c = render_oracle(sc.meshlets, sc.materials, v.world_to_clip, *size, cull_bitmap=bits, binning=binning,
                               textures=[t.o for t in texs])
        total += np.asarray(c[:3], np.uint64)
        oracle.append(ofb)
    for _ in range(repeat):
        b.reset_counters()
        b.render()
        assert list(b.counters()[:3]) == list(total)
        for i, (fb, ofb) in enumerate(zip(fbs, oracle)):
            assert_visbuffer_equal(fb, ofb)


@pytest.mark.parametrize("binning", [False, True])
@pytest.mark.parametrize("cull", [False, True])
@pytest.mark.parametrize("count,views", [(31, 1), (400, 3), (5000, 5)])
def test_few_views(count, views, cull, binning):
    sc = scenes.volume_scene(n=count, width=64, height=36, n_materials=1, extent=8.0, texture_size=64)
    _batch(sc, [], (132, 76), [(np.sin(i) * 6.0, 1.0, -5.0 + np.cos(i)) for i in range(views)], binning, cull)


@pytest.mark.parametrize("views", [2046, 2047, 2050])
def test_many_views(views):
    sc = scenes.volume_scene(n=33, width=64, height=36, n_materials=1, extent=6.0, texture_size=64)
    _batch(sc, [], (8, 4), [(np.sin(i) * 9.0, 1.0, -9.0 + np.cos(i)) for i in range(views)], False, False, repeat=1)


def test_alpha_tested():
    sc = scenes.volume_scene(n=3000, width=64, height=36, n_materials=2, extent=12.0, texture_size=64, alpha_every=2)
    texs = [TexturePair([sc.texture_pixels(i, 0)], 64) for i in range(2)]
    _batch(sc, texs, (132, 76), [(np.sin(i) * 9.0, 1.0, -7.0 + np.cos(i)) for i in range(4)], False, True)
