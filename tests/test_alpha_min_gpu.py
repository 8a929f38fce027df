"""Alpha-tested materials whose textures hold no texel below the cutoff draw as opaque ones do (the textures
keep the least alpha of each level): bit for bit the oracle's alpha test, for least alphas around the cutoff,
through every way texels are written, and after they change under an unchanged material."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.helpers import GpuRenderer, TexturePair, assert_visbuffer_equal, render_oracle

pytestmark = pytest.mark.gpu
SIZE = 64


def _pixels(least, seed=3):
    rng = np.random.default_rng(seed)
    p = scenes.value_noise_rgba(SIZE, seed, cells=8, layer=0).astype(np.uint32) & 0x00FFFFFF
    a = rng.integers(least, 256, (SIZE, SIZE)).astype(np.uint32)
    a[SIZE // 2, SIZE // 3] = least
    return p | (a << 24)


@pytest.fixture(scope="module")
def scene():
    sc = scenes.volume_scene(n=2000, width=324, height=180, n_materials=2, extent=12.0, texture_size=SIZE, alpha_every=2)
    texs = [TexturePair([_pixels(0)], SIZE), TexturePair([_pixels(0, 4)], SIZE)]
    view = scenes.make_view(324, 180, eye=(0.0, 0.0, 0.0), target=(0.3, 0.1, 1.0))
    return sc, texs, GpuRenderer(sc.meshlets, sc.materials, [t.g for t in texs]), view


def _write(t, px, how):
    t.o.set_pixels(px, 0)
    t.o.generate_mips()
    if how == "device":
        import torch
        d = torch.from_numpy(px.astype(np.uint32).view(np.int32)).cuda()
        t.g.set_pixels_device(d)
        torch.cuda.synchronize()
    elif how == "host":
        t.g.set_pixels(px)
    if how == "data":
        t.g.set_data(t.o.data[: t.g.words])
    else:
        t.g.generate_mips()


@pytest.mark.parametrize("how", ["host", "device", "data"])
def test_least_alpha_around_the_cutoff(scene, how):
    sc, texs, g, view = scene
    cutoff = int(sc.materials["alpha_cutoff"][0])
    shown = []
    for least in (cutoff, cutoff - 1, 255, 0, cutoff + 1):  # rises and falls under the same materials
        _write(texs[0], _pixels(least), how)
        gfb, gc = g.render(view.world_to_clip, view.width, view.height, binning=False)
        ofb, oc = render_oracle(sc.meshlets, sc.materials, view.world_to_clip, view.width, view.height, binning=False,
                                textures=[t.o for t in texs])
        assert_visbuffer_equal(gfb, ofb)
        assert list(gc[:3]) == list(oc[:3])
        shown.append(gfb.get_pixels(0))
    assert np.array_equal(shown[0], shown[2]) and np.any(shown[0] != shown[3])


def test_pixels_without_new_mips(scene):
    """Level 0 turns opaque while the other levels keep their holes, and the other way round."""
    sc, texs, g, view = scene
    for first, then in ((0, 255), (255, 0)):
        _write(texs[0], _pixels(first), "host")
        texs[0].g.set_pixels(_pixels(then))
        texs[0].o.set_pixels(_pixels(then), 0)
        for eye in ((0.0, 0.0, 0.0), (0.0, 0.0, -60.0)):  # magnified and minified
            v = scenes.make_view(324, 180, eye=eye, target=(0.3, 0.1, 1.0))
            gfb, _ = g.render(v.world_to_clip, v.width, v.height)
            ofb, _ = render_oracle(sc.meshlets, sc.materials, v.world_to_clip, v.width, v.height, textures=[t.o for t in texs])
            assert_visbuffer_equal(gfb, ofb)
