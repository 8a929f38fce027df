"""Vertex normals and tangents from the scene's table: random words (all 65,536 codes come up) shade as the oracle
does, and a scene without meshlets, which has no table, resolves as one with meshlets that are not drawn.
The bounds are the resolve's contract (tests/test_shade_gpu.py): 1/255, and 99.9 % of the pixels equal."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.helpers import GpuRenderer, TexturePair, default_lights, gpu_lights, render_oracle

pytestmark = pytest.mark.gpu


def test_random_normals():
    from glimpsw_gb300 import api
    from oracle import oracle as O
    sc = scenes.volume_scene(n=3000, width=640, height=360, n_materials=2, extent=20.0, texture_size=64)
    rng = np.random.default_rng(11)
    sc.meshlets["NormalTangents"] = rng.integers(0, 1 << 32, sc.meshlets["NormalTangents"].shape, dtype=np.uint64).astype(np.uint32)
    texs = [TexturePair([sc.texture_pixels(i, 0), sc.texture_pixels(i, 1)], 64) for i in range(2)]
    g = GpuRenderer(sc.meshlets, sc.materials, [t.g for t in texs])
    v = scenes.make_view(640, 360, eye=(0.0, 0.0, -30.0), target=(0.0, 0.0, 0.0))
    gfb, _ = g.render(v.world_to_clip, 640, 360)
    ofb, _ = render_oracle(sc.meshlets, sc.materials, v.world_to_clip, 640, 360, threads=8)
    lights = default_lights()
    api.ShadingContext(g.scene, v.world_to_clip, world_to_clip=v.world_to_clip, view_pos=v.eye,
                       lights=gpu_lights(lights)).resolve(g.rast, gfb)
    O.resolve(ofb, O.Context(sc.meshlets, sc.materials, v.world_to_clip, world_to_clip=v.world_to_clip,
                             textures=[t.o for t in texs], lights=lights, view_pos=v.eye))
    a = gfb.get_pixels(0).view(np.uint8).astype(np.int32)
    b = ofb.get_pixels(0).view(np.uint8).astype(np.int32)
    assert np.abs(a - b).max() <= 1
    assert (gfb.get_pixels(0) == ofb.get_pixels(0)).mean() > 0.999


@pytest.mark.parametrize("depth", [0.0, 0.5])
def test_scene_without_meshlets(depth):
    from glimpsw_gb300 import api
    api.load_library()
    sc = scenes.volume_scene(n=4, width=64, height=36, n_materials=1, extent=4.0, texture_size=64)
    v = sc.views[0]
    full = GpuRenderer(sc.meshlets, sc.materials)
    empty = api.Scene()
    out = []
    for scene in (full.scene, empty):
        fb = api.Framebuffer(64, 36)
        fb.clear(0xFF000000, depth)
        api.ShadingContext(scene, v.world_to_clip, world_to_clip=v.world_to_clip, view_pos=v.eye,
                           lights=gpu_lights(default_lights())).resolve(full.rast, fb)
        out.append(fb.get_pixels(0))
    assert np.array_equal(*out)
