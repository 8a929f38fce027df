"""The resolve's per-lane surface and material handling against the oracle: tiles whose pixels mix materials
with textures of different sizes (the filter is chosen per material over the whole tile), one and two
layers, meshlets without a material, and light counts on both sides of what the kernel's parameters hold.
The bounds are the resolve's contract (tests/test_shade_gpu.py): 1/255, and 99.9 % of the pixels equal."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.helpers import GpuRenderer, TexturePair, gpu_lights, make_light, render_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mixed():
    sc = scenes.volume_scene(n=6000, width=324, height=180, n_materials=4, extent=40.0, texture_size=64, env_size=128)
    meshlets = sc.meshlets.copy()
    meshlets["MaterialId"][::11] = 0xFFFFFFFF
    sizes = [(64, 2), (512, 2), (16, 1), (128, 2)]
    texs = [TexturePair([scenes.value_noise_rgba(s, 40 + i, cells=8, layer=k) for k in range(n)], s)
            for i, (s, n) in enumerate(sizes)]
    env = TexturePair([scenes.env_map_r11g11b10(128, 5)], 128, fmt=1)
    return sc, meshlets, texs, env, GpuRenderer(meshlets, sc.materials, [t.g for t in texs])


def _lights(n):
    rng = np.random.default_rng(n)
    out = [make_light(0, direction=(0.3, -0.8, 0.5), intensity=900.0)]
    for i in range(1, n):
        out.append(make_light(1 + i % 2, position=rng.uniform(-30, 30, 3), direction=rng.normal(size=3), color=rng.uniform(0.2, 1, 3),
                              intensity=1.0e5, radius=40.0, inner=0.3, outer=0.9))
    return np.concatenate(out[:n]) if n else np.zeros(0, dtype=make_light(0).dtype)


@pytest.mark.parametrize("lights", [0, 1, 16, 17])
def test_mixed_materials_and_light_counts(mixed, lights):
    from glimpsw_gb300 import api
    from oracle import oracle as O
    sc, meshlets, texs, env, g = mixed
    v, ls = sc.views[0], _lights(lights)
    w, h = v.width, v.height
    gfb, _ = g.render(v.world_to_clip, w, h)
    ofb, _ = render_oracle(meshlets, sc.materials, v.world_to_clip, w, h)
    O.resolve(ofb, O.Context(meshlets, sc.materials, v.world_to_clip, world_to_clip=v.world_to_clip,
                             textures=[t.o for t in texs], lights=ls, skybox=env.o, view_pos=v.eye), threads=8)
    api.ShadingContext(g.scene, v.world_to_clip, world_to_clip=v.world_to_clip, skybox=env.g, view_pos=v.eye,
                       lights=gpu_lights(ls)).resolve(g.rast, gfb)
    a = gfb.get_pixels(0).view(np.uint8).reshape(h, w, 4).astype(np.int32)
    b = ofb.get_pixels(0).view(np.uint8).reshape(h, w, 4).astype(np.int32)
    diff = np.abs(a - b)
    assert diff.max() <= 1
    assert (diff.max(axis=2) == 0).mean() > 0.999
