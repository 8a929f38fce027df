"""The neural resolve's pixel records and request counts at material counts around a counter line (32) and past the
number of copies, and frames of one tile, of part of a block and of many blocks: with materials of one colour
per layer, whose networks give that colour, the image equals the plain resolve's, magnified (shared quads) and
minified (nearest texels), and the counts add up."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from oracle import neural as N
from tests.helpers import GpuRenderer, default_lights, gpu_lights
from tests.test_neural_gpu import LEVELS, SIZE, _device_texture, _setup_stream

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[1, 31, 32, 33, 70])
def colours(request):
    api = _setup_stream()
    count = request.param
    sc = scenes.volume_scene(n=1500, width=320, height=180, n_materials=count, extent=20.0, texture_size=SIZE)
    rng = np.random.default_rng(count)
    cols = rng.integers(0, 256, (count, 2, 4)).astype(np.uint32)
    cols[:, 0, 3] = 255
    words = cols[..., 0] | (cols[..., 1] << 8) | (cols[..., 2] << 16) | (cols[..., 3] << 24)
    texs = [_device_texture([np.full((SIZE, SIZE), words[i, l], np.uint32) for l in range(2)]) for i in range(count)]
    m = api.NeuralMaterials(texs, latent_levels=LEVELS, seed=3)
    for i in range(count):
        p = np.zeros(N.PARAMS, np.float32)
        p[N.PB3:N.PARAMS] = np.concatenate([cols[i, 0, :3], cols[i, 1, :4], [255]]) / np.float32(255.0)
        m.set_params(i, p)
    return api, m, GpuRenderer(sc.meshlets, sc.materials, texs), texs


@pytest.mark.parametrize("size", [(4, 4), (20, 12), (324, 180)])
@pytest.mark.parametrize("eye", [(0.0, 0.0, 0.0), (0.0, 0.0, -60.0)])
def test_constant_materials(colours, size, eye):
    api, m, g, _ = colours
    v = scenes.make_view(*size, eye=eye, target=(0.5, 0.2, 1.0))
    ctx = api.ShadingContext(g.scene, v.world_to_clip, world_to_clip=v.world_to_clip, view_pos=v.eye, lights=gpu_lights(default_lights()))
    a, _ = g.render(v.world_to_clip, *size)
    b, _ = g.render(v.world_to_clip, *size)
    ctx.resolve(g.rast, a)
    requests, tiles, per_level = ctx.resolve_neural(g.rast, b, m, want_stats=True)
    assert sum(per_level) == requests and tiles * 128 >= requests
    assert np.array_equal(a.get_pixels(0), b.get_pixels(0))
    assert np.array_equal(a.get_pixels(1), b.get_pixels(1))
