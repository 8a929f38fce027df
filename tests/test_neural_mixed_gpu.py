"""The neural resolve on tiles that mix decoded pixels with pixels of plain textures, so that the second pass
reconstructs the surface instead of reading the emit pass's records: materials the model does not have (none, or past its
last), a scene texture of another size than the model's, one without a second layer, one without any texture, and
texture levels above the latents'. Decoded materials are of one colour per layer, which their networks give; what
is not decoded has texels of its own, in the deeper levels too. The image equals the plain resolve's."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from oracle import neural as N
from tests.helpers import GpuRenderer, default_lights, gpu_lights
from tests.test_neural_gpu import _device_texture, _setup_stream

pytestmark = pytest.mark.gpu
SIZE, LATENTS = 64, 1  # levels 0 to 2 of 5 are decoded
DECODED = LATENTS + 2


def _words(c):
    return c[..., 0] | (c[..., 1] << 8) | (c[..., 2] << 16) | (c[..., 3] << 24)


@pytest.fixture(scope="module")
def mixed():
    api = _setup_stream()
    rng = np.random.default_rng(8)

    def random_texture(size, layers):
        return _device_texture([rng.integers(0, 1 << 32, (size, size), dtype=np.uint64).astype(np.uint32) | np.uint32(0xFF << 24)
                                for _ in range(layers)], size)

    cols = rng.integers(0, 256, (6, 2, 4)).astype(np.uint32)
    cols[:, 0, 3] = 255
    words = _words(cols)

    def constant_texture(i, layers, deep=False):
        t = _device_texture([np.full((SIZE, SIZE), words[i, l], np.uint32) for l in range(layers)], SIZE)
        if deep:  # the levels above the decoded ones are another texture's
            data = t.get_data()
            for l in range(layers):
                at = l * t.layer_stride + t.mip_offsets[DECODED]
                data[at: (l + 1) * t.layer_stride] = rng.integers(0, 1 << 32, t.layer_stride - t.mip_offsets[DECODED], dtype=np.uint64)
            t.set_data(data)
        return t

    # 0: decoded; 1: not in the model; 2: decoded, deep levels of its own; 3: the scene's texture is larger than the
    # model's; 4: decoded, one layer; 5: past the model's materials; 6: no texture
    model = [constant_texture(0, 2), None, constant_texture(2, 2, True), constant_texture(3, 2), constant_texture(4, 1)]
    texs = [model[0], random_texture(SIZE, 2), model[2], random_texture(2 * SIZE, 2), model[4], random_texture(SIZE, 2)]
    m = api.NeuralMaterials(model, latent_levels=LATENTS, seed=3)
    for i in (0, 2, 3, 4):
        p = np.zeros(N.PARAMS, np.float32)
        second = cols[i, 1, :4] if i != 4 else np.zeros(4)
        p[N.PB3:N.PARAMS] = np.concatenate([cols[i, 0, :3], second, [255]]) / np.float32(255.0)
        m.set_params(i, p)
    sc = scenes.volume_scene(n=2500, width=324, height=180, n_materials=7, extent=18.0, texture_size=SIZE)
    sc.materials["texture"] = np.arange(7)
    return api, m, GpuRenderer(sc.meshlets, sc.materials, texs)


@pytest.mark.parametrize("size", [(4, 4), (20, 12), (324, 180), (1004, 516)])
@pytest.mark.parametrize("eye", [(0.0, 0.0, 0.0), (0.0, 0.0, -20.0), (0.0, 0.0, -60.0), (0.0, 0.0, -300.0)])
def test_mixed_tiles(mixed, size, eye):
    api, m, g = mixed
    v = scenes.make_view(*size, eye=eye, target=(0.5, 0.2, 1.0))
    ctx = api.ShadingContext(g.scene, v.world_to_clip, world_to_clip=v.world_to_clip, view_pos=v.eye, lights=gpu_lights(default_lights()))
    a, _ = g.render(v.world_to_clip, *size)
    b, _ = g.render(v.world_to_clip, *size)
    ids = a.get_pixels(0)
    ctx.resolve(g.rast, a)
    requests, tiles, per_level = ctx.resolve_neural(g.rast, b, m, want_stats=True)
    assert sum(per_level) == requests and tiles * 128 >= requests and not any(per_level[DECODED:])
    if size[0] >= 324 and eye[2] > -300.0:
        assert requests > 100
        # tiles of several surfaces, hence of several of the materials
        t = ids.reshape(size[1] // 4, 4, size[0] // 4, 4).transpose(0, 2, 1, 3).reshape(-1, 16)
        assert (t.min(1) != t.max(1)).sum() > 100
    assert np.array_equal(a.get_pixels(0), b.get_pixels(0))
    assert np.array_equal(a.get_pixels(1), b.get_pixels(1))
