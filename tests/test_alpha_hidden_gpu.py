"""Alpha-tested meshlets behind, on and in front of opaque layers, bit for bit against the oracle, with the same
triangle counts: the alpha pass leaves out a meshlet whose box of tiles is nearer than all of it, and counts
its triangles. Depths one rounding apart, boxes across a layer's edge, the frame's edge and past the
tested size, fewer than 64 vertices, and triangles that use slots past the vertices."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.helpers import CLIP_FROM_OBJECT, GpuRenderer, TexturePair, assert_visbuffer_equal, meshlet_from_clip_triangles, render_oracle

pytestmark = pytest.mark.gpu
SIZE = 64


def _texture():
    p = scenes.value_noise_rgba(SIZE, 5, cells=8, layer=0).astype(np.uint32) & 0x00FFFFFF
    a = np.random.default_rng(5).integers(0, 256, (SIZE, SIZE)).astype(np.uint32)
    return TexturePair([p | (a << 24)], SIZE)


def _quad(x0, y0, x1, y1, w):
    c = [(x0, y0), (x1, y0), (x1, y1), (x0, y1)]
    v = [[w * x, w * y, w] for x, y in c]
    return [[v[0], v[1], v[2]], [v[0], v[2], v[3]]]


def _scene(vertices):
    rng = np.random.default_rng(vertices)
    wall = np.float32(2.0)
    parts = [meshlet_from_clip_triangles(_quad(-0.9, -0.9, 0.5, 0.8, wall), 1),
             meshlet_from_clip_triangles(_quad(-1.0, -1.0, 1.0, 1.0, np.float32(7.0)), 1)]
    for i in range(160):
        c, s = rng.uniform(-1.0, 1.0, 2), 10 ** rng.uniform(-2.0, -0.2)
        w = [wall, np.nextafter(wall, np.float32(9)), np.nextafter(wall, np.float32(0)), wall * np.float32(1.001), wall * np.float32(0.999),
             np.float32(3.0), np.float32(1.0), np.float32(8.0)][i % 8]
        tilt = 0.0 if i % 3 else 0.05
        tris = []
        for _ in range(vertices // 3):
            o = c + rng.uniform(-s, s, 2)
            p = o + rng.uniform(-s, s, (3, 2)) * 0.5
            d = w * (1.0 + tilt * rng.uniform(0.0, 1.0, 3))
            tris.append([[d[k] * p[k, 0], d[k] * p[k, 1], d[k]] for k in range(3)])
        m = meshlet_from_clip_triangles(tris, 0)
        uv = rng.uniform(0.0, 2.0, (2,) + m["TexCoords"].shape).astype(np.float16).view(np.uint16).astype(np.uint32)
        m["TexCoords"] = uv[0] | (uv[1] << 16)
        if i % 16 == 9:
            m["NumVertices"] = 3  # the triangles use slots past them
        if i % 16 == 10:
            m["NumVertices"] = 64
        parts.append(m)
    mats = np.zeros(2, dtype=scenes.MATERIAL_DTYPE)
    mats["alpha_cutoff"], mats["is_double_sided"] = [128, 255], 1
    return scenes.concat_meshlets(parts), mats


@pytest.mark.parametrize("vertices", [3, 33, 63])
@pytest.mark.parametrize("size", [(4, 4), (36, 60), (252, 140), (1004, 516)])
def test_layers_bit_exact(vertices, size):
    m, mats = _scene(vertices)
    t = _texture()
    g = GpuRenderer(m, mats, [t.g])
    gfb, gc = g.render(CLIP_FROM_OBJECT, *size, binning=False)
    ofb, oc = render_oracle(m, mats, CLIP_FROM_OBJECT, *size, binning=False, textures=[t.o])
    assert_visbuffer_equal(gfb, ofb)
    assert list(gc[:3]) == list(oc[:3])
