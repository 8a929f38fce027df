"""The chunk stage's coarse tests (32x32-pixel block bounds, one chunk per lane) and the mesh stage's
warp-wide queue append against the oracle, bit for bit: layers of large triangles, near ones in front
of far ones and behind them, at frame sizes around multiples of the block size; a second draw whose keys
are rebuilt from the depth layer (block bounds start empty); queues of about a warp's triangles."""
import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.helpers import CLIP_FROM_OBJECT, GpuRenderer, assert_visbuffer_equal, meshlet_from_clip_triangles, render_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def layers():
    rng = np.random.default_rng(23)
    parts = []
    for i in range(60):
        near = rng.uniform(0.2, 20.0)  # one depth per meshlet, tilted: whole meshlets hide others
        tris = []
        for _ in range(12):
            c, s = rng.uniform(-1.0, 1.0, 2), 10 ** rng.uniform(-1.5, 0.3)
            w = near * rng.uniform(0.9, 1.1, 3)
            tris.append([[w[k] * (c[0] + s * rng.normal()), w[k] * (c[1] + s * rng.normal()), w[k]] for k in range(3)])
        parts.append(meshlet_from_clip_triangles(tris))
    m = scenes.concat_meshlets(parts)
    mats = np.zeros(1, dtype=scenes.MATERIAL_DTYPE)
    mats["alpha_cutoff"], mats["is_double_sided"] = 255, 1
    return m, mats, GpuRenderer(m, mats)


@pytest.mark.parametrize("size", [(4, 4), (28, 32), (32, 28), (36, 60), (64, 64), (68, 252), (1004, 516)])
@pytest.mark.parametrize("binning", [True, False])
def test_layers_bit_exact(layers, size, binning):
    m, mats, g = layers
    w, h = size
    gfb, gc = g.render(CLIP_FROM_OBJECT, w, h, binning=binning)
    ofb, oc = render_oracle(m, mats, CLIP_FROM_OBJECT, w, h, binning=binning)
    assert_visbuffer_equal(gfb, ofb)
    assert list(gc[:3]) == list(oc[:3])


@pytest.mark.parametrize("depth", [0.0, 0.03, -1.0])
def test_second_draw_from_the_depth_layer(layers, depth):
    """Half of the meshlets, the keys dropped, then the other half over a cleared depth below, between and
    above theirs."""
    m, mats, g = layers
    n = len(m) // 2
    w, h, clear = 252, 140, (0xFF000000, depth)
    gfb, _ = g.render(CLIP_FROM_OBJECT, w, h, count=n, clear=clear)
    gfb.invalidate()
    gfb, _ = g.render(CLIP_FROM_OBJECT, w, h, count=len(m) - n, meshlet_offset=n, fb=gfb)
    ofb, _ = render_oracle(m, mats, CLIP_FROM_OBJECT, w, h, count=n, clear=clear)
    ofb, _ = render_oracle(m, mats, CLIP_FROM_OBJECT, w, h, count=len(m) - n, meshlet_offset=n, fb=ofb)
    assert_visbuffer_equal(gfb, ofb)


@pytest.mark.parametrize("capacity", [1, 11, 12, 13, 31, 33])
def test_queue_of_about_a_packet(layers, capacity):
    m, mats, g = layers
    ofb, _ = render_oracle(m, mats, CLIP_FROM_OBJECT, 500, 300)
    g.rast.set_queue_capacity(capacity)
    try:
        gfb, _ = g.render(CLIP_FROM_OBJECT, 500, 300)
    finally:
        g.rast.set_queue_capacity(0)
    assert_visbuffer_equal(gfb, ofb)
