"""The unit vectors' table is one per device, not per scene: what a scene takes, scenes that outlive the one whose upload
made it, scenes after all have gone, uploads from several threads, and a scene whose room is reserved on one stream
(with work ahead of it) and which is filled, drawn and resolved on another. Resolved frames equal the first one's."""
import threading

import numpy as np
import pytest

from glimpsw_gb300 import scenes
from tests.helpers import default_lights, gpu_lights

pytestmark = pytest.mark.gpu
W, H = 160, 92


@pytest.fixture(scope="module")
def content():
    sc = scenes.volume_scene(n=200, width=W, height=H, n_materials=1, extent=6.0, texture_size=64)
    rng = np.random.default_rng(3)
    sc.meshlets["NormalTangents"] = rng.integers(0, 1 << 32, sc.meshlets["NormalTangents"].shape, dtype=np.uint64).astype(np.uint32)
    return np.ascontiguousarray(sc.meshlets)


def _frame(scene, count):
    from glimpsw_gb300 import api
    v = scenes.make_view(W, H, eye=(0.0, 0.0, -9.0), target=(0.0, 0.0, 0.0))
    fb, rast = api.Framebuffer(W, H), api.Rasterizer()
    fb.clear(0xFF000000, 0.0)
    ctx = api.ShadingContext(scene, v.world_to_clip, world_to_clip=v.world_to_clip, view_pos=v.eye, lights=gpu_lights(default_lights()))
    rast.draw_meshlets(fb, count, ctx)
    assert np.count_nonzero(fb.get_pixels(1)) > 100
    ctx.resolve(rast, fb)
    return fb.get_pixels(0)


def _scene(m):
    from glimpsw_gb300 import api
    api.load_library()
    s = api.Scene()
    s.upload_meshlets(m)
    return s


def test_room_of_many_scenes(content):
    import torch
    first = _scene(content[:1])
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    more = [_scene(content[:1]) for _ in range(64)]
    torch.cuda.synchronize()
    taken = free - torch.cuda.mem_get_info()[0]
    assert taken <= 16 << 20, f"64 scenes of one meshlet take {taken >> 20} MB"
    del more, first


def test_scenes_outlive_the_first(content):
    a, b = _scene(content), _scene(content)
    want = _frame(a, len(content))
    del a
    assert np.array_equal(_frame(b, len(content)), want)
    del b
    assert np.array_equal(_frame(_scene(content), len(content)), want)


def test_uploads_from_threads(content):
    want = _frame(_scene(content), len(content))
    got = [None] * 8

    def work(i):
        for _ in range(3):
            got[i] = _frame(_scene(content), len(content))

    ts = [threading.Thread(target=work, args=(i,)) for i in range(8)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert all(g is not None and np.array_equal(g, want) for g in got)


def test_reserved_on_another_stream(content):
    import torch
    from glimpsw_gb300 import api
    want = _frame(_scene(content), len(content))
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    try:
        s = api.Scene()
        with torch.cuda.stream(a):
            torch.cuda._sleep(20_000_000)
        api.set_stream(a)
        api._check(api._lib.swr_scene_upload_meshlets(s.h, None, len(content), 0))
        api.set_stream(b)
        s.upload_meshlets(content)
        got = _frame(s, len(content))
    finally:
        api.set_stream(0)
    assert np.array_equal(got, want)
