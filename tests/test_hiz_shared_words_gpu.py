"""The depth pyramid into textures whose words several texels share, bit for bit against the oracle (which writes them one
after the other) and the same every time: tall and wide frames into textures of the usual size, and textures
narrower, lower or with fewer levels than the frame's."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frame(w, h):
    import torch
    from glimpsw_gb300 import api
    from oracle import oracle as O
    api.load_library()
    ofb, gfb = O.Framebuffer(w, h), api.Framebuffer(w, h)
    ofb.clear(0, 0.0)
    gfb.clear(0, 0.0)
    words = np.random.default_rng(w * 4096 + h).uniform(0.0, 1.0, w * h).astype(np.float32).view(np.uint32)
    ofb.data[ofb.layer_stride: ofb.layer_stride + w * h] = words
    src = torch.from_numpy(words.view(np.int32).copy()).cuda()
    rt = ctypes.CDLL("libcudart.so.13")
    torch.cuda.synchronize()
    assert rt.cudaMemcpy(ctypes.c_void_p(gfb.layer_data(1)), ctypes.c_void_p(src.data_ptr()), ctypes.c_size_t(4 * w * h), 3) == 0
    torch.cuda.synchronize()
    return ofb, gfb


def _fits(w, h, o):
    """Whether every level's words lie inside the texture (what the library accepts)."""
    root = max(w, h).bit_length()
    for m in range(root - 2):
        r = 1 << (m + 4)
        cols, rows = (-(-w // r) * 8, -(-h // r) * 8) if m + 4 <= root else (4, 4)
        s = o.s.row_shift - m
        off = o.s.mip_offsets[m] if m < o.s.mip_levels else 0
        if s < 0 or off + 7 + ((cols - 1) << 3) + ((rows - 1) << s) >= o.data.size:
            return False
    return True


def _check(w, h, textures):
    from glimpsw_gb300 import api
    from oracle import oracle as O
    ofb, gfb = _frame(w, h)
    tested = 0
    for tw, th, levels in textures:
        o, g = O.Texture(tw, th, levels, 1, fmt=2), api.Texture2D(api.FORMAT_R32F, tw, th, levels, 1)
        if not _fits(w, h, o):
            with pytest.raises(Exception):
                api.downsample_depth(gfb, g)
            continue
        O.downsample_depth(ofb, o)
        for _ in range(3):
            g.set_data(np.zeros(o.data.size, np.uint32))
            api.downsample_depth(gfb, g)
            got = g.get_data()[: o.data.size]
            assert np.array_equal(got, o.data), f"{tw}x{th}, {levels} levels: {(got != o.data).sum()} texels differ"
        tested += 1
    return tested


@pytest.mark.parametrize("w,h", [(12, 36), (12, 48), (16, 40), (16, 44), (32, 76), (32, 100), (48, 140), (56, 172), (68, 312), (96, 268),
                                 (96, 508), (208, 852), (252, 1000), (76, 32), (312, 68), (1000, 252), (540, 960), (1080, 1920)])
def test_usual_size(w, h):
    from glimpsw_gb300 import api
    api.load_library()
    hw, hh = api.hiz_texture_size(w, h)
    _check(w, h, [(max(hw, 8), max(hh, 4), 16)])


@pytest.mark.parametrize("w,h", [(20, 60), (64, 128), (100, 36), (132, 516), (260, 252), (500, 1900)])
def test_other_textures(w, h):
    sizes = [8, 16, 32, 64, 128, 256, 512, 1024]
    assert _check(w, h, [(tw, th, levels) for tw in sizes for th in sizes for levels in (1, 2, 4, 16)]) > 8
