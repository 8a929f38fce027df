"""The depth pyramid into textures that lack some of its levels, bit for bit against the oracle: every level lands at
the texture's start in ascending order, also where several 128-pixel regions write the same words. Each frame is
written repeatedly, with the texture's words reset in between."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SENTINEL = 0x7F7FFFFE


@pytest.mark.parametrize("levels", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("w,h", [(32, 16), (132, 128), (256, 128), (252, 260), (516, 508), (1028, 1024), (2052, 1032), (2896, 2896)])
def test_missing_levels(w, h, levels):
    import torch
    from glimpsw_gb300 import api
    from oracle import oracle as O
    api.load_library()
    ofb, gfb = O.Framebuffer(w, h), api.Framebuffer(w, h)
    ofb.clear(0, 0.0)
    gfb.clear(0, 0.0)
    rng = np.random.default_rng(w + h + levels)
    d = rng.uniform(-0.1, 1.0, w * h).astype(np.float32)
    d[rng.integers(0, 64, w * h) == 0] = -0.0
    words = d.view(np.uint32)
    ofb.data[ofb.layer_stride: ofb.layer_stride + w * h] = words
    src = torch.from_numpy(words.view(np.int32).copy()).cuda()
    rt = ctypes.CDLL("libcudart.so.13")
    torch.cuda.synchronize()
    assert rt.cudaMemcpy(ctypes.c_void_p(gfb.layer_data(1)), ctypes.c_void_p(src.data_ptr()), ctypes.c_size_t(4 * w * h), 3) == 0
    torch.cuda.synchronize()
    hw, hh = api.hiz_texture_size(w, h)
    hw, hh = 2 * max(hw, 8), 2 * max(hh, 8)  # a texture of few levels has to be larger to hold the frame
    o, g = O.Texture(hw, hh, levels, 1, fmt=2), api.Texture2D(api.FORMAT_R32F, hw, hh, levels, 1)
    o.data[:] = SENTINEL
    reset = o.data.copy()
    O.downsample_depth(ofb, o)
    for _ in range(3):
        g.set_data(reset)
        api.downsample_depth(gfb, g)
        got = g.get_data()[: o.data.size]
        assert np.array_equal(got, o.data), f"{(got != o.data).sum()} texels differ"
