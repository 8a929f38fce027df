"""The depth pyramid bit for bit against the oracle: frames around the 128-pixel regions that one block takes and
the 1024-pixel ones its highest level covers, depths of either sign and both zeros, and textures with fewer
levels than the frame has (the levels they lack land at their start)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SENTINEL = 0x7F7FFFFE


def _depths(words, seed):
    rng = np.random.default_rng(seed)
    d = rng.uniform(0.0, 1.0, words).astype(np.float32)
    pick = rng.integers(0, 64, words)
    d[pick == 0] = 0.0
    d[pick == 1] = -0.0
    d[pick == 2] *= -1.0
    return d.view(np.uint32)


@pytest.mark.parametrize("w,h,levels", [(16, 16, 16), (20, 12, 16), (64, 48, 16), (128, 128, 16), (132, 128, 16), (252, 132, 16),
                                        (260, 256, 16), (512, 508, 16), (1024, 1020, 16), (1028, 1024, 16), (2052, 1032, 16),
                                        (128, 64, 1), (128, 128, 2), (64, 64, 3), (252, 132, 4), (1028, 1024, 5), (2052, 1032, 6)])
def test_pyramid(w, h, levels):
    import torch
    from glimpsw_gb300 import api
    from oracle import oracle as O
    api.load_library()
    ofb, gfb = O.Framebuffer(w, h), api.Framebuffer(w, h)
    ofb.clear(0, 0.0)
    gfb.clear(0, 0.0)
    words = _depths(w * h, w + h)
    ofb.data[ofb.layer_stride: ofb.layer_stride + w * h] = words
    src = torch.from_numpy(words.view(np.int32).copy()).cuda()
    rt = ctypes.CDLL("libcudart.so.13")
    torch.cuda.synchronize()
    assert rt.cudaMemcpy(ctypes.c_void_p(gfb.layer_data(1)), ctypes.c_void_p(src.data_ptr()), ctypes.c_size_t(4 * w * h), 3) == 0
    torch.cuda.synchronize()
    hw, hh = api.hiz_texture_size(w, h)
    hw, hh = max(hw, 8), max(hh, 4)
    if levels < 16:
        hw, hh = 2 * hw, 2 * hh  # a texture of few levels has to be larger to hold the frame
    o, g = O.Texture(hw, hh, levels, 1, fmt=2), api.Texture2D(api.FORMAT_R32F, hw, hh, levels, 1)
    o.data[:] = SENTINEL
    g.set_data(o.data)
    api.downsample_depth(gfb, g)
    O.downsample_depth(ofb, o)
    got = g.get_data()[: o.data.size]
    assert np.array_equal(got, o.data), f"{(got != o.data).sum()} texels differ"
    assert (o.data != SENTINEL).sum() > 0
