"""Room for a sky's unpacked level: only textures with a level 2 hold it, and maps without one give the oracle's
irradiance bit for bit; so do calls on several streams at once that unpack the same sky."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _env(w, h, levels, seed):
    from glimpsw_gb300 import api
    from oracle import oracle as O
    api.load_library()
    px = np.random.default_rng(seed).integers(0, 1 << 32, (h, w), dtype=np.uint64).astype(np.uint32) & 0xBFF7FDFF
    o, g = O.Texture(w, h, levels, 1, fmt=1), api.Texture2D(api.FORMAT_R11G11B10F, w, h, levels, 1)
    o.set_pixels(px, 0)
    o.generate_mips()
    g.set_pixels(px)
    g.generate_mips()
    return o, g


def _irradiance(g):
    from glimpsw_gb300 import api
    irr = api.Texture2D(api.FORMAT_R11G11B10F, 8, 4, 1, 1)
    api._check(api._lib.swr_ibl_irradiance_map(g.h, irr.h))
    data = irr.get_data()
    return np.array([[data[(y & 7) | (x << 3)] for x in range(8)] for y in range(4)], np.uint32)


def _expected(o):
    from oracle import oracle as O
    return np.array([[O.ibl_irradiance_texel(o, x, y, 8, 4) for x in range(8)] for y in range(4)], np.uint32)


@pytest.mark.parametrize("w,h,levels", [(64, 64, 1), (64, 64, 2), (64, 64, 3), (16, 8, 16), (16, 16, 16), (512, 512, 1)])
def test_few_levels(w, h, levels):
    o, g = _env(w, h, levels, w + levels)
    assert np.array_equal(_irradiance(g), _expected(o))


def test_room_of_maps_without_level_2():
    import torch
    from glimpsw_gb300 import api
    api.load_library()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    maps = [api.Texture2D(api.FORMAT_R11G11B10F, 512, 512, 1, 1) for _ in range(32)]
    torch.cuda.synchronize()
    taken = free - torch.cuda.mem_get_info()[0]
    assert taken <= 32 * (2 << 20) + (16 << 20), f"32 maps of 1 MB take {taken >> 20} MB"
    del maps


def test_one_sky_on_several_streams():
    import torch
    from glimpsw_gb300 import api
    o, g = _env(256, 256, 16, 5)
    want = _expected(o)
    torch.cuda.synchronize()
    got = [None] * 4

    def work(i):
        s = torch.cuda.Stream()
        api.set_stream(s)
        for _ in range(5):
            got[i] = _irradiance(g)
        api.set_stream(0)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert all(np.array_equal(x, want) for x in got)
