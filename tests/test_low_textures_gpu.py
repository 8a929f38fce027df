"""Textures whose last level is 4 texels high and more than 8 wide: its 8-row columns reach past the texture's words. They
have to lie in memory of their own: the IBL maps of such skies equal the oracle's (on storage with room for
them) bit for bit, the words of the texture equal its words, and textures around it keep theirs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _oracle_texture(w, h, levels, layers, fmt):
    import ctypes as C
    from oracle import oracle as O
    t = O.Texture(w, h, levels, layers, fmt=fmt)
    t.words = t.data.size
    t.data = np.zeros(t.data.size + 8 * w + 128, np.uint32)
    O.lib().orc_texture_init(C.byref(t.s), w, h, levels, layers, O._fptr(t.data))
    return t


@pytest.mark.parametrize("w,h", [(16, 4), (64, 4), (256, 16), (1024, 16), (2048, 64), (8192, 16), (8192, 4)])
def test_sky(w, h):
    from glimpsw_gb300 import api
    from oracle import oracle as O
    api.load_library()
    px = np.random.default_rng(w + h).integers(0, 1 << 32, (h, w), dtype=np.uint64).astype(np.uint32) & 0xBFF7FDFF
    o, g = _oracle_texture(w, h, 16, 1, 1), api.Texture2D(api.FORMAT_R11G11B10F, w, h, 16, 1)
    o.set_pixels(px)
    o.generate_mips()
    g.set_pixels(px)
    g.generate_mips()
    irr = api.Texture2D(api.FORMAT_R11G11B10F, 8, 4, 1, 1)
    rad = api.Texture2D(api.FORMAT_R11G11B10F, 16, 8, 16, 1)
    for _ in range(2):
        api._check(api._lib.swr_ibl_irradiance_map(g.h, irr.h))
        data = irr.get_data()
        got = np.array([[data[(y & 7) | (x << 3)] for x in range(8)] for y in range(4)], np.uint32)
        exp = np.array([[O.ibl_irradiance_texel(o, x, y, 8, 4) for x in range(8)] for y in range(4)], np.uint32)
        assert np.array_equal(got, exp)
    api._check(api._lib.swr_ibl_radiance_map(g.h, rad.h))
    data = rad.get_data()
    for level in range(rad.mip_levels):
        lw, lh = 16 >> level, 8 >> level
        got = [data[rad.mip_offsets[level] + ((y & 7) | (x << 3))] for y in range(lh) for x in range(lw)]
        assert got == [O.ibl_radiance_texel(o, level, rad.mip_levels, x, y, 16, 8) for y in range(lh) for x in range(lw)]
    assert np.array_equal(g.get_data()[: o.words], o.data[: o.words])


@pytest.mark.parametrize("fmt", [0, 1, 2])
@pytest.mark.parametrize("w,h,layers", [(16, 4, 1), (32, 4, 2), (512, 8, 2), (4096, 4, 3), (16384, 4, 1), (16384, 32, 1)])
def test_neighbours(w, h, layers, fmt):
    from glimpsw_gb300 import api
    api.load_library()
    rng = np.random.default_rng(w + h + layers)
    gfmt = [api.FORMAT_RGBA8U, api.FORMAT_R11G11B10F, api.FORMAT_R32F][fmt]
    mask = np.uint32([0xFFFFFFFF, 0xBFF7FDFF, 0x3FFFFFFF][fmt])
    small = [api.Texture2D(gfmt, 8, 8, 1, 1) for _ in range(3)]
    low = [api.Texture2D(gfmt, w, h, 16, layers) for _ in range(3)]
    small += [api.Texture2D(gfmt, 8, 8, 1, 1) for _ in range(3)]
    before = []
    for t in small:
        t.set_pixels(rng.integers(0, 1 << 32, (8, 8), dtype=np.uint64).astype(np.uint32) & mask)
        before.append(t.get_data())
    o = _oracle_texture(w, h, 16, layers, fmt)
    for t in low:
        for layer in range(layers):
            px = rng.integers(0, 1 << 32, (h, w), dtype=np.uint64).astype(np.uint32) & mask
            t.set_pixels(px, layer)
            if t is low[0]:
                o.set_pixels(px, layer)
        t.generate_mips()
    o.generate_mips()
    assert np.array_equal(low[0].get_data()[: o.words], o.data[: o.words])
    for t, want in zip(small, before):
        assert np.array_equal(t.get_data(), want)
