"""The IBL maps of wide skies, bit for bit against the oracle. One unit in the last place of a coordinate is an eighth of
the sampler's step on 8192 texels, so a coordinate or a blend that is not rounded as the reference rounds it shows
in the maps, as it hardly ever does on small square skies. Skies read packed and unpacked; last levels of 8 rows."""
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


def _texel(data, offset, stride, x, y):
    return data[offset + ((y & 7) | (x << 3) | ((y & ~7) << stride))]


@pytest.mark.parametrize("w,h,levels", [(1024, 8, 1), (4096, 8, 1), (8192, 16, 1), (8192, 64, 1), (8192, 16, 2), (8192, 64, 3), (8192, 32, 3),
                                        (4096, 64, 3), (1024, 1024, 3)])
@pytest.mark.parametrize("seed", [1, 2])
def test_irradiance(w, h, levels, seed):
    from glimpsw_gb300 import api
    from oracle import oracle as O
    o, g = _env(w, h, levels, seed)
    irr = api.Texture2D(api.FORMAT_R11G11B10F, 32, 16, 1, 1)
    api._check(api._lib.swr_ibl_irradiance_map(g.h, irr.h))
    data = irr.get_data()
    got = np.array([[_texel(data, 0, 5, x, y) for x in range(32)] for y in range(16)], np.uint32)
    exp = np.array([[O.ibl_irradiance_texel(o, x, y, 32, 16) for x in range(32)] for y in range(16)], np.uint32)
    assert np.array_equal(got, exp), f"{(got != exp).sum()} texels differ"


@pytest.mark.parametrize("w,h,levels", [(1024, 8, 1), (8192, 16, 1), (8192, 64, 3), (8192, 128, 4), (2048, 2048, 9)])
def test_radiance(w, h, levels):
    from glimpsw_gb300 import api
    from oracle import oracle as O
    o, g = _env(w, h, levels, 3)
    rad = api.Texture2D(api.FORMAT_R11G11B10F, 64, 64, 16, 1)
    api._check(api._lib.swr_ibl_radiance_map(g.h, rad.h))
    data = rad.get_data()
    for level in range(rad.mip_levels):
        n = 64 >> level
        got = np.array([_texel(data, rad.mip_offsets[level], 6 - level, x, y) for y in range(n) for x in range(n)], np.uint32)
        exp = np.array([O.ibl_radiance_texel(o, level, rad.mip_levels, x, y, 64, 64) for y in range(n) for x in range(n)], np.uint32)
        assert np.array_equal(got, exp), f"level {level}: {(got != exp).sum()} texels differ"
