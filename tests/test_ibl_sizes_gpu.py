"""IBL maps from environment maps of other shapes, bit for bit against the oracle: maps with fewer than three
levels, non-square ones, and both sides of the size up to which the irradiance map's level is unpacked
first (512x512 texels)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _env(w, h, seed):
    from glimpsw_gb300 import api
    from oracle import oracle as O
    api.load_library()
    px = np.random.default_rng(seed).integers(0, 1 << 32, (h, w), dtype=np.uint64).astype(np.uint32) & 0xBFF7FDFF
    o, g = O.Texture(w, h, 16, 1, fmt=1), api.Texture2D(api.FORMAT_R11G11B10F, w, h, 16, 1)
    o.set_pixels(px, 0)
    o.generate_mips()
    g.set_pixels(px)
    g.generate_mips()
    return o, g


@pytest.mark.parametrize("w,h", [(8, 4), (8, 8), (64, 16), (2048, 2048), (4096, 2048)])
def test_irradiance_and_radiance(w, h):
    from glimpsw_gb300 import api
    from oracle import oracle as O
    o, g = _env(w, h, w + h)
    irr = api.Texture2D(api.FORMAT_R11G11B10F, 8, 4, 1, 1)
    api._check(api._lib.swr_ibl_irradiance_map(g.h, irr.h))
    data = irr.get_data()
    got = np.array([[data[(y & 7) | (x << 3)] for x in range(8)] for y in range(4)], np.uint32)
    exp = np.array([[O.ibl_irradiance_texel(o, x, y, 8, 4) for x in range(8)] for y in range(4)], np.uint32)
    assert np.array_equal(got, exp)
    rad = api.Texture2D(api.FORMAT_R11G11B10F, 8, 8, 16, 1)
    api._check(api._lib.swr_ibl_radiance_map(g.h, rad.h))
    data = rad.get_data()
    for level in range(rad.mip_levels):
        n = 8 >> level
        got = [data[rad.mip_offsets[level] + ((y & 7) | (x << 3))] for y in range(n) for x in range(n)]
        assert got == [O.ibl_radiance_texel(o, level, rad.mip_levels, x, y, 8, 8) for y in range(n) for x in range(n)]


@pytest.mark.parametrize("w,h", [(8, 4), (16, 8), (32, 16), (64, 32)])
def test_brdf_table_sizes(w, h):
    """Blocks of 32 texels over several rows (a narrow table) and over one."""
    from glimpsw_gb300 import api
    from oracle import oracle as O
    api.load_library()
    out = api.Texture2D(api.FORMAT_RG16F, w, h, 1, 1)
    api._check(api._lib.swr_ibl_env_brdf_lut(out.h))
    data = out.get_data()
    stride = max(w, 8).bit_length() - 1
    got = np.array([[data[(y & 7) | (x << 3) | ((y & ~7) << stride)] for x in range(w)] for y in range(h)], np.uint32)
    exp = np.array([[O.ibl_env_brdf_texel(x, y, w, h) for x in range(w)] for y in range(h)], np.uint32)
    assert np.array_equal(got, exp)
