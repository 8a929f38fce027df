// RGBA8 surface sampling shared by the rasterizer's alpha test and the resolve:
// Texture2D<RGBA8u, TiledY8>::SampleLevel<SurfaceSampler> (Texture.h:412-459, 506-556) with the
// sampler of Shading.cpp:6-10 (Repeat wrap, bilinear magnification, nearest minification, the
// filter chosen once for the whole 4x4 tile by the caller).
#pragma once
#include <cuda_fp16.h>

#include "swr_device.cuh"
#include "swr_internal.h"

namespace swr {

// Texture2D::GetTexelOffset for TiledY8 (Texture.h:493-501).
__device__ __forceinline__ uint32_t texel_offset(int32_t x, int32_t y, int32_t stride) {
    return (uint32_t)((y & 7) | (x << 3) | ((y & ~7) << stride));
}

// vcvtph2ps of one half (exact).
__device__ __forceinline__ float h2f(uint32_t h) { return __half2float(__ushort_as_half((unsigned short)h)); }

// simd::ilog2 (SIMD.h:426) where a NaN reads as the x86 default NaN 0xFFC00000 (every NaN on the
// paths that take it comes from an invalid operation, which x86 answers with that pattern).
__device__ __forceinline__ int32_t ilog2_x86(float x) {
    uint32_t b = (x != x) ? 0xFFC00000u : __float_as_uint(x);
    return (int32_t)(b - (127u << 23)) >> 23;
}

// simd::lerp16 (SIMD.h:450), a + mulhrs(b - a, 128 w), of the 8-bit values in both 16-bit halves with a weight
// w of 0..255: mulhrs is ((b - a) 128 w + 2^14) >> 15 = ((b - a) w + 128) >> 8, so the blend is
// (a (256 - w) + b w + 128) >> 8 in each half, at most 65408: two multiplies serve both (about 4
// operations instead of 16; equal for all 2^24 (a, b, w)).
__device__ __forceinline__ uint32_t lerp8x2(uint32_t a, uint32_t b, uint32_t w) {
    return ((a * (256u - w) + b * w + 0x00800080u) >> 8) & 0x00FF00FFu;
}

// Bilinear blend of four RGBA8 texels (the 16-bit lane lerps of SampleLevel<SurfaceSampler>,
// Texture.h:540-556); fx and fy hold the 1.15 fixed-point weight (a multiple of 128) in both halves.
__device__ __forceinline__ uint32_t filter_rgba8(uint32_t d00, uint32_t d10, uint32_t d01, uint32_t d11, uint32_t fx, uint32_t fy) {
    const uint32_t wx = (fx >> 7) & 255u, wy = (fy >> 7) & 255u, k = 0x00FF00FFu;
    const uint32_t rb = lerp8x2(lerp8x2(d00 & k, d10 & k, wx), lerp8x2(d01 & k, d11 & k, wx), wy);
    const uint32_t ga = lerp8x2(lerp8x2((d00 >> 8) & k, (d10 >> 8) & k, wx), lerp8x2((d01 >> 8) & k, (d11 >> 8) & k, wx), wy);
    return rb | (ga << 8);
}

// The texel coordinates one lane's SampleLevel<SurfaceSampler> reads (Texture.h:412-459): level m,
// the nearest texel (tx, ty), or for bilinear the top-left texel, whether its right / lower
// neighbours are inside the level, and the packed 1.15 weights.
struct TexelQuad {
    int32_t m, stride, tx, ty;
    bool inX, inY;
    uint32_t fx, fy;
};
__device__ __forceinline__ TexelQuad texel_quad(const DevTexture& t, float u, float v, int32_t mipIn, bool nearest) {
    TexelQuad q;
    int32_t ix = round2i(__fmul_rn(u, t.scale_lerp_u)) & t.mask_lerp_u;
    int32_t iy = round2i(__fmul_rn(v, t.scale_lerp_v)) & t.mask_lerp_v;
    q.m = min(max(mipIn, 0), (int32_t)t.mip_levels - 1);
    q.stride = (int32_t)t.row_shift - q.m;
    ix >>= q.m, iy >>= q.m;
    if (nearest) {
        q.tx = ix >> 8, q.ty = iy >> 8, q.inX = q.inY = false, q.fx = q.fy = 0;
        return q;
    }
    int32_t xf = max(ix - 127, 0), yf = max(iy - 127, 0);
    q.tx = xf >> 8, q.ty = yf >> 8;
    q.inX = ((q.tx + 1) << q.m) < (int32_t)t.width, q.inY = ((q.ty + 1) << q.m) < (int32_t)t.height;
    uint32_t fx = (uint32_t)(xf & 255) << 7, fy = (uint32_t)(yf & 255) << 7;
    q.fx = q.inX ? ((fx << 16) | fx) : 0u, q.fy = (fy << 16) | fy;
    return q;
}

// The texel of one layer at a quad (SampleLevel<SurfaceSampler>, Texture.h:412-459).
__device__ __forceinline__ uint32_t sample_quad(const DevTexture& t, const TexelQuad& q, int layer, bool nearest) {
    const uint32_t* base = t.data + (size_t)layer * t.layer_stride + t.mip_offsets[q.m & 15];
    if (nearest) return base[texel_offset(q.tx, q.ty, q.stride)];
    const uint32_t i00 = texel_offset(q.tx, q.ty, q.stride), i01 = texel_offset(q.tx, q.ty + (q.inY ? 1 : 0), q.stride);
    return filter_rgba8(base[i00], base[i00 + 8], base[i01], base[i01 + 8], q.fx, q.fy);
}

// The alpha of layer 0's SampleLevel<SurfaceSampler>: what `texel >= cutoff << 24` decides (the lower bytes can
// only raise the word).
__device__ __forceinline__ uint32_t sample_alpha8(const DevTexture& t, float u, float v, int32_t mipIn, bool nearest) {
    const TexelQuad q = texel_quad(t, u, v, mipIn, nearest);
    const uint32_t* base = t.data + t.mip_offsets[q.m & 15];
    if (nearest) return base[texel_offset(q.tx, q.ty, q.stride)] >> 24;
    const uint32_t i00 = texel_offset(q.tx, q.ty, q.stride), i01 = texel_offset(q.tx, q.ty + (q.inY ? 1 : 0), q.stride);
    const uint32_t a00 = base[i00] >> 24, a10 = base[i00 + 8] >> 24, a01 = base[i01] >> 24, a11 = base[i01 + 8] >> 24;
    const uint32_t wx = (q.fx >> 7) & 255u, wy = (q.fy >> 7) & 255u;
    const uint32_t top = (a00 * (256u - wx) + a10 * wx + 128u) >> 8, bot = (a01 * (256u - wx) + a11 * wx + 128u) >> 8;
    return (top * (256u - wy) + bot * wy + 128u) >> 8;
}

// SampleLevel<SurfaceSampler> for one lane once the tile's filter is known (Texture.h:412-459).
__device__ __forceinline__ uint32_t sample_rgba8(const DevTexture& t, float u, float v, int layer, int32_t mipIn, bool nearest) {
    return sample_quad(t, texel_quad(t, u, v, mipIn, nearest), layer, nearest);
}

}  // namespace swr
