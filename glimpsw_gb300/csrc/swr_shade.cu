// Meshlet culling (ShadingContext::CullMeshlets), the Hi-Z depth pyramid (texutil::DownsampleDepth)
// and the vis-buffer resolve (ShadingContext::Resolve) for sm_103a.
//
// The translation unit is compiled with -fmad=false, so every float expression below is evaluated
// in source order with one rounding per operation, as the reference's C++ is written; fmaf()
// stands for the reference's explicit simd::fma. simd::approx_rcp / approx_rsqrt / approx_sqrt
// (the AVX-512 instructions VRCP14PS and VRSQRT14PS) are reproduced bit for bit by the integer
// segment tables of include/swr/approx14.h.
//
// Resolve layout: a half-warp shades one 4x4 tile (lane = pixel), so the reference's tile-wide
// decisions (`any(mipLevel > 0)` filter choice, normal-map enable, light skipping, sky branch)
// become ballots over the half-warp, evaluated over all 16 pixels like the 16 AVX-512 lanes.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/swr/approx14.h"
#include "../../include/swr/hostmath.h"
#include "swr_device.cuh"
#include "swr_internal.h"
#include "swr_neural.h"
#include "swr_sample.cuh"
#include "swr_surface.cuh"

namespace swr {
namespace {


// =========================================================================== culling
struct CullArgs {
    const uint8_t* meshlets;
    uint32_t first, count;
    uint16_t* bitmap;
    unsigned int* visibleCount;
    float planes[5][4];
    float objectToPrevView[16];
    float objectToWorldScale;
    float projFactors[3];
    float frameW, frameH;
    const uint32_t* depthData;  // R32f Hi-Z storage or null
    uint32_t mipOffsets[16];
    uint32_t mipLevels, rowShift;
    // backface-cone culling (cone_culled): camera centre in object space, materials
    uint32_t cone;
    float eye[3];
    const DevMaterial* materials;
    uint32_t numMaterials;
};

// ShadingContext::CullMeshlets (Shading.cpp:775-869) + ProjectSphere (264-279), one meshlet per
// thread; a warp's ballot gives two of the reference's 16-bit masks. With a.cone, meshlets that
// pass the frustum test and face away as a whole (cone_culled) are dropped before the Hi-Z test.
__global__ void __launch_bounds__(256) k_cull(CullArgs a) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    bool visible = i < a.count;
    if (visible) {
        const float* b = (const float*)(a.meshlets + (size_t)(a.first + i) * kMeshletSize);  // BoundCenter, BoundRadius
        const float4 s = *(const float4*)b;
        const F3 c = { s.x, s.y, s.z };
        const float r = s.w;
        for (int k = 0; k < 5; k++) {
            float dist = fmaf(c.x, a.planes[k][0], fmaf(c.y, a.planes[k][1], c.z * a.planes[k][2])) + a.planes[k][3];
            visible = visible && (dist > -r);
        }
        if (a.cone && visible)
            visible = !cone_culled((const uint8_t*)b, a.eye[0], a.eye[1], a.eye[2], a.materials, a.numMaterials);
        if (a.depthData != nullptr && visible) {
            float vw;
            F3 vs = xform4(a.objectToPrevView, c, vw);
            const float rvs = r * a.objectToWorldScale;
            // ProjectSphere
            float cx = vs.x, cy = vs.y, cz = vs.z * -1.0f;
            bool projMask = cz >= rvs + a.projFactors[0];
            if (projMask) {
                float crx = cx * rvs, cry = cy * rvs, crz = cz * rvs;
                float vx = approx_sqrt(cx * cx + cz * cz - rvs * rvs);
                float vy = approx_sqrt(cy * cy + cz * cz - rvs * rvs);
                float sx = a.projFactors[1] * 0.5f, sy = a.projFactors[2] * 0.5f;
                float bb0 = (vx * cx - crz) * approx_rcp(vx * cz + crx) * sx + 0.5f;
                float bb1 = (vy * cy + crz) * approx_rcp(vy * cz - cry) * sy + 0.5f;
                float bb2 = (vx * cx + crz) * approx_rcp(vx * cz - crx) * sx + 0.5f;
                float bb3 = (vy * cy - crz) * approx_rcp(vy * cz + cry) * sy + 0.5f;
                float bw = (bb2 - bb0) * a.frameW, bh = (bb3 - bb1) * a.frameH;
                int32_t mip = ilog2_x86(vmax(bw, bh));
                mip = min(max(mip, 1), (int32_t)a.mipLevels - 1);
                int32_t x0 = max(trunc2i(bb0 * a.frameW), 0) >> mip;
                int32_t y0 = max(trunc2i(bb1 * a.frameH), 0) >> mip;
                int32_t x1 = min(trunc2i(bb2 * a.frameW), (int32_t)a.frameW - 1) >> mip;
                int32_t y1 = min(trunc2i(bb3 * a.frameH), (int32_t)a.frameH - 1) >> mip;
                float depthSphere = a.projFactors[0] / (-vs.z - rvs);
                float depthVisible = FLT_MAX;
                const uint32_t level = (uint32_t)(mip - 1);
                const int32_t stride = (int32_t)a.rowShift - (int32_t)level;
                const uint32_t* base = a.depthData + a.mipOffsets[level & 15];
                for (int32_t y = y0; y <= y1; y++)
                    for (int32_t x = x0; x <= x1; x++)
                        depthVisible = vmin(depthVisible, __uint_as_float(base[texel_offset(x, y, stride)]));
                visible = depthSphere > depthVisible;
            }
        }
    }
    const unsigned m = __ballot_sync(0xFFFFFFFFu, visible);
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t w0 = i & ~31u;
    if (lane == 0 && w0 < a.count) {
        a.bitmap[w0 / 16] = (uint16_t)(m & 0xFFFF);
        if (w0 + 16 < a.count) a.bitmap[w0 / 16 + 1] = (uint16_t)(m >> 16);
        if (a.visibleCount) atomicAdd(a.visibleCount, (unsigned)__popc(m));
    }
}

// =========================================================================== Hi-Z
// texutil::DownsampleDepth (ImageHelpers.cpp:150-247). Mip m texels hold the min of the frame
// depths they cover (FLT_MAX where they cover none). The reference writes mip m (m <= root-4) in
// 8x8-texel blocks of 2^(m+4)-pixel regions whose origin lies inside the frame, and mip root-3
// as one 4x4 tile. Two launches write exactly those texels: k_hiz_local makes levels 0-6 of one
// 128x128-pixel region per block, k_hiz_tail the levels above in one block, level by level. A texel is the min
// of its four children in the order vmin(vmin(00, 01), vmin(10, 11)); a child whose origin lies outside the frame
// counts as FLT_MAX.
struct HizOffsets { uint32_t off[16]; };  // MipOffsets of the levels written (0 for levels the texture lacks)
constexpr uint32_t kHizRegion = 128;      // pixels per side of a k_hiz_local block (level 6's texel)

__device__ __forceinline__ float min4(float c00, float c01, float c10, float c11) { return vmin(vmin(c00, c01), vmin(c10, c11)); }
// The same across lanes, for the lanes whose bits `down` (y + 1) and `right` (x + 1) are clear.
__device__ __forceinline__ float min4_lanes(float v, uint32_t down, uint32_t right) {
    const float p = vmin(v, __shfl_down_sync(0xFFFFFFFFu, v, down));
    return vmin(p, __shfl_down_sync(0xFFFFFFFFu, p, right));
}

// A thread takes a 4x4 depth tile (four 16-byte loads), a warp 8 x 4 tiles, with lanes down the columns as the
// texture's 8-texel columns run; levels 0 and 1 are the thread's, 2 and 3 the warp's, 4 to 6 the first warp's.
// Bound by latency (a load, three shuffles, a barrier, two shuffles): all of 2560x1440
// 22.1 -> 9.1 us (a thread per texel of levels 0-3 through shared memory, and one block for the levels above),
// 1280x720 14.4 -> 6.4 us.
__global__ void __launch_bounds__(1024) k_hiz_local(const float* __restrict__ depth, uint32_t fbW, uint32_t fbH,
                                                    uint32_t* __restrict__ tex, HizOffsets offs, int32_t rowShift,
                                                    uint32_t nLocal) {
    __shared__ float s3[8][8];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t X = blockIdx.x * 32 + (warp & 3) * 8 + (lane >> 2), Y = blockIdx.y * 32 + (warp >> 2) * 4 + (lane & 3);
    // texel (x, y) of level m is written if its 8x8 block's region is in the frame
    auto written = [&](uint32_t x, uint32_t y, uint32_t m) {
        return m < nLocal && ((x & ~7u) << (m + 1)) < fbW && ((y & ~7u) << (m + 1)) < fbH;
    };
    auto write = [&](uint32_t x, uint32_t y, uint32_t m, float v) {
        if (written(x, y, m)) tex[offs.off[m] + texel_offset(x, y, rowShift - (int32_t)m)] = __float_as_uint(v);
    };
    float v00 = FLT_MAX, v01 = FLT_MAX, v10 = FLT_MAX, v11 = FLT_MAX;
    if (X * 4 < fbW && Y * 4 < fbH) {
        const float4* t = (const float4*)(depth + ((size_t)Y * (fbW >> 2) + X) * 16);
        const float4 r0 = t[0], r1 = t[1], r2 = t[2], r3 = t[3];
        v00 = min4(r0.x, r1.x, r0.y, r1.y), v10 = min4(r0.z, r1.z, r0.w, r1.w);
        v01 = min4(r2.x, r3.x, r2.y, r3.y), v11 = min4(r2.z, r3.z, r2.w, r3.w);
    }
    if (written(2 * X, 2 * Y, 0)) {
        *(float2*)&tex[offs.off[0] + texel_offset(2 * X, 2 * Y, rowShift)] = make_float2(v00, v01);
        *(float2*)&tex[offs.off[0] + texel_offset(2 * X + 1, 2 * Y, rowShift)] = make_float2(v10, v11);
    }
    const float v1 = min4(v00, v01, v10, v11);
    write(X, Y, 1, v1);
    const float v2 = min4_lanes(v1, 1, 4);
    if ((lane & 5) == 0) write(X >> 1, Y >> 1, 2, v2);
    const float v3 = min4_lanes(v2, 2, 8);
    if ((lane & 15) == 0) {
        write(X >> 2, Y >> 2, 3, v3);
        s3[warp >> 2][(warp & 3) * 2 + (lane >> 4)] = v3;
    }
    if (nLocal <= 4) return;
    __syncthreads();
    if (warp != 0) return;
    const uint32_t x = (lane >> 2) & 3, y = lane & 3;  // of the region's 4x4 level 4 texels
    const float v4 = min4(s3[2 * y][2 * x], s3[2 * y + 1][2 * x], s3[2 * y][2 * x + 1], s3[2 * y + 1][2 * x + 1]);
    if (lane < 16) write(blockIdx.x * 4 + x, blockIdx.y * 4 + y, 4, v4);
    const float v5 = min4_lanes(v4, 1, 4);
    if (lane < 16 && (lane & 5) == 0) write(blockIdx.x * 2 + (x >> 1), blockIdx.y * 2 + (y >> 1), 5, v5);
    const float v6 = min4_lanes(v5, 2, 8);
    if (lane == 0) write(blockIdx.x, blockIdx.y, 6, v6);
}

// The levels above k_hiz_local's (first = 7 or fewer .. last = root-3) in one block, out of shared memory:
// the texels of level first-1 whose origin lies in the frame are read once (the others count as
// FLT_MAX), then each level is computed from the previous one in shared memory and written out.
// lvl[k] holds level first-1+k as a (fbW >> (first+k) rounded up) x (fbH >> ...) array.
__host__ __device__ inline uint32_t hiz_extent(uint32_t n, uint32_t level) { return (n + (2u << level) - 1) >> (level + 1); }

__global__ void __launch_bounds__(1024) k_hiz_tail(uint32_t fbW, uint32_t fbH, uint32_t* tex, HizOffsets offs,
                                                   int32_t rowShift, uint32_t first, uint32_t last, uint32_t root) {
    extern __shared__ float lvl[];
    {  // level first-1 from the texture
        const uint32_t m = first - 1, w = hiz_extent(fbW, m), h = hiz_extent(fbH, m);
        const int32_t stride = rowShift - (int32_t)m;
        for (uint32_t t = threadIdx.x; t < w * h; t += blockDim.x)
            lvl[t] = __uint_as_float(tex[offs.off[m] + texel_offset(t % w, t / w, stride)]);
    }
    __syncthreads();
    float* src = lvl;
    for (uint32_t m = first; m <= last; m++) {
        const uint32_t sw = hiz_extent(fbW, m - 1), sh = hiz_extent(fbH, m - 1);
        const uint32_t dw = hiz_extent(fbW, m), dh = hiz_extent(fbH, m);
        float* dst = src + sw * sh;
        uint32_t regionsX = 1, regionsY = 1, blockTexels = 16;
        if (m + 4 <= root) {
            const uint32_t region = 1u << (m + 4);
            regionsX = (fbW + region - 1) / region, regionsY = (fbH + region - 1) / region, blockTexels = 64;
        }
        const uint32_t bs = blockTexels == 64 ? 8 : 4, n = regionsX * regionsY * blockTexels;
        for (uint32_t t = threadIdx.x; t < n; t += blockDim.x) {
            const uint32_t blk = t / blockTexels, within = t - blk * blockTexels;
            const uint32_t by = blk / regionsX, bx = blk - by * regionsX;
            const uint32_t tx = bx * bs + within % bs, ty = by * bs + within / bs;
            // children at mip m-1 cover 2^m pixels; one whose origin is outside the frame covers none
            auto c = [&](uint32_t x, uint32_t y) -> float { return (x < sw && y < sh) ? src[y * sw + x] : FLT_MAX; };
            const uint32_t x = tx * 2, y = ty * 2;
            const float v = vmin(vmin(c(x, y), c(x, y + 1)), vmin(c(x + 1, y), c(x + 1, y + 1)));
            tex[offs.off[m] + texel_offset(tx, ty, rowShift - (int32_t)m)] = __float_as_uint(v);
            if (tx < dw && ty < dh) dst[ty * dw + tx] = v;
        }
        __syncthreads();
        src = dst;
    }
}

// One level's texels (cols x rows, as written) from a scratch pyramid to a texture whose words several of them may share:
// a texel's word is (y & 7) | x << 3 | (y & ~7) << stride, and in a texture narrower than what is written
// x and the bands of 8 rows overlap. The reference writes bands in order and texels from left to right: of
// the texels of a word the one of the last band, and there of the last column, stays.
__global__ void __launch_bounds__(256) k_hiz_place(const uint32_t* __restrict__ src, int32_t srcStride, uint32_t* __restrict__ dst,
                                                   int32_t stride, uint32_t cols, uint32_t rows) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < cols * rows; i += gridDim.x * blockDim.x) {
        const uint32_t x = i % cols, y = i / cols, band = y >> 3, low = x & ((1u << stride) - 1u);
        const uint32_t word = (x >> stride) | band;  // the bits that columns and bands share
        uint32_t last = (rows + 7) / 8 - 1;
        while (last > band && ((last & ~word) || ((word & ~last) << stride | low) >= cols)) last--;
        uint32_t column = (cols - 1) >> stride;
        while (((column << stride | low) >= cols) || (column & ~word) || ((column | last) != word)) column--;
        if (last == band && column == x >> stride)
            dst[texel_offset((int32_t)x, (int32_t)y, stride)] = src[texel_offset((int32_t)x, (int32_t)y, srcStride)];
    }
}

// =========================================================================== resolve
// Up to this many lights travel in the kernel's parameters; more are copied to a device allocation (an
// allocation, a copy and a free per frame cost more host and stream time than a small frame's resolve).
constexpr uint32_t kParamLights = 16;
struct ResolveArgs {
    const uint8_t* meshlets;
    uint32_t numMeshlets;
    const DevMaterial* materials;
    uint32_t numMaterials;
    const float4* octTable;
    uint32_t* color;        // layer 0 (surface ids in, RGBA8 out)
    float* depth;           // layer 1
    const unsigned long long* keys;  // draws not yet in the layers (nullptr: the layers are up to date)
    uint32_t width, height;
    float objectToClip[16];
    float objectToWorld[9];
    float invProj[16];
    float viewPos[3];
    float exposure;
    const swr_light* lights;  // device copy (nullptr: the lights are in `light`)
    uint32_t numLights;
    swr_light light[kParamLights];
    DevTexture sky;
    int hasSky;
    uint32_t debugLayer;    // SWR_DEBUG_* of the debug mode
};

// Neural resolve: the emit pass records, per pixel, what the texels of the levels the model decodes
// are (4 slots: the nearest texel, or the bilinear quad's 00 10 01 11 texels) and counts them per material; the
// second pass reads the decoded texels from the same slots. Within a 4x4 tile a slot's texel is
// decoded by the lowest lane that needs it at the same quad position (its leader): a magnified texture
// gives most of a tile's pixels the same quad.
enum { kResolvePlain = 0, kResolveEmit = 1, kResolveNeural = 2, kResolveDebug = 3 };
struct NeuralResolve {
    const DevTexture* tex;             // model textures (data == nullptr: not decoded)
    uint32_t numMaterials, decodedLevels;  // texture levels below decodedLevels are decoded
    uint32_t* counts;                  // [copy][material]
    const uint2* decoded;              // [pixel * 4 + k] layer-0 RGBA8, layer-1 RGBA8
    uint4* surf;                       // [pixel], then [pixels + pixel]: the emit pass's record
    uint32_t pixels;
};
// The emit pass's record of a pixel, which spares the second pass the reconstruction of a tile whose pixels all have
// it (kSurfFast). First plane: barycentrics b1, b2 and two vertices' normal/tangent words. Second plane, which
// k_neural_scatter reads too: the third vertex's word, the flags (kSurf*, swr_neural.h) with the quad's
// filter weights, the texel (level << 28 | ty << 14 | tx, the quad's first) and the material with the slots' leaders
// (4 bits each from bit 16). 32 bytes a pixel instead of 64 with a word per slot, at
// 2560x1440: emit pass 171 -> 162 us, scatter 59 -> 27, second pass 134 -> 118.
__device__ __forceinline__ uint32_t surf_weight(uint32_t f) { return (f >> 7) & 255u; }             // of a packed 1.15 weight
__device__ __forceinline__ uint32_t packed_weight(uint32_t w) { return (w << 7) | (w << 23); }      // and back

__device__ __forceinline__ uint32_t sat_u8(int32_t v) { return (uint32_t)min(max(min(max(v, -32768), 32767), 0), 255); }
__device__ __forceinline__ float unpack_f11(uint32_t x) { x <<= 17; return __uint_as_float((x & 0x0FFE0000u) + 0x38000000u); }
__device__ __forceinline__ float unpack_f10(uint32_t x) { x <<= 18; return __uint_as_float((x & 0x0FFC0000u) + 0x38000000u); }
__device__ __forceinline__ F3 unpack_r11(uint32_t p) { return { unpack_f11(p >> 21), unpack_f11(p >> 10), unpack_f10(p) }; }

// SampleOctLevel<EnvSampler>(dir, 1) on an R11G11B10 map (Texture.h:467-480; level 1 has no fraction).
__device__ F3 sample_env(const DevTexture& t, F3 dir) {
    float w = approx_rcp(fabsf(dir.x) + fabsf(dir.y) + fabsf(dir.z));
    float tt = vmax(-dir.z * w, 0.0f);
    float u = fmaf(dir.x, w, mulsign(tt, dir.x)) * 0.5f + 0.5f;
    float v = fmaf(dir.y, w, mulsign(tt, dir.y)) * 0.5f + 0.5f;
    int32_t m = min(max(1, 0), (int32_t)t.mip_levels - 1);
    int32_t x = min(max(round2i(u * t.scale_lerp_u), 0), t.mask_lerp_u);
    int32_t y = min(max(round2i(v * t.scale_lerp_v), 0), t.mask_lerp_v);
    int32_t stride = (int32_t)t.row_shift - m;
    x >>= m, y >>= m;
    const uint32_t* base = t.data + t.mip_offsets[m & 15];
    int32_t xf = max(x - 127, 0), yf = max(y - 127, 0);
    int32_t tx = xf >> 8, ty = yf >> 8;
    bool inX = ((tx + 1) << m) < (int32_t)t.width, inY = ((ty + 1) << m) < (int32_t)t.height;
    uint32_t i00 = texel_offset(tx, ty, stride), i01 = texel_offset(tx, ty + (inY ? 1 : 0), stride);
    F3 c00 = unpack_r11(base[i00]), c10 = unpack_r11(base[i00 + 8]), c01 = unpack_r11(base[i01]), c11 = unpack_r11(base[i01 + 8]);
    const float fs = 1.0f / 256;
    float fx = (float)(xf & 255) * fs, fy = (float)(yf & 255) * fs;
    if (!inX) fx = 0;
    F3 ra = { c00.x + (c10.x - c00.x) * fx, c00.y + (c10.y - c00.y) * fx, c00.z + (c10.z - c00.z) * fx };
    F3 rb = { c01.x + (c11.x - c01.x) * fx, c01.y + (c11.y - c01.y) * fx, c01.z + (c11.z - c01.z) * fx };
    return { ra.x + (rb.x - ra.x) * fy, ra.y + (rb.y - ra.y) * fy, ra.z + (rb.z - ra.z) * fy };
}

// Turbo colormap (Google Research 2019, polynomial fit; Shading.cpp:249-260) in the reference's
// Horner order.
__device__ __forceinline__ F3 colormap_turbo(float x) {
    constexpr float c[18] = {
        0.13572138f, 4.61539260f,  -42.66032258f, 132.13108234f, -152.94239396f, 59.28637943f,
        0.09140261f, 2.19418839f,  4.84296658f,   -14.18503333f, 4.27729857f,    2.82956604f,
        0.10667330f, 12.64194608f, -60.58204836f, 110.36276771f, -89.90310912f,  27.34824973f,
    };
    auto poly = [&](int k) { return x * (x * (x * (x * (x * c[k + 5] + c[k + 4]) + c[k + 3]) + c[k + 2]) + c[k + 1]) + c[k]; };
    return { poly(0), poly(6), poly(12) };
}

// RGBA8u::Unpack of the RGB bytes (Texture.h:28-36).
__device__ __forceinline__ F3 unpack_rgb8(uint32_t p) {
    const float s = 1.0f / 255;
    return { (float)(p & 255) * s, (float)((p >> 8) & 255) * s, (float)((p >> 16) & 255) * s };
}

// ResolveDebug's colour of one non-sky pixel (Shading.cpp:748-768) as RGBA8u::Pack({c, 1}); data is
// the pixel's layer-0 word, the surface values are read for layers 1-3 only.
__device__ __forceinline__ uint32_t debug_pixel(uint32_t layer, uint32_t data, uint32_t albedo, F3 N, float metallic,
                                                float roughness) {
    F3 c = { 0.0f, 0.0f, 0.0f };
    if (layer == SWR_DEBUG_BASE_COLOR) c = unpack_rgb8(albedo);
    else if (layer == SWR_DEBUG_NORMALS) c = { N.x * 0.5f + 0.5f, N.y * 0.5f + 0.5f, N.z * 0.5f + 0.5f };
    else if (layer == SWR_DEBUG_METALLIC_ROUGHNESS) c = { metallic, roughness, 0.0f };
    else if (layer == SWR_DEBUG_MESHLET_ID) c = unpack_rgb8((data / 128u) * 123456789u);
    else if (layer == SWR_DEBUG_TRIANGLE_ID) c = unpack_rgb8(data * 123456789u);
    else if (layer == SWR_DEBUG_OVERDRAW_PIXEL) c = colormap_turbo((float)(data >> 16) / 30.0f);
    else if (layer == SWR_DEBUG_OVERDRAW_QUAD) c = colormap_turbo(((float)(data >> 16) + (float)(data & 0xFFFF) * 0.5f) / 30.0f);
    return sat_u8(round2i(c.x * 255.0f)) | (sat_u8(round2i(c.y * 255.0f)) << 8) | (sat_u8(round2i(c.z * 255.0f)) << 16) |
           (255u << 24);
}

__global__ void k_oct_table(float4* table) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    const F3 v = unpack_unit(i);
    table[i] = make_float4(v.x, v.y, v.z, 0.0f);
}

// Bound by instruction issue (73 % of the slots, 82 M instructions at 1080p, 57 registers; 1080p: 1600 instructions a warp and 106 us with a load round per
// surface id and a sampling round per material, 1400 and 90 us without, 82 us with the table of unit vectors).
template <int kMode>
__global__ void __launch_bounds__(256) k_resolve(const __grid_constant__ ResolveArgs a, const __grid_constant__ NeuralResolve nr) {
    const uint32_t lane = threadIdx.x & 31, l = lane & 15, half = lane >> 4;
    const unsigned hm = 0xFFFFu << (16 * half);
    const uint32_t tilesX = a.width >> 2, numTiles = tilesX * (a.height >> 2);
    const uint32_t tile = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    if (tile >= numTiles) return;  // whole half-warps leave together
    const uint32_t ty = tile / tilesX, tx = tile - ty * tilesX;
    const uint32_t x0 = tx * 4, y0 = ty * 4;
    const uint32_t px = x0 + (l & 3), py = y0 + (l >> 2);
    const uint32_t off = pixel_offset(x0, y0, a.width) + l;

    // Pending draws are taken from the keys, and their depths (for the second neural pass also their ids) reach
    // the layers here: a pass over keys and layers of its own took 3 to 11 us.
    uint32_t id;
    float d;
    const unsigned long long key = (kMode == kResolvePlain || kMode == kResolveEmit) && a.keys ? a.keys[off] : kKeyEmptyLow;
    if ((uint32_t)key != kKeyEmptyLow) {
        id = rank_surface_id(0xFFFFFFFEu - (uint32_t)key);
        d = float_unorder((uint32_t)(key >> 32));
        a.depth[off] = d;
        if constexpr (kMode == kResolveEmit) a.color[off] = id;
    } else {
        id = a.color[off];
        d = a.depth[off];
    }
    const bool isSky = d <= 0.0f;
    const float fpx = (float)(int32_t)px, fpy = (float)(int32_t)py;
    float qw;
    F3 q = xform4(a.invProj, { fpx, fpy, isSky ? 1.0f : d }, qw);
    const float rw = 1.0f / qw;
    const F3 world = { q.x * rw, q.y * rw, q.z * rw };
    const float W = (float)a.width, H = (float)a.height;
    const float scaleU = 2.0f / W, scaleV = 2.0f / H;
    const float su = fpx * scaleU + (0.5f * scaleU - 1.0f), sv = fpy * scaleV + (0.5f * scaleV - 1.0f);
    const unsigned skyBits = (__ballot_sync(hm, isSky) >> (16 * half)) & 0xFFFF;

    F3 color = { 0.f, 0.f, 0.f };
    // ResolveDebug: sky pixels get a checkerboard of 4x4 tiles; layers other than the surface
    // ones need no surface
    const uint32_t background = ((x0 ^ y0) & 4) ? 0xFFA0A0A0u : 0xFFFFFFFFu;
    if constexpr (kMode == kResolveDebug) {
        if (skyBits == 0xFFFF || a.debugLayer - 1u >= 3u) {
            a.color[off] = isSky ? background : debug_pixel(a.debugLayer, id, 0u, F3{}, 0.0f, 0.0f);
            return;
        }
    }
    if constexpr (kMode == kResolveEmit) {
        if (skyBits == 0xFFFF) {
            nr.surf[nr.pixels + off] = make_uint4(0u, 0u, 0u, 0u);  // nothing to decode
            return;
        }
    }
    if (skyBits != 0xFFFF) {
        uint32_t ntg[3] = {}, hand = 0, albedo = 0, nmr = 0;
        float b[3];
        bool fast = false;  // the neural pass found the emit pass's records for the whole tile
        if constexpr (kMode == kResolveNeural) {
            uint4 s0 = make_uint4(0u, 0u, 0u, 0u), s1 = make_uint4(0u, 0u, 0u, 0u);
            if (!isSky) s0 = nr.surf[off], s1 = nr.surf[nr.pixels + off];
            fast = (__ballot_sync(hm, isSky || (s1.y & kSurfFast)) & hm) == hm;
            if (fast) {
                const float nan = __int_as_float(0x7FFFFFFF);  // what the full path gives sky pixels
                b[1] = isSky ? nan : __uint_as_float(s0.x);
                b[2] = isSky ? nan : __uint_as_float(s0.y);
                b[0] = 1 - b[1] - b[2];
                ntg[0] = s0.z, ntg[1] = s0.w, ntg[2] = s1.x;
                hand = s1.y & kSurfHand;
                if (!isSky && (s1.y & kSurfDecoded)) {
                    auto at = [&](uint32_t k) { return nr.decoded[(size_t)((off & ~15u) + ((s1.w >> (16 + 4 * k)) & 15u)) * 4 + k]; };
                    const bool inX = s1.y & kSurfInX, inY = s1.y & kSurfInY;
                    const uint2 d00 = at(0);
                    uint2 r0 = d00;
                    if (!(s1.y & kSurfNearest)) {
                        const uint2 d10 = inX ? at(1) : d00, d01 = inY ? at(2) : d00;
                        const uint2 d11 = inY ? (inX ? at(3) : d01) : d10;
                        const uint32_t fx = packed_weight((s1.y >> 8) & 255u), fy = packed_weight((s1.y >> 16) & 255u);
                        r0.x = filter_rgba8(d00.x, d10.x, d01.x, d11.x, fx, fy);
                        r0.y = filter_rgba8(d00.y, d10.y, d01.y, d11.y, fx, fy);
                    }
                    albedo = r0.x;
                    if (s1.y & kSurfTwoLayers) nmr = r0.y;
                }
            }
        }
        if (!fast) {
        // ---- ResolveSurface (Shading.cpp:471-579). The reference's waterfall over the tile's surface ids loads
        // each id's record for the lanes that hold it; here every lane loads its own (a pixel without a
        // surface takes part only if a covered pixel holds its id). A tile of small triangles had one
        // round of dependent loads per id.
        F3 pos[3] = {};
        uint32_t tc[3] = {}, matId = 0;
        uint32_t sflags = kSurfFast, stexel = 0, slead = 0;  // the emit pass's record of this pixel
        const unsigned covered = ((~skyBits) & 0xFFFF) << (16 * half);
        const bool holds = skyBits == 0 || (__match_any_sync(hm, id) & covered) != 0;
        const uint32_t mId = id / 128, tri = id % 128;
        if (holds && mId < a.numMeshlets) {
            const uint8_t* mp = a.meshlets + (size_t)mId * kMeshletSize;
            const float* P = (const float*)(mp + kOffPositions);
            const uint32_t* TC = (const uint32_t*)(mp + kOffTexCoords);
            const uint32_t* NT = (const uint32_t*)(mp + kOffNormalTangents);
            const uint8_t* I = mp + kOffIndices;
            const unsigned long long handBits = *(const unsigned long long*)(mp + kOffHandedness);
#pragma unroll
            for (int vi = 0; vi < 3; vi++) {
                const uint32_t idx = I[vi * 128 + tri] & 63;
                pos[vi] = { P[idx], P[64 + idx], P[128 + idx] };
                tc[vi] = TC[idx];
                ntg[vi] = NT[idx];
                if (vi == 0 && ((handBits >> idx) & 1)) hand = 1u << 31;
            }
            matId = *(const uint32_t*)(mp + kOffMaterialId);
        }
        // IntersectTriangle (Shading.cpp:417-464)
        float w0, w1, w2;
        F3 c0 = xform4(a.objectToClip, pos[0], w0), c1 = xform4(a.objectToClip, pos[1], w1), c2 = xform4(a.objectToClip, pos[2], w2);
        const float iw0 = 1.0f / w0, iw1 = 1.0f / w1, iw2 = 1.0f / w2;
        const float p0x = c0.x * iw0, p0y = c0.y * iw0, p1x = c1.x * iw1, p1y = c1.y * iw1, p2x = c2.x * iw2, p2y = c2.y * iw2;
        const float m0x = p2x - p1x, m0y = p2y - p1y, m1x = p0x - p1x, m1y = p0y - p1y;
        const float invDet = 1.0f / (m0x * m1y - m1x * m0y);
        const float s0 = invDet * iw0, s1 = invDet * iw1, s2 = invDet * iw2;
        float dx[3] = { (p1y - p2y) * s0, (p2y - p0y) * s1, (p0y - p1y) * s2 };
        float dy[3] = { (p2x - p1x) * s0, (p0x - p2x) * s1, (p1x - p0x) * s2 };
        float dxs = dx[0] + dx[1] + dx[2], dys = dy[0] + dy[1] + dy[2];
        const float r0x = su - p0x, r0y = sv - p0y;
        const float interpInvW = iw0 + r0x * dxs + r0y * dys;
        const float interpW = 1.0f / interpInvW;
        b[1] = interpW * (r0x * dx[1] + r0y * dy[1]);
        b[2] = interpW * (r0x * dx[2] + r0y * dy[2]);
        b[0] = 1 - b[1] - b[2];
        const float kx = 2.0f / W, ky = -(2.0f / H);
#pragma unroll
        for (int k = 0; k < 3; k++) dx[k] *= kx, dy[k] *= ky;
        dxs *= kx, dys *= ky;
        const float wdx = 1.0f / (interpInvW + dxs), wdy = 1.0f / (interpInvW + dys);
#pragma unroll
        for (int k = 0; k < 3; k++) {
            dx[k] = wdx * (b[k] * interpInvW + dx[k]) - b[k];
            dy[k] = wdy * (b[k] * interpInvW + dy[k]) - b[k];
        }
        const float t0x = h2f(tc[0] & 0xFFFF), t0y = h2f(tc[0] >> 16);
        const float t10x = h2f(tc[1] & 0xFFFF) - t0x, t10y = h2f(tc[1] >> 16) - t0y;
        const float t20x = h2f(tc[2] & 0xFFFF) - t0x, t20y = h2f(tc[2] >> 16) - t0y;
        const float texU = t0x + t10x * b[1] + t20x * b[2];
        const float texV = t0y + t10y * b[1] + t20y * b[2];
        const float g0 = t10x * dx[1] + t20x * dx[2], g1 = t10y * dx[1] + t20y * dx[2];
        const float g2 = t10x * dy[1] + t20x * dy[2], g3 = t10y * dy[1] + t20y * dy[2];

        // Materials. The reference's waterfall picks the filter over the whole tile per material: nearest if
        // any of the 16 pixels' gradients, scaled by that material's texture, calls for a level above 0.
        // Textures of one size (the usual case) give one answer; others are asked per material.
        bool sampled = (skyBits == 0 || (__match_any_sync(hm, matId) & covered) != 0) && matId < a.numMaterials;
        if (sampled) sampled = a.materials[matId].has_texture;
        const unsigned sampledBits = __ballot_sync(hm, sampled) & hm;
        if (sampledBits) {
            const DevTexture& tex = a.materials[sampled ? matId : 0].tex;
            const float d1 = fmaf(g0, g0, g1 * g1), d2 = fmaf(g2, g2, g3 * g3);
            const float sU = sampled ? tex.scale_u : 0.0f, sV = sampled ? tex.scale_v : 0.0f;
            const float lU = __shfl_sync(hm, sU, __ffs(sampledBits) - 1), lV = __shfl_sync(hm, sV, __ffs(sampledBits) - 1);
            auto level = [&](float u, float v) { return ilog2_x86(vmax(d1 * (u * u), d2 * (v * v))) >> 1; };
            int32_t mip = level(lU, lV);
            bool nearest = __ballot_sync(hm, mip > 0) & hm;
            if (__ballot_sync(hm, sampled && (sU != lU || sV != lV)) & hm) {
                unsigned pm = sampledBits;
                while (pm) {
                    const int src = __ffs(pm) - 1;
                    const uint32_t mid = __shfl_sync(hm, matId, src);
                    const float u = __shfl_sync(hm, sU, src), v = __shfl_sync(hm, sV, src);
                    const unsigned iter = __ballot_sync(hm, matId == mid) & hm;
                    pm &= ~iter;
                    const int32_t m = level(u, v);
                    const bool n = __ballot_sync(hm, m > 0) & hm;
                    if (matId == mid) mip = m, nearest = n;
                }
            }
            const TexelQuad q = texel_quad(tex, texU, texV, mip, nearest);
            const uint32_t mid = matId;
            // decoded when the model covers the level and its texture has this texture's size
            bool dec = false;
            if constexpr (kMode == kResolveEmit || kMode == kResolveNeural)
                dec = sampled && mid < nr.numMaterials && q.m < (int32_t)nr.decodedLevels && nr.tex[mid].data != nullptr &&
                      nr.tex[mid].width == tex.width && nr.tex[mid].height == tex.height;
            if constexpr (kMode == kResolveEmit) {
                uint32_t nq = 0;
                if (sampled)
                    sflags = dec ? kSurfFast | kSurfDecoded | (nearest ? kSurfNearest : 0u) | (q.inX ? kSurfInX : 0u) |
                                       (q.inY ? kSurfInY : 0u) | (tex.num_layers >= 2 ? kSurfTwoLayers : 0u) |
                                       (surf_weight(q.fx) << 8) | (surf_weight(q.fy) << 16)
                                 : 0u;  // sampled from the plain texture: the second pass reconstructs
                if (dec) stexel = ((uint32_t)q.m << 28) | ((uint32_t)q.ty << 14) | (uint32_t)q.tx;
                slead = dec ? mid : 0u;
                // a slot's leader: the lowest lane with its texel in the slot, of the same material
                const unsigned sameMaterial = __match_any_sync(hm, dec ? mid : ~0u);
#pragma unroll
                for (uint32_t k = 0; k < 4; k++) {
                    const bool has = dec && surf_has_slot(sflags, k);
                    const uint32_t texel = has ? surf_slot_texel(stexel, k) : ~0u;
                    const int lead = __ffs(__match_any_sync(hm, texel) & sameMaterial) - 1;
                    if (!has) continue;
                    slead |= ((uint32_t)lead & 15u) << (16 + 4 * k);
                    if (lead == (int)lane) nq++;
                }
                unsigned pm = __ballot_sync(hm, nq != 0) & hm;
                while (pm) {  // the requests of each of the tile's materials
                    const uint32_t m = __shfl_sync(hm, mid, __ffs(pm) - 1);
                    const unsigned iter = __ballot_sync(hm, nq != 0 && mid == m) & hm;
                    pm &= ~iter;
                    if ((iter >> lane) & 1) {
                        const uint32_t total = __reduce_add_sync(iter, nq);
                        if ((int)lane == __ffs(iter) - 1)
                            atomicAdd(&nr.counts[(blockIdx.x % kCountCopies) * count_stride(nr.numMaterials) + m], total);
                    }
                }
            } else if (dec) {
                const uint32_t leads = nr.surf[nr.pixels + off].w >> 16;
                auto at = [&](uint32_t k) { return nr.decoded[(size_t)((off & ~15u) + ((leads >> (4 * k)) & 15u)) * 4 + k]; };
                const uint2 d00 = at(0);
                uint2 r0 = d00;
                if (!nearest) {
                    const uint2 d10 = q.inX ? at(1) : d00, d01 = q.inY ? at(2) : d00;
                    const uint2 d11 = q.inY ? (q.inX ? at(3) : d01) : d10;
                    r0.x = filter_rgba8(d00.x, d10.x, d01.x, d11.x, q.fx, q.fy);
                    r0.y = filter_rgba8(d00.y, d10.y, d01.y, d11.y, q.fx, q.fy);
                }
                albedo = r0.x;
                if (tex.num_layers >= 2) nmr = r0.y;
            } else if (sampled) {
                albedo = sample_quad(tex, q, 0, nearest);
                if (tex.num_layers >= 2) nmr = sample_quad(tex, q, 1, nearest);
            }
        }
        if constexpr (kMode == kResolveEmit) {
            nr.surf[off] = make_uint4(__float_as_uint(b[1]), __float_as_uint(b[2]), ntg[0], ntg[1]);
            nr.surf[nr.pixels + off] = make_uint4(ntg[2], sflags | hand, stexel, slead);
            return;
        }
        }  // !fast
        F3 nrm[3];
        unpack_units(a.octTable, ntg, nrm);
        const float* M = a.objectToWorld;
        auto bl = [&](const F3* v) {
            return F3{ fmaf(v[0].x, b[0], fmaf(v[1].x, b[1], v[2].x * b[2])), fmaf(v[0].y, b[0], fmaf(v[1].y, b[1], v[2].y * b[2])),
                       fmaf(v[0].z, b[0], fmaf(v[1].z, b[1], v[2].z * b[2])) };
        };
        auto m3 = [&](F3 n) {
            return F3{ fmaf(n.x, M[0], fmaf(n.y, M[3], n.z * M[6])), fmaf(n.x, M[1], fmaf(n.y, M[4], n.z * M[7])),
                       fmaf(n.x, M[2], fmaf(n.y, M[5], n.z * M[8])) };
        };
        const F3 nws = normalize3(m3(bl(nrm)));
        F3 N = nws;
        if (__ballot_sync(hm, (nmr & 0xFFFF) != 0) & hm) {
            F3 tan[3];
            const uint32_t tw[3] = { ntg[0] >> 16, ntg[1] >> 16, ntg[2] >> 16 };
            unpack_units(a.octTable, tw, tan);
            const F3 tws = normalize3(m3(bl(tan)));
            F3 bws = { fmaf(nws.y, tws.z, -nws.z * tws.y), fmaf(nws.z, tws.x, -nws.x * tws.z), fmaf(nws.x, tws.y, -nws.y * tws.x) };
            bws = { __uint_as_float(__float_as_uint(bws.x) ^ hand), __uint_as_float(__float_as_uint(bws.y) ^ hand),
                    __uint_as_float(__float_as_uint(bws.z) ^ hand) };
            const float tx_ = (float)(nmr & 255) * (1.0f / 127.5f) - 1.0f;
            const float ty_ = (float)((nmr >> 8) & 255) * (1.0f / 127.5f) - 1.0f;
            const float tz_ = approx_sqrt(1.0f - (tx_ * tx_ + ty_ * ty_));
            N = normalize3({ tx_ * tws.x + ty_ * bws.x + tz_ * nws.x, tx_ * tws.y + ty_ * bws.y + tz_ * nws.y,
                             tx_ * tws.z + ty_ * bws.z + tz_ * nws.z });
        }
        const float metallic = (float)((nmr >> 16) & 255) * (1.0f / 255);
        const float roughness = (float)((nmr >> 24) & 255) * (1.0f / 255);
        if constexpr (kMode == kResolveDebug) {
            a.color[off] = isSky ? background : debug_pixel(a.debugLayer, id, albedo, N, metallic, roughness);
            return;
        }

        // ---- EvalLighting (Shading.cpp:602-645)
        const float invPi = 0.3183098861837907f;
        uint32_t rb1 = ((albedo << 8) & 0xFF00FF00u) + 0x00FF00FFu, ag1 = (albedo & 0xFF00FF00u) + 0x00FF00FFu;
        uint32_t rb2 = (((rb1 & 0xFFFF) * (rb1 & 0xFFFF)) >> 16) | ((((rb1 >> 16) * (rb1 >> 16)) >> 16) << 16);
        uint32_t ag2 = (((ag1 & 0xFFFF) * (ag1 & 0xFFFF)) >> 16) | ((((ag1 >> 16) * (ag1 >> 16)) >> 16) << 16);
        const float s65 = 1.0f / 65535;
        const F3 base = { (float)(rb2 & 65535) * s65, (float)(ag2 & 65535) * s65, (float)(rb2 >> 16) * s65 };
        const float alphaR = vmax(roughness * roughness, 1e-4f);
        const float f0d = 0.16f * 0.5f * 0.5f;
        const F3 f0 = { lerpf(f0d, base.x, metallic), lerpf(f0d, base.y, metallic), lerpf(f0d, base.z, metallic) };
        const float dm = 1.0f - metallic;
        const F3 diffuse = { base.x * dm, base.y * dm, base.z * dm };
        const F3 vp = { a.viewPos[0], a.viewPos[1], a.viewPos[2] };
        const F3 viewDir = normalize3({ vp.x - world.x, vp.y - world.y, vp.z - world.z });
        const float NoV = fabsf(dot3(N, viewDir)) + 1e-5f;
        const float exposure = a.exposure * 0.001f;
        for (uint32_t i = 0; i < a.numLights; i++) {
            const swr_light& li = a.lights ? a.lights[i] : a.light[i];
            F3 ld = li.type == 0 ? F3{ -li.direction[0], -li.direction[1], -li.direction[2] }
                                 : normalize3({ li.position[0] - world.x, li.position[1] - world.y, li.position[2] - world.z });
            const float NoL = dot3(N, ld);
            if ((__ballot_sync(hm, NoL < 1e-4f) & hm) == hm) continue;
            float att = 1.0f;
            if (li.type != 0) {
                const F3 p2l = { li.position[0] - world.x, li.position[1] - world.y, li.position[2] - world.z };
                const float d2 = dot3(p2l, p2l);
                const float f = d2 * li.inv_radius_sq;
                const float sm = vmax(1.0f - f * f, 0.0f);
                att = (sm * sm) * approx_rcp(vmax(d2, 1e-4f));
                if (li.type == 2) {
                    const float cd = dot3({ -li.direction[0], -li.direction[1], -li.direction[2] }, normalize3(p2l));
                    const float sa = vmin(vmax(cd * li.spot_scale + li.spot_offset, 0.0f), 1.0f);
                    att *= sa * sa;
                }
            }
            att = att * li.intensity * exposure;
            if ((__ballot_sync(hm, NoL * att < 1e-4f) & hm) == hm) continue;
            const F3 h = normalize3({ viewDir.x + ld.x, viewDir.y + ld.y, viewDir.z + ld.z });
            const float NoH = vmin(vmax(dot3(N, h), 0.0f), 1.0f);
            const float LoH = vmin(vmax(dot3(ld, h), 0.0f), 1.0f);
            const float aa = NoH * alphaR;
            const float k = alphaR * approx_rcp(1.0f - NoH * NoH + aa * aa);
            const float D = k * k * invPi;
            const float V = 0.5f / lerpf(2.0f * NoL * NoV, NoL + NoV, alphaR);
            const float x = 1.0f - LoH;
            const float f = (x * x) * (x * x) * x;
            const F3 F = { f + f0.x * (1.0f - f), f + f0.y * (1.0f - f), f + f0.z * (1.0f - f) };
            const float DV = D * V;
            const float wgt = vmax(NoL * att, 0.0f);
            color.x += (diffuse.x * invPi + DV * F.x) * li.color[0] * wgt;
            color.y += (diffuse.y * invPi + DV * F.y) * li.color[1] * wgt;
            color.z += (diffuse.z * invPi + DV * F.z) * li.color[2] * wgt;
        }
        color.x += base.x * 0.05f;
        color.y += base.y * 0.05f;
        color.z += base.z * 0.05f;
    }
    if (skyBits != 0 && a.hasSky && isSky) color = sample_env(a.sky, { world.x - a.viewPos[0], world.y - a.viewPos[1], world.z - a.viewPos[2] });
    // Tonemap_Unreal (Shading.cpp:221-226) + RGBA8u::Pack
    const float e = a.exposure;
    const F3 c = { color.x * e, color.y * e, color.z * e };
    const uint32_t r = sat_u8(round2i(c.x / (c.x + 0.155f) * 1.019f * 255.0f));
    const uint32_t g = sat_u8(round2i(c.y / (c.y + 0.155f) * 1.019f * 255.0f));
    const uint32_t bch = sat_u8(round2i(c.z / (c.z + 0.155f) * 1.019f * 255.0f));
    a.color[off] = r | (g << 8) | (bch << 16) | (255u << 24);
}

}  // namespace

cudaError_t fill_oct_table(float4* table) {
    cudaStream_t st = nullptr;
    cudaError_t e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
    if (e != cudaSuccess) return e;
    {
        LaunchScope ls("k_oct_table", st);
        k_oct_table<<<kOctTable / 256, 256, 0, st>>>(table);
        e = cudaGetLastError();
    }
    const cudaError_t w = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = w;
    cudaStreamDestroy(st);
    return e;
}
}  // namespace swr

using namespace swr;

namespace {
// ShadingContext::Resolve's per-frame constants (Shading.cpp:658-690); the lights are copied to a
// stream-ordered device allocation that the caller frees after the launch.
// takesKeys: the kernel reads pending draws of both layers from the keys (it sets a.keys then); else they
// are written to the layers first.
swr_status build_resolve_args(swr_framebuffer fb, const swr_shading_context* ctx, ResolveArgs& a, const char* fn, bool takesKeys) {
    if (!fb || !ctx || !ctx->scene) return swr_internal_fail(SWR_EINVAL, (std::string(fn) + ": NULL argument").c_str());
    if (ctx->num_lights && !ctx->lights) return swr_internal_fail(SWR_EINVAL, (std::string(fn) + ": lights is NULL").c_str());
    if (ctx->skybox && ctx->skybox->format != SWR_FORMAT_R11G11B10F)
        return swr_internal_fail(SWR_EINVAL, (std::string(fn) + ": the skybox must be R11G11B10f").c_str());
    takesKeys = takesKeys && fb->layers_stale == kStaleAll;
    swr_status fst = takesKeys ? SWR_OK : swr_internal_finalize(fb);
    if (fst != SWR_OK) return fst;
    cudaStream_t st = swr_internal_stream();
    a = {};
    a.keys = takesKeys ? fb->keys : nullptr;
    a.meshlets = ctx->scene->meshlets;
    a.numMeshlets = ctx->scene->count;
    a.materials = ctx->scene->materials;
    a.numMaterials = ctx->scene->num_materials;
    a.octTable = ctx->scene->octTable.get();
    a.color = fb->layers;
    a.depth = (float*)(fb->layers + fb->layer_stride);
    a.width = fb->width, a.height = fb->height;
    memcpy(a.objectToClip, ctx->object_to_clip, sizeof(a.objectToClip));
    memcpy(a.objectToWorld, ctx->object_to_world, sizeof(a.objectToWorld));
    if (!swr_hostmath::inverse_screen_proj(ctx->world_to_clip, fb->width, fb->height, a.invProj))
        return swr_internal_fail(SWR_EINVAL, (std::string(fn) + ": singular world_to_clip").c_str());
    memcpy(a.viewPos, ctx->view_pos, sizeof(a.viewPos));
    a.exposure = ctx->exposure;
    if (ctx->skybox) a.sky = ctx->skybox->d, a.hasSky = 1;
    if (ctx->num_lights && ctx->num_lights <= kParamLights) {
        memcpy(a.light, ctx->lights, ctx->num_lights * sizeof(swr_light));
    } else if (ctx->num_lights) {
        swr_light* dl = nullptr;
        cudaError_t e = cudaMallocAsync(&dl, ctx->num_lights * sizeof(swr_light), st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(dl, ctx->lights, ctx->num_lights * sizeof(swr_light), cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) return swr_internal_cuda_fail(e, fn);
        a.lights = dl;
    }
    a.numLights = ctx->num_lights;
    return SWR_OK;
}
}  // namespace

extern "C" {

swr_status swr_cull_meshlets(swr_scene s, uint32_t first, uint32_t count, uint16_t* bitmap_device, const float proj[16],
                             const float view[16], const float model[16], const float prev_view[16], float frame_width,
                             float frame_height, swr_texture depth_map, uint32_t* visible_count) {
    return swr_cull_meshlets_ex(s, first, count, bitmap_device, proj, view, model, prev_view, frame_width, frame_height,
                                depth_map, visible_count, 0u);
}

swr_status swr_cull_meshlets_ex(swr_scene s, uint32_t first, uint32_t count, uint16_t* bitmap_device, const float proj[16],
                                const float view[16], const float model[16], const float prev_view[16], float frame_width,
                                float frame_height, swr_texture depth_map, uint32_t* visible_count, uint32_t flags) {
    if (!s || !bitmap_device || !proj || !view || !model || !prev_view)
        return swr_internal_fail(SWR_EINVAL, "swr_cull_meshlets: NULL argument");
    if (flags & ~(uint32_t)SWR_CULL_BACKFACE_CONE) return swr_internal_fail(SWR_EINVAL, "swr_cull_meshlets_ex: unknown flags");
    if ((uint64_t)first + count > s->count) return swr_internal_fail(SWR_EINVAL, "swr_cull_meshlets: range outside the scene");
    if (depth_map && depth_map->format != SWR_FORMAT_R32F)
        return swr_internal_fail(SWR_EINVAL, "swr_cull_meshlets: the depth map must be R32f");
    if (!(frame_width >= 1.0f && frame_width <= 65536.0f && frame_height >= 1.0f && frame_height <= 65536.0f))
        return swr_internal_fail(SWR_EINVAL, "swr_cull_meshlets: frame size outside [1, 65536]");
    // Texel reads stay inside the map when it is at least half the frame in each dimension (the
    // frame driver's sizing, Main.cpp:54-56) and has two levels (mip clamps to [1, levels-1]).
    if (depth_map && ((float)(depth_map->d.width * 2) < frame_width || (float)(depth_map->d.height * 2) < frame_height ||
                      depth_map->d.mip_levels < 2))
        return swr_internal_fail(SWR_EINVAL, "swr_cull_meshlets: depth map smaller than half the frame or without mips");
    cudaStream_t st = swr_internal_stream();
    CullArgs a = {};
    a.meshlets = s->meshlets;
    a.first = first, a.count = count;
    a.bitmap = bitmap_device;
    float objToPrev[16], pv[16], objToClip[16], planes[6][4];
    swr_hostmath::mat4_mul(prev_view, model, objToPrev);
    swr_hostmath::mat4_mul(proj, view, pv);
    swr_hostmath::mat4_mul(pv, model, objToClip);
    swr_hostmath::frustum_planes(objToClip, planes);
    memcpy(a.planes, planes, sizeof(a.planes));  // planes 0..4 (the reference skips the last, Shading.cpp:806)
    if (flags & SWR_CULL_BACKFACE_CONE) {
        a.cone = swr_hostmath::cone_camera(objToClip, a.eye) ? 1u : 0u;
        a.materials = s->materials;
        a.numMaterials = s->num_materials;
    }
    memcpy(a.objectToPrevView, objToPrev, sizeof(objToPrev));
    a.objectToWorldScale = swr_hostmath::column0_length(model);
    a.projFactors[0] = proj[3 * 4 + 2], a.projFactors[1] = proj[0], a.projFactors[2] = proj[1 * 4 + 1];
    a.frameW = frame_width, a.frameH = frame_height;
    if (depth_map) {
        a.depthData = depth_map->d.data;
        memcpy(a.mipOffsets, depth_map->d.mip_offsets, sizeof(a.mipOffsets));
        a.mipLevels = depth_map->d.mip_levels;
        a.rowShift = depth_map->d.row_shift;
    }
    unsigned int* cnt = nullptr;
    cudaError_t e = cudaSuccess;
    if (visible_count) {
        e = cudaMallocAsync(&cnt, sizeof(unsigned int), st);
        if (e == cudaSuccess) e = cudaMemsetAsync(cnt, 0, sizeof(unsigned int), st);
        if (e != cudaSuccess) return swr_internal_cuda_fail(e, "swr_cull_meshlets");
        a.visibleCount = cnt;
    }
    if (count) {
        LaunchScope ls("k_cull", st);
        k_cull<<<(count + 255) / 256, 256, 0, st>>>(a);
        e = cudaGetLastError();
    }
    if (visible_count) {
        unsigned int h = 0;
        if (e == cudaSuccess) e = cudaMemcpyAsync(&h, cnt, sizeof(h), cudaMemcpyDeviceToHost, st);
        cudaFreeAsync(cnt, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        *visible_count = h;
    }
    if (e != cudaSuccess) return swr_internal_cuda_fail(e, "swr_cull_meshlets");
    return SWR_OK;
}

swr_status swr_downsample_depth(swr_framebuffer fb, swr_texture dest) {
    if (!fb || !dest) return swr_internal_fail(SWR_EINVAL, "swr_downsample_depth: NULL argument");
    if (dest->format != SWR_FORMAT_R32F) return swr_internal_fail(SWR_EINVAL, "swr_downsample_depth: destination must be R32f");
    swr_status fst = swr_internal_finalize(fb);
    if (fst != SWR_OK) return fst;
    const uint32_t root = 32 - __builtin_clz(std::max(fb->width, fb->height));
    if (root < 4) return swr_internal_fail(SWR_EINVAL, "swr_downsample_depth: framebuffer smaller than 16 pixels");
    cudaStream_t st = swr_internal_stream();
    const float* depth = (const float*)(fb->layers + fb->layer_stride);
    uint32_t* tex = (uint32_t*)dest->d.data;
    auto blocks = [&](uint32_t m, uint32_t& rx, uint32_t& ry, uint32_t& bt) {
        if (m + 4 <= root) {
            const uint32_t region = 1u << (m + 4);
            rx = (fb->width + region - 1) / region, ry = (fb->height + region - 1) / region, bt = 64;
        } else {
            rx = ry = 1, bt = 16;
        }
    };
    // Levels the texture does not have use MipOffsets[m] = 0, as the reference's zero-filled table
    // does (for non-square frames its root tile lands at the start of mip 0). Every written texel
    // must fall inside the texture's storage.
    auto mipOff = [&](uint32_t m) { return m < dest->d.mip_levels ? dest->d.mip_offsets[m] : 0u; };
    for (uint32_t m = 0; m + 3 <= root; m++) {
        uint32_t rx, ry, bt;
        blocks(m, rx, ry, bt);
        const uint32_t side = bt == 64 ? 8 : 4;
        const int32_t stride = (int32_t)dest->d.row_shift - (int32_t)m;
        const uint64_t maxX = (uint64_t)rx * side - 1, maxY = (uint64_t)ry * side - 1;
        if (stride < 0 || mipOff(m) + 7 + (maxX << 3) + (maxY << stride) >= dest->words)
            return swr_internal_fail(SWR_EINVAL, "swr_downsample_depth: destination too small for this framebuffer");
    }
    // The levels above k_hiz_local's that the texture lacks land at its start one after the other (k_hiz_tail). Where more
    // words are shared, blocks writing them at once would leave them to whichever came last: by the lower levels of
    // a texture of fewer than 4, by the texels of a level wider than the texture's, or by a level that reaches into
    // the next. Such a texture gets its levels from a scratch pyramid in which nothing is shared, one launch a level.
    const uint32_t levels = dest->d.mip_levels;
    bool place = levels < std::min(root - 3, 4u);
    uint32_t columns = 8;
    for (uint32_t m = 0; m + 3 <= root; m++) {
        uint32_t rx, ry, bt;
        blocks(m, rx, ry, bt);
        const uint32_t side = bt == 64 ? 8 : 4, cols = rx * side, rows = ry * side, stride = dest->d.row_shift - m;
        columns = std::max(columns, cols << m);
        place = place || (cols > 1u << stride && rows > 8);
        const uint64_t end = 8 * (uint64_t)cols + ((uint64_t)((rows - 1) & ~7u) << stride);
        place = place || (m + 1 < levels && m + 4 <= root && end > dest->d.mip_offsets[m + 1] - dest->d.mip_offsets[m]);
    }
    HizOffsets offs = {};
    uint32_t* pyramid = tex;
    int32_t rowShift = (int32_t)dest->d.row_shift;
    cudaError_t e = cudaSuccess;
    if (place) {
        rowShift = 32 - __builtin_clz(columns - 1);  // as wide as the widest level
        size_t words = 0;
        for (uint32_t m = 0; m + 3 <= root; m++) {
            uint32_t rx, ry, bt;
            blocks(m, rx, ry, bt);
            const uint32_t side = bt == 64 ? 8 : 4;
            offs.off[m] = (uint32_t)words;
            words += (size_t)((ry * side + 7) / 8) << (rowShift - (int32_t)m + 3);
        }
        e = cudaMallocAsync(&pyramid, words * sizeof(uint32_t), st);
        if (e != cudaSuccess) return swr_internal_cuda_fail(e, "swr_downsample_depth: scratch");
    } else {
        for (uint32_t m = 0; m + 3 <= root && m < 16; m++) offs.off[m] = mipOff(m);
    }
    const uint32_t nLocal = std::min(root - 3, place ? 7u : std::min(7u, levels));  // levels with 8x8-texel blocks
    {
        LaunchScope ls("k_hiz_local", st);
        // whole blocks of the highest level
        const uint32_t side = std::max(kHizRegion, 8u << nLocal), per = side / kHizRegion;
        const dim3 grid((fb->width + side - 1) / side * per, (fb->height + side - 1) / side * per);
        k_hiz_local<<<grid, 1024, 0, st>>>(depth, fb->width, fb->height, pyramid, offs, rowShift, nLocal);
    }
    if (root - 3 >= nLocal) {
        size_t smem = 0;  // levels nLocal-1 .. root-3, texels whose origin lies in the frame
        for (uint32_t m = nLocal - 1; m <= root - 3; m++)
            smem += (size_t)hiz_extent(fb->width, m) * hiz_extent(fb->height, m) * sizeof(float);
        if (smem > 48 * 1024) cudaFuncSetAttribute(k_hiz_tail, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        LaunchScope ls("k_hiz_tail", st);
        k_hiz_tail<<<1, 1024, smem, st>>>(fb->width, fb->height, pyramid, offs, rowShift, nLocal, root - 3,
                                           root);
    }
    if (place) {
        for (uint32_t m = 0; m + 3 <= root; m++) {
            uint32_t rx, ry, bt;
            blocks(m, rx, ry, bt);
            const uint32_t side = bt == 64 ? 8 : 4, cols = rx * side, rows = ry * side;
            LaunchScope ls("k_hiz_place", st);
            k_hiz_place<<<std::min((cols * rows + 255) / 256, 1216u), 256, 0, st>>>(
                pyramid + offs.off[m], rowShift - (int32_t)m, tex + mipOff(m), (int32_t)(dest->d.row_shift - m), cols, rows);
        }
        e = cudaGetLastError();
        cudaFreeAsync(pyramid, st);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) return swr_internal_cuda_fail(e, "swr_downsample_depth");
    return SWR_OK;
}

swr_status swr_resolve(swr_rasterizer r, swr_framebuffer fb, const swr_shading_context* ctx) {
    (void)r;
    ResolveArgs a = {};
    swr_status s = build_resolve_args(fb, ctx, a, "swr_resolve", true);
    if (s != SWR_OK) return s;
    cudaStream_t st = swr_internal_stream();
    const uint32_t tiles = (fb->width / 4) * (fb->height / 4);
    cudaError_t e;
    {
        LaunchScope ls("k_resolve", st);
        k_resolve<kResolvePlain><<<(tiles * 16 + 255) / 256, 256, 0, st>>>(a, NeuralResolve{});
        e = cudaGetLastError();
    }
    if (a.lights) cudaFreeAsync((void*)a.lights, st);
    if (e != cudaSuccess) return swr_internal_cuda_fail(e, "swr_resolve");
    fb->layers_stale = kStaleNone;
    fb->keys_valid = false;  // layer 0 now holds colour; a later draw rebuilds its keys from depth
    return SWR_OK;
}

swr_status swr_resolve_debug(swr_rasterizer r, swr_framebuffer fb, const swr_shading_context* ctx, uint32_t layer) {
    (void)r;
    if (layer > SWR_DEBUG_OVERDRAW_QUAD) return swr_internal_fail(SWR_EINVAL, "swr_resolve_debug: unknown debug layer");
    ResolveArgs a = {};
    swr_status s = build_resolve_args(fb, ctx, a, "swr_resolve_debug", false);
    if (s != SWR_OK) return s;
    a.debugLayer = layer;
    cudaStream_t st = swr_internal_stream();
    const uint32_t tiles = (fb->width / 4) * (fb->height / 4);
    cudaError_t e;
    {
        LaunchScope ls("k_resolve_debug", st);
        k_resolve<kResolveDebug><<<(tiles * 16 + 255) / 256, 256, 0, st>>>(a, NeuralResolve{});
        e = cudaGetLastError();
    }
    if (a.lights) cudaFreeAsync((void*)a.lights, st);
    if (e != cudaSuccess) return swr_internal_cuda_fail(e, "swr_resolve_debug");
    fb->keys_valid = false;  // layer 0 now holds colour
    return SWR_OK;
}

swr_status swr_resolve_neural(swr_rasterizer r, swr_framebuffer fb, const swr_shading_context* ctx, swr_neural n,
                              swr_neural_stats* stats) {
    (void)r;
    if (!n) return swr_internal_fail(SWR_EINVAL, "swr_resolve_neural: NULL model");
    ResolveArgs a = {};
    swr_status s = build_resolve_args(fb, ctx, a, "swr_resolve_neural", true);
    if (s != SWR_OK) return s;
    cudaStream_t st = swr_internal_stream();
    const uint32_t M = n->d.numMaterials;
    const size_t slots = (size_t)fb->width * fb->height * 4;
    cudaError_t e = cudaSuccess;
    if (n->scratchSlots < slots) {
        if (n->sorted) cudaFree(n->sorted);
        if (n->decoded) cudaFree(n->decoded);
        if (n->surf) cudaFree(n->surf);
        n->sorted = nullptr, n->decoded = nullptr, n->surf = nullptr, n->scratchSlots = 0;
        e = cudaMalloc(&n->sorted, slots * sizeof(unsigned long long));
        if (e == cudaSuccess) e = cudaMalloc(&n->decoded, slots * sizeof(uint2));
        if (e == cudaSuccess) e = cudaMalloc(&n->surf, slots / 4 * 2 * sizeof(uint4));
        if (e != cudaSuccess) {
            if (a.lights) cudaFreeAsync((void*)a.lights, st);
            return swr_internal_cuda_fail(e, "swr_resolve_neural: scratch");
        }
        n->scratchSlots = slots;
    }
    neural_sync_half(n, st);
    uint32_t* counts = n->counters;
    uint32_t* cursor = counts + kCountCopies * count_stride(M);
    uint32_t* reqOffset = cursor + (M + 1);
    uint32_t* tileOffset = reqOffset + (M + 1);
    uint32_t* levelCount = tileOffset + (M + 1);
    NeuralResolve nr = {};
    nr.tex = n->d.tex, nr.numMaterials = M, nr.decodedLevels = n->d.levels + 2;
    nr.counts = counts, nr.decoded = n->decoded, nr.surf = n->surf, nr.pixels = (uint32_t)(slots / 4);
    const uint32_t tiles = (fb->width / 4) * (fb->height / 4), blocks = (tiles * 16 + 255) / 256;
    e = cudaMemsetAsync(counts, 0, (kCountCopies * count_stride(M) + M + 1) * sizeof(uint32_t), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(levelCount, 0, kNeuralMaxDecoded * sizeof(uint32_t), st);
    if (e == cudaSuccess) {
        LaunchScope ls("k_resolve_emit", st);
        k_resolve<kResolveEmit><<<blocks, 256, 0, st>>>(a, nr);
        e = cudaGetLastError();
        if (e == cudaSuccess) fb->layers_stale = kStaleNone;
    }
    if (e == cudaSuccess) {
        LaunchScope ls("k_neural_offsets", st);
        launch_neural_offsets(counts, reqOffset, tileOffset, M, st);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        LaunchScope ls("k_neural_scatter", st);
        launch_neural_scatter(n->surf + slots / 4, (uint32_t)(slots / 4), reqOffset, cursor, n->sorted, levelCount, M, st);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        NeuralDecodeArgs d = {};
        d.n = n->d;
        d.sorted = n->sorted, d.reqOffset = reqOffset, d.tileOffset = tileOffset;
        d.out = n->decoded;
        d.status = n->status;
        LaunchScope ls("k_neural_decode", st);
        launch_neural_decode(d, neural_decode_blocks_per_sm() * neural_num_sms(), st);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        LaunchScope ls("k_resolve_neural", st);
        k_resolve<kResolveNeural><<<blocks, 256, 0, st>>>(a, nr);
        e = cudaGetLastError();
    }
    if (a.lights) cudaFreeAsync((void*)a.lights, st);
    if (e != cudaSuccess) return swr_internal_cuda_fail(e, "swr_resolve_neural");
    fb->keys_valid = false;
    if (stats) {
        uint32_t v[2] = {};
        e = cudaMemcpyAsync(&v[0], reqOffset + M, 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&v[1], tileOffset + M, 4, cudaMemcpyDeviceToHost, st);
        uint32_t status = 0;
        if (e == cudaSuccess) e = cudaMemcpyAsync(&status, n->status, 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(stats->level_texels, levelCount, kNeuralMaxDecoded * 4, cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) return swr_internal_cuda_fail(e, "swr_resolve_neural: stats");
        stats->requests = v[0], stats->tiles = v[1];
        if (status) {
            cudaMemsetAsync(n->status, 0, 4, st);
            return swr_internal_fail(SWR_ETIMEOUT, "swr_resolve_neural: a tensor-core wait timed out");
        }
    }
    return SWR_OK;
}

}  // extern "C"
