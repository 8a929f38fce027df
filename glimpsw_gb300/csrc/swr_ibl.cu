// Image-based lighting precompute (Shading.cpp:35-219): the diffuse irradiance map
// (GenerateIrradianceMap / PrefilterDiffuseIrradiance), the GGX-prefiltered radiance map with one
// roughness per mip level (GenerateRadianceMap / PrefilterEnvMap, Karis 2014) and the split-sum
// environment BRDF table (GenerateEnvBRDFLut / IntegrateBRDF). The reference computes them on the
// CPU and its frame driver never calls them. Each texel is a serial sum of many samples, and there are too few
// texels to give each a thread: a block takes a few texels, its compute warps work out sample terms
// (a lane is one texel and one of several consecutive samples) into shared memory and one warp adds them in
// sample order (ordered_sum).
//
// Exactness: every texel is an independent sum in the reference's order (its 16-lane tile
// decisions, `any(NoL > 0)` and SampleOctLevel's `any(mipFrac > 0)`, give the same value as a
// per-lane decision, because the lanes they add are exact zeros), with the reference's float
// operations in source order. The scalar terms the reference computes once per sample step
// (cosf / sinf of the irradiance integral's angles, the Hammersley points and simd::sincos of their
// azimuths) are computed once on the host in the same operations and travel in the kernels' parameters.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <algorithm>
#include <cstring>

#include "swr_internal.h"
#include "swr_sample.cuh"
#include "swr_surface.cuh"

namespace swr {
namespace {

constexpr float kPi = 3.141592653589793f, kTau = 6.283185307179586f, kInvPi = 0.3183098861837907f;

// The per-sample scalars of the three integrals.
constexpr uint32_t kMaxPhi = 368, kMaxTheta = 96;  // the reference's float loops take 360 and 90 steps, or one more
struct IrradianceTables {
    float cosPhi[kMaxPhi], sinPhi[kMaxPhi];          // cosf(phi), sinf(phi) of each phi step
    float cosTheta[kMaxTheta], sinTheta[kMaxTheta];  // cosf(theta), sinf(theta) of each theta step
    uint32_t numPhi, numTheta;
    float scale;                                     // simd::pi * 1.0f / sampleCount
    float one;                                       // 1 (round_sum)
};
template <uint32_t N>
struct HammersleyTable {
    float t[3 * N];  // Hammersley(i, N): Xi.y, cos(phi), sin(phi) with phi = 2 pi Xi.x
    float one;       // 1 (round_sum)
};

__device__ __forceinline__ float unpack_f11_(uint32_t x) { x <<= 17; return __uint_as_float((x & 0x0FFE0000u) + 0x38000000u); }
__device__ __forceinline__ float unpack_f10_(uint32_t x) { x <<= 18; return __uint_as_float((x & 0x0FFC0000u) + 0x38000000u); }
__device__ __forceinline__ F3 unpack_r11g11b10(uint32_t p) { return { unpack_f11_(p >> 21), unpack_f11_(p >> 10), unpack_f10_(p) }; }
// R11G11B10f::Pack (Texture.h:146-167): clamping only.
__device__ __forceinline__ uint32_t pack_r11g11b10(F3 c) {
    auto f11 = [](float x) {
        x = vmax(x, 1.0f / (1 << 15));
        x = vmin(x, 130048.0f);
        return ((__float_as_uint(x) >> 17) & 0x3FFF) - 0x1C00;
    };
    auto f10 = [](float x) {
        x = vmax(x, 1.0f / (1 << 15));
        x = vmin(x, 129024.0f);
        return ((__float_as_uint(x) >> 18) & 0x1FFF) - 0x0E00;
    };
    return f11(c.x) << 21 | f11(c.y) << 10 | f10(c.z);
}

// Two values at a time (__ffma2_rn, __fmul2_rn): the same IEEE operations on each.
// a + p for a product p, each rounded. A packed product that feeds a packed addition comes out as one fma, whatever
// -fmad says (measured: __fadd2_rn(a, __fmul2_rn(b, c)) equals fma(b, c, a) on 1.6 million random operands, and
// add.rn.f32x2 of mul.rn.f32x2 does, too): the sum is a fma with a one that only the launch knows.
__device__ __forceinline__ float2 round_sum(float2 a, float2 p, float one) { return __ffma2_rn(p, make_float2(one, one), a); }
// a + (b - a) f, rounded after each operation (b - a as the exact product's fma).
__device__ __forceinline__ float2 lerp2(float2 a, float2 b, float f, float one) {
    const float2 d = __ffma2_rn(a, make_float2(-1.0f, -1.0f), b);
    return round_sum(a, __fmul2_rn(d, make_float2(f, f)), one);
}

// One level of an environment map as the sampler reads it.
struct EnvLevel {
    const uint32_t* base;
    int32_t m, stride, width, height;  // the level's size
};
__device__ __forceinline__ EnvLevel env_level(const DevTexture& t, int32_t mipIn) {
    EnvLevel e;
    e.m = min(max(mipIn, 0), (int32_t)t.mip_levels - 1);
    e.stride = (int32_t)t.row_shift - e.m;
    e.base = t.data + t.mip_offsets[e.m & 15];
    e.width = (int32_t)t.width >> e.m, e.height = (int32_t)t.height >> e.m;  // powers of two
    return e;
}

// SampleLevel<EnvSampler> (Texture.h:412-459: ClampToEdge, linear in both directions) of an
// R11G11B10 texture at (u, v) on one level, with SampleLinear's float path (Texture.h:506-575).
__device__ __forceinline__ F3 sample_env_level(const DevTexture& t, const EnvLevel& e, float u, float v, float one) {
    // round2i without its range checks: a NaN gives 0 here instead of INT_MIN and clamps to the same 0, and u and
    // v lie in [0, 1] otherwise
    const int32_t ix = min(max(__float2int_rn(u * t.scale_lerp_u), 0), t.mask_lerp_u) >> e.m;
    const int32_t iy = min(max(__float2int_rn(v * t.scale_lerp_v), 0), t.mask_lerp_v) >> e.m;
    const int32_t xf = max(ix - 127, 0), yf = max(iy - 127, 0);
    const int32_t tx = xf >> 8, ty = yf >> 8;
    const bool inX = tx + 1 < e.width, inY = ty + 1 < e.height;
    const uint32_t i00 = texel_offset(tx, ty, e.stride), i01 = texel_offset(tx, ty + (inY ? 1 : 0), e.stride);
    const F3 c00 = unpack_r11g11b10(e.base[i00]), c10 = unpack_r11g11b10(e.base[i00 + 8]);
    const F3 c01 = unpack_r11g11b10(e.base[i01]), c11 = unpack_r11g11b10(e.base[i01 + 8]);
    const float fs = 1.0f / 256;
    const float fx = inX ? (float)(xf & 255) * fs : 0.0f, fy = (float)(yf & 255) * fs;
    const float2 ra = lerp2(make_float2(c00.x, c00.y), make_float2(c10.x, c10.y), fx, one);
    const float2 rb = lerp2(make_float2(c01.x, c01.y), make_float2(c11.x, c11.y), fx, one);
    const float2 rz = lerp2(make_float2(c00.z, c01.z), make_float2(c10.z, c11.z), fx, one);
    const float2 r = lerp2(ra, rb, fy, one);
    return { r.x, r.y, rz.x + (rz.y - rz.x) * fy };
}

// A level unpacked for the irradiance integral: rows of width + 1 texels, the last one repeated, so that a sample's
// right neighbour is always the next texel. A texel holds its x and y and those of the row below (the last row's:
// its own) as the top halves of floats, which channels of at most 6 mantissa bits fit, and both z: a sample's
// operands are two loads. (Whole floats in four loads took the caches' bandwidth: 1.12 ms.)
__global__ void k_unpack_env(const __grid_constant__ DevTexture env, uint4* __restrict__ texels) {
    const EnvLevel e = env_level(env, 2);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, pitch = (uint32_t)e.width + 1;
    if (i >= pitch * (uint32_t)e.height) return;
    const int32_t x = min((int32_t)(i % pitch), e.width - 1), y = (int32_t)(i / pitch);
    const F3 c = unpack_r11g11b10(e.base[texel_offset(x, y, e.stride)]);
    const F3 d = unpack_r11g11b10(e.base[texel_offset(x, min(y + 1, e.height - 1), e.stride)]);
    texels[i] = make_uint4((__float_as_uint(c.x) >> 16) | __float_as_uint(c.y), (__float_as_uint(d.x) >> 16) | __float_as_uint(d.y),
                           __float_as_uint(c.z), __float_as_uint(d.z));
}
__device__ __forceinline__ float2 unpacked_xy(uint32_t p) { return make_float2(__uint_as_float(p << 16), __uint_as_float(p & 0xFFFF0000u)); }
__device__ __forceinline__ float2 unpacked_z(uint4 p) { return make_float2(__uint_as_float(p.z), __uint_as_float(p.w)); }
// A coordinate's texel and fraction: the float path's round2i by adding 2^23 (the product is below 2^22 and not
// below -1/2, level sizes are at most 8192 << m), whose bits then take the clamp and the shift.
__device__ __forceinline__ int32_t env_coordinate(float s, int32_t mask, int32_t m, float& frac) {
    constexpr int32_t kTwo23 = 0x4B000000;
    const int32_t i = min(__float_as_int(s + 8388608.0f), kTwo23 + mask) >> m;
    const int32_t f = max(i - ((kTwo23 >> m) + 127), 0);
    frac = __int_as_float(0x3F800000 | ((f << 15) & 0x7F8000)) - 1.0f;  // (f & 255) / 256
    return f >> 8;
}
// sample_env_level from them.
__device__ __forceinline__ void sample_env_unpacked(const DevTexture& t, const EnvLevel& e, const uint4* __restrict__ texels, float u, float v,
                                                    float one, float2& xy, float& z) {
    float fx, fy;
    const int32_t tx = env_coordinate(u * t.scale_lerp_u, t.mask_lerp_u, e.m, fx);
    const int32_t ty = env_coordinate(v * t.scale_lerp_v, t.mask_lerp_v, e.m, fy);
    const uint4* p = texels + (uint32_t)(ty * (e.width + 1) + tx);
    const uint4 l = p[0], r = p[1];
    xy = lerp2(lerp2(unpacked_xy(l.x), unpacked_xy(r.x), fx, one), lerp2(unpacked_xy(l.y), unpacked_xy(r.y), fx, one), fy, one);
    const float2 rz = lerp2(unpacked_z(l), unpacked_z(r), fx, one);
    z = rz.x + (rz.y - rz.x) * fy;
}

// swr_rcp14 of a positive number with a normal reciprocal, its segments in shared memory.
__device__ __forceinline__ float rcp14_normal(float x, const uint2* segments) {
    const uint32_t u = __float_as_uint(x);
    const uint2 ab = *(const uint2*)((const char*)segments + ((u >> 14) & 0x1F8));
    const uint32_t sig = ((ab.x - ab.y * ((u >> 7) & 1023)) >> 9) << 7;  // bit 23 set
    return __uint_as_float((252u * 0x800000u - (u & 0x7F800000u)) + ((u & 0x7FFFFFu) ? sig : 0x1000000u));
}
// map_oct of a direction within a percent of unit length (the sum of its absolute coordinates is normal). Halving
// is exact, so its fma is the product and the sum.
__device__ __forceinline__ void map_oct_unit(F3 n, float& u, float& v, const uint2* segments) {
    const float w = rcp14_normal(fabsf(n.x) + fabsf(n.y) + fabsf(n.z), segments);
    const float t = fmaxf(-n.z * w, 0.0f);
    u = fmaf(fmaf(n.x, w, mulsign(t, n.x)), 0.5f, 0.5f);
    v = fmaf(fmaf(n.y, w, mulsign(t, n.y)), 0.5f, 0.5f);
}

// SampleOctLevel<EnvSampler> (Texture.h:467-480): between mips trunc(level) and trunc(level) + 1.
__device__ __forceinline__ F3 sample_oct_level(const DevTexture& t, F3 dir, float level, float one) {
    float u, v;
    map_oct(dir, u, v);
    const int32_t baseMip = trunc2i(level);
    const F3 b = sample_env_level(t, env_level(t, baseMip), u, v, one);
    const float frac = level - (float)baseMip;
    if (frac > 0.0f && baseMip < (int32_t)t.mip_levels - 1) {
        const F3 l = sample_env_level(t, env_level(t, baseMip + 1), u, v, one);
        return { b.x + (l.x - b.x) * frac, b.y + (l.y - b.y) * frac, b.z + (l.z - b.z) * frac };
    }
    return b;
}

// TonemapSample / TonemapSampleInv (Shading.cpp:36-44).
__device__ __forceinline__ F3 tonemap_sample(F3 c, float sign) {
    const float luma = dot3(c, { 0.299f, 0.587f, 0.114f });
    const float r = approx_rcp(sign > 0 ? 1.0f + luma : 1.0f - luma);
    return { c.x * r, c.y * r, c.z * r };
}

// The tangent frame of ImportanceSampleGGX / PrefilterDiffuseIrradiance around N (Shading.cpp:64-67, 74-77).
__device__ __forceinline__ void tangent_frame(F3 N, F3& tx, F3& ty) {
    const bool nz = fabsf(N.z) < 0.999f;
    const F3 up = { nz ? 0.0f : 1.0f, 0.0f, nz ? 1.0f : 0.0f };
    tx = normalize3(cross3(up, N));
    ty = cross3(N, tx);
}

// ImportanceSampleGGX (Shading.cpp:56-70) with the sample's Xi.y and simd::cos / sin of its azimuth: the half vector
// around +z, and in the frame of N.
__device__ __forceinline__ F3 ggx_half_vector(const float* q, float roughness) {
    const float a = roughness * roughness;
    const float cosTheta = __fsqrt_rn((1.0f - q[0]) / (1.0f + (a * a - 1.0f) * q[0]));
    const float sinTheta = __fsqrt_rn(1.0f - cosTheta * cosTheta);
    return { q[1] * sinTheta, q[2] * sinTheta, cosTheta };
}
__device__ __forceinline__ F3 in_frame(F3 H, F3 N, F3 tx, F3 ty) {
    return { tx.x * H.x + ty.x * H.y + N.x * H.z, tx.y * H.x + ty.y * H.y + N.y * H.z, tx.z * H.x + ty.z * H.y + N.z * H.z };
}

// D_GGX (Shading.cpp:19-23).
__device__ __forceinline__ float d_ggx(float NoH, float roughness) {
    const float a = NoH * roughness;
    const float k = roughness * approx_rcp(1.0f - NoH * NoH + a * a);
    return k * k * kInvPi;
}

// simd::approx_log2 (SIMD.h:416-419).
__device__ __forceinline__ float approx_log2(float x) {
    return fmaf(__uint2float_rn(__float_as_uint(x)), 1.1920928955078125e-7f, -126.94269504f);
}

// Sums the terms of chunk after chunk of samples for the block's T texels, C channels each, in sample order.
// A block has one adding warp (warp 0) and W compute warps; a compute lane is texel lane % T and sample
// lane / T of the 32 / T samples its warp takes at a time. chunk(c) prepares chunk c for the lane and returns
// its number of samples (at most K, 0 past the last); term(k, t) gives sample k's terms. While the compute
// warps fill one of the two buffers the adding warp, a lane per texel and channel (per texel where those are
// more than 32), adds the other: its dependent adds take a fraction of the time a chunk's terms do. sum
// receives the adding lane's sums: channel lane / T of texel lane % T, or all channels of texel lane.
template <int T, int C>
constexpr int lane_sums() { return T * C <= 32 ? 1 : C; }
// A lane with one sum reads four samples at a time: the buffer then holds a row of samples (padded to the
// banks) per channel and texel; else a sample's channels and texels are together.
template <int T, int C, int K>
struct SumBuffer {
    static constexpr bool kRows = lane_sums<T, C>() == 1;
    static constexpr int kPitch = kRows ? (K + 31) / 32 * 32 + 8 : 0;
    static constexpr int kSize = 2 * (kRows ? T * C * kPitch : K * C * T);
    static_assert(!kRows || T == 4, "8 words of a row step over the banks of 4 rows");
};
template <int W, int T, int C, int K, class ChunkFn, class TermFn>
__device__ __forceinline__ void ordered_sum(float* buf, float (&sum)[lane_sums<T, C>()], ChunkFn chunk, TermFn term) {
    constexpr uint32_t kStep = 32 / T;
    constexpr int kSums = lane_sums<T, C>();
    using B = SumBuffer<T, C, K>;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, texel = lane % T;
#pragma unroll
    for (int j = 0; j < kSums; j++) sum[j] = 0.0f;
    uint32_t before = 0;
    for (uint32_t c = 0;; c++) {
        const uint32_t n = chunk(c);
        float* b = buf + (c & 1) * (B::kSize / 2) + (B::kRows ? texel * B::kPitch : texel);
        if (warp > 0) {
            for (uint32_t k = (warp - 1) * kStep + lane / T; k < n; k += W * kStep) {
                float t[C];
                term(k, t);
#pragma unroll
                for (int j = 0; j < C; j++) b[B::kRows ? j * T * B::kPitch + k : (k * C + j) * T] = t[j];
            }
        } else if (before && lane < (kSums == 1 ? T * C : T)) {  // the chunk of the last barrier
            const float* q = buf + ((c + 1) & 1) * (B::kSize / 2) + (B::kRows ? lane * B::kPitch : texel);
            if constexpr (B::kRows) {
                uint32_t k = 0;
#pragma unroll 4
                for (; k + 4 <= before; k += 4) {
                    const float4 v = *(const float4*)(q + k);
                    sum[0] = sum[0] + v.x;
                    sum[0] = sum[0] + v.y;
                    sum[0] = sum[0] + v.z;
                    sum[0] = sum[0] + v.w;
                }
                for (; k < before; k++) sum[0] = sum[0] + q[k];
            } else {
#pragma unroll 8
                for (uint32_t k = 0; k < before; k++)
#pragma unroll
                    for (int j = 0; j < kSums; j++) sum[j] = sum[j] + q[(k * C + j) * T];
            }
        }
        if (n == 0) break;
        before = n;
        __syncthreads();
    }
}

// Lookups of the block's sums by the lane that writes texel t.
template <int T, int C>
__device__ __forceinline__ void gather_sums(float acc, uint32_t t, float (&sum)[C]) {
#pragma unroll
    for (int c = 0; c < C; c++) sum[c] = __shfl_sync(0xFFFFFFFFu, acc, (t % T) + c * T);
}

// 4 texels a block: 1024 blocks for a 64x64 map, about 7 per SM (blocks of 32 texels were 128, fewer than the
// SMs, each with a barrier every two samples of a warp): 1.47 -> 1.01 ms for 133 M samples. Bound by instruction
// issue (67 % of the slots, about 160 operations a sample) and by the texel loads' lines (75 % of the load
// unit): the texels with both rows in 16 bytes, the phi steps' rows made by one warp, four sums a read
// and reciprocals without their special cases, 1.01 -> 0.84 ms. 6 compute warps 0.94 ms, 10 0.84; a warp over two phi steps at once
// 0.85; 8 texels a block was slower (1.07 against 1.01); with the level read as it is packed (a larger map) 0.94.
constexpr int kIrrWarps = 8, kIrrTexels = 4;
constexpr int kIrrRows = 2;  // phi steps a chunk
// The other two have texels enough for 32 a block, a lane each: a warp's lanes then share the sample, and its
// Hammersley point is one read of the parameters.
constexpr int kRadWarps = 4, kRadChunk = 16;
constexpr int kBrdfWarps = 7, kBrdfChunk = 28;

// GenerateIrradianceMap (Shading.cpp:177-186) with PrefilterDiffuseIrradiance (72-102): level 0 of
// out. A chunk is a phi step, its samples the theta steps; the term s * cos(theta) * sin(theta) is added to the
// texel's sum in that order, as the reference's nested loops do.
// kUnpacked: the level's texels come unpacked (k_unpack_env).
template <bool kUnpacked>
__global__ void __launch_bounds__((kIrrWarps + 1) * 32) k_ibl_irradiance(const __grid_constant__ DevTexture env, const uint4* __restrict__ texels, const __grid_constant__ DevTexture out,
                                                                          uint32_t* outData, const __grid_constant__ IrradianceTables tb) {
    __shared__ __align__(16) float buf[SumBuffer<kIrrTexels, 3, kIrrRows * (int)kMaxTheta>::kSize];
    __shared__ uint2 segments[64];
    __shared__ float4 rows[2][kIrrRows][kIrrTexels];  // cos(phi) right + sin(phi) up of a chunk's phi steps
    __shared__ float2 theta[kMaxTheta], phi[kMaxPhi];  // cos, sin
    for (uint32_t i = threadIdx.x; i < tb.numTheta; i += blockDim.x) theta[i] = make_float2(tb.cosTheta[i], tb.sinTheta[i]);
    for (uint32_t i = threadIdx.x; i < tb.numPhi; i += blockDim.x) phi[i] = make_float2(tb.cosPhi[i], tb.sinPhi[i]);
    for (uint32_t i = threadIdx.x; i < 64; i += blockDim.x) segments[i] = swr_a14_device_segments[i];
    __syncthreads();
    const uint32_t n = out.width * out.height;
    const uint32_t i = min(blockIdx.x * kIrrTexels + (threadIdx.x & 31) % kIrrTexels, n - 1);  // lanes past the end repeat the last texel
    const uint32_t x = i % out.width, y = i / out.width;
    const float u = ((float)x + 0.5f) * (1.0f / (float)out.width), v = ((float)y + 0.5f) * (1.0f / (float)out.height);
    const F3 N = unmap_oct(u, v);
    F3 right, up;
    tangent_frame(N, right, up);
    const EnvLevel level = env_level(env, 2);  // SampleOctLevel at level 2: no second mip
    const float4(*row)[kIrrTexels] = rows[0];
    float acc[1];
    // the adding warp prepares the next chunk's rows, a lane per row and texel
    auto prepare = [&](uint32_t c) {
        const uint32_t r = threadIdx.x / kIrrTexels, step = c * kIrrRows + r;
        if (r < (uint32_t)kIrrRows && step < tb.numPhi) {
            const float cp = phi[step].x, sp = phi[step].y;
            rows[c & 1][r][threadIdx.x % kIrrTexels] =
                make_float4(cp * right.x + sp * up.x, cp * right.y + sp * up.y, cp * right.z + sp * up.z, 0.0f);
        }
    };
    prepare(0);
    __syncthreads();
    ordered_sum<kIrrWarps, kIrrTexels, 3, kIrrRows * (int)kMaxTheta>(buf, acc,
        [&](uint32_t c) -> uint32_t {
            if (threadIdx.x < 32) prepare(c + 1);
            row = rows[c & 1];
            return c * kIrrRows < tb.numPhi ? min((uint32_t)kIrrRows, tb.numPhi - c * kIrrRows) * tb.numTheta : 0u;
        },
        [&](uint32_t k, float (&t)[3]) {
            const bool second = k >= tb.numTheta;
            const float4 a = row[second ? 1 : 0][threadIdx.x % kIrrTexels];
            const float2 cs = theta[second ? k - tb.numTheta : k];
            const float ct = cs.x, st = cs.y;
            const float2 d = round_sum(__fmul2_rn(make_float2(ct, ct), make_float2(N.x, N.y)),
                                       __fmul2_rn(make_float2(st, st), make_float2(a.x, a.y)), tb.one);
            const F3 dir = { d.x, d.y, ct * N.z + st * a.z };
            float su, sv, z;
            float2 xy;
            map_oct_unit(dir, su, sv, segments);
            if constexpr (kUnpacked) {
                sample_env_unpacked(env, level, texels, su, sv, tb.one, xy, z);
            } else {
                const F3 s = sample_env_level(env, level, su, sv, tb.one);
                xy = make_float2(s.x, s.y), z = s.z;
            }
            // tonemap_sample, then times cos(theta) sin(theta)
            const float r = rcp14_normal(1.0f + dot3({ xy.x, xy.y, z }, { 0.299f, 0.587f, 0.114f }), segments);
            xy = __fmul2_rn(__fmul2_rn(__fmul2_rn(xy, make_float2(r, r)), make_float2(ct, ct)), make_float2(st, st));
            t[0] = xy.x, t[1] = xy.y, t[2] = z * r * ct * st;
        });
    if (threadIdx.x >= 32) return;
    float color[3];
    gather_sums<kIrrTexels, 3>(acc[0], threadIdx.x, color);
    if (threadIdx.x >= kIrrTexels || blockIdx.x * kIrrTexels + threadIdx.x >= n) return;
    const float k = tb.scale;
    const F3 r = tonemap_sample({ color[0] * k, color[1] * k, color[2] * k }, -1.0f);
    outData[out.mip_offsets[0] + texel_offset((int32_t)x, (int32_t)y, (int32_t)out.row_shift)] = pack_r11g11b10(r);
}

// GenerateRadianceMap (Shading.cpp:187-201) with PrefilterEnvMap (105-147, 128 samples): every mip
// level of out, level L prefiltered at roughness L / (MipLevels - 1). A sample with NoL <= 0 adds +0.
// (87k texels of a 256x256 map: one thread a texel left 18 warps on an SM, 209 us; 176 us with the samples spread
// over four warps.)
__global__ void __launch_bounds__((kRadWarps + 1) * 32) k_ibl_radiance(const __grid_constant__ DevTexture env, const __grid_constant__ DevTexture out,
                                                                        uint32_t* outData, const __grid_constant__ HammersleyTable<128> ham,
                                                                        uint32_t totalTexels) {
    constexpr uint32_t numSamples = 128;
    __shared__ float buf[SumBuffer<32, 4, kRadChunk>::kSize];
    const uint32_t i = min(blockIdx.x * 32 + (threadIdx.x & 31), totalTexels - 1);  // lanes past the end repeat the last texel
    uint32_t level = 0, j = i;
    while (j >= (out.width >> level) * (out.height >> level)) j -= (out.width >> level) * (out.height >> level), level++;
    const uint32_t w = out.width >> level, h = out.height >> level;
    const uint32_t x = j % w, y = j / w;
    const float u = ((float)x + 0.5f) * (1.0f / (float)w), v = ((float)y + 0.5f) * (1.0f / (float)h);
    const F3 R = unmap_oct(u, v);
    const float roughness = vmax((float)level / ((float)out.mip_levels - 1.0f), 0.01f);  // std::max
    F3 tx, ty;
    tangent_frame(R, tx, ty);
    const float omegaP = 4.0f * kPi / (float)(6u * env.width * env.width);
    uint32_t first = 0;
    float pre[4];
    ordered_sum<kRadWarps, 32, 4, kRadChunk>(buf, pre,
        [&](uint32_t c) -> uint32_t {
            first = c * kRadChunk;
            return first < numSamples ? (uint32_t)kRadChunk : 0u;
        },
        [&](uint32_t k, float (&t)[4]) {
            const F3 H = in_frame(ggx_half_vector(ham.t + 3 * (first + k), roughness), R, tx, ty);
            const float VoH = dot3(R, H);
            const float NoH = vmax(VoH, 0.0f);
            const F3 L = { 2.0f * VoH * H.x - R.x, 2.0f * VoH * H.y - R.y, 2.0f * VoH * H.z - R.z };
            const float NoL = vmax(dot3(R, L), 0.0f);
            t[0] = 0.0f, t[1] = 0.0f, t[2] = 0.0f, t[3] = 0.0f;
            if (NoL > 0.0f) {
                const float pdf = d_ggx(NoH, roughness) / 4.0f + 0.001f;
                const float omegaS = 1.0f / ((float)numSamples * pdf);
                const float mip = vmax(0.5f * approx_log2(omegaS / omegaP), 0.0f);
                const F3 c = tonemap_sample(sample_oct_level(env, L, mip, ham.one), 1.0f);
                t[0] = c.x * NoL, t[1] = c.y * NoL, t[2] = c.z * NoL, t[3] = NoL;
            }
        });
    if (threadIdx.x >= 32 || blockIdx.x * 32 + threadIdx.x >= totalTexels) return;
    const F3 r = tonemap_sample({ pre[0] / pre[3], pre[1] / pre[3], pre[2] / pre[3] }, -1.0f);
    outData[out.mip_offsets[level & 15] + texel_offset((int32_t)x, (int32_t)y, (int32_t)out.row_shift - (int32_t)level)] =
        pack_r11g11b10(r);
}

// GenerateEnvBRDFLut (Shading.cpp:202-210) with IntegrateBRDF (149-175, 1024 samples): RG16f texel
// (scale, bias) at NoV = u, roughness = v. A sample with NoL <= 0 adds +0, as the reference's lanes
// with Gv = 0 do (Shading.cpp:167).
__global__ void __launch_bounds__((kBrdfWarps + 1) * 32) k_ibl_env_brdf(const __grid_constant__ DevTexture out, uint32_t* outData,
                                                                        const __grid_constant__ HammersleyTable<1024> ham) {
    constexpr uint32_t sampleCount = 1024;
    __shared__ float buf[SumBuffer<32, 2, kBrdfChunk>::kSize];
    __shared__ float4 half[sampleCount];
    const uint32_t n = out.width * out.height;
    const uint32_t i = min(blockIdx.x * 32 + (threadIdx.x & 31), n - 1);
    const uint32_t x = i % out.width, y = i / out.width;
    const float NoV = ((float)x + 0.5f) * (1.0f / (float)out.width), roughness = ((float)y + 0.5f) * (1.0f / (float)out.height);
    const F3 N = { 0.0f, 0.0f, 1.0f };
    const F3 V = { __fsqrt_rn(1.0f - NoV * NoV), 0.0f, NoV };
    F3 tx, ty;
    tangent_frame(N, tx, ty);
    // The block's texels are of one row, hence one roughness and one set of half vectors, in a table 32 or more
    // texels wide: 82 -> 67 us for 128x128 (two square roots and a division a sample less; the radiance map, whose
    // levels share theirs the same way, gains 1 % by it).
    const uint32_t shared = __syncthreads_and(y == __shfl_sync(0xFFFFFFFFu, y, 0));
    if (shared) {
        for (uint32_t k = threadIdx.x; k < sampleCount; k += blockDim.x) {
            const F3 H = in_frame(ggx_half_vector(ham.t + 3 * k, roughness), N, tx, ty);
            half[k] = make_float4(H.x, H.y, H.z, 0.0f);
        }
        __syncthreads();
    }
    uint32_t first = 0;
    float acc[2];
    ordered_sum<kBrdfWarps, 32, 2, kBrdfChunk>(buf, acc,
        [&](uint32_t c) -> uint32_t {
            first = c * kBrdfChunk;
            return first < sampleCount ? min((uint32_t)kBrdfChunk, sampleCount - first) : 0u;
        },
        [&](uint32_t k, float (&t)[2]) {
            const float4 h = half[first + k];
            const F3 H = shared ? F3{ h.x, h.y, h.z } : in_frame(ggx_half_vector(ham.t + 3 * (first + k), roughness), N, tx, ty);
            const float VdH = dot3(V, H);
            const F3 L = { 2.0f * VdH * H.x - V.x, 2.0f * VdH * H.y - V.y, 2.0f * VdH * H.z - V.z };
            const float VoH = vmax(0.0f, VdH), NoL = vmax(0.0f, L.z), NoH = vmax(0.0f, H.z);
            t[0] = 0.0f, t[1] = 0.0f;
            if (NoL > 0.0f) {
                // V_SmithGGXCorrelatedFast (Shading.cpp:24-28) with roughness^2
                const float r2 = roughness * roughness;
                const float a = 2.0f * NoL * NoV, b = NoL + NoV;
                const float G = 0.5f / fmaf(r2, b, fmaf(-r2, a, a));
                const float Gv = G * 4.0f * VoH * NoL / NoH;
                const float om = 1.0f - VoH;
                const float Fc = (om * om) * (om * om) * om;  // pow5
                t[0] = Gv * (1.0f - Fc), t[1] = Gv * Fc;
            }
        });
    if (threadIdx.x >= 32 || blockIdx.x * 32 + threadIdx.x >= n) return;
    const uint32_t hx = __half_as_ushort(__float2half_rn(acc[0] * (1.0f / sampleCount)));
    const uint32_t hy = __half_as_ushort(__float2half_rn(acc[1] * (1.0f / sampleCount)));
    outData[out.mip_offsets[0] + texel_offset((int32_t)x, (int32_t)y, (int32_t)out.row_shift)] = hx | (hy << 16);
}

// ---------------------------------------------------------------------------- host tables
// simd::sincos_2pi (SIMD.h:390-409): sin and cos of 2 pi x by the reference's polynomials.
void sincos_2pi(float x, float& s, float& c) {
    x = x + 0.25f;
    x = x - std::nearbyint(x);
    const float x1 = std::fabs(x) - 0.25f;
    const float x2 = x1 * x1;
    s = std::fma(x2, std::fma(x2, std::fma(x2, -70.993433272f, 81.340768887f), -41.337142371f), 6.283164044f) * x1;
    c = std::fma(x2, std::fma(x2, std::fma(x2, -78.216131988f, 64.660541218f), -19.735752060f), 0.999993295f);
    uint32_t cb, xb;
    memcpy(&cb, &c, 4);
    memcpy(&xb, &x, 4);
    cb ^= xb & 0x80000000u;  // mulsign(r_cos, x)
    memcpy(&c, &cb, 4);
}

// Hammersley(i, n) (Shading.cpp:46-54), with simd::cos / sin (SIMD.h:411-413) of phi = 2 pi Xi.x
// (ImportanceSampleGGX, Shading.cpp:59): Xi.y, cos(phi), sin(phi) per sample.
template <uint32_t n>
HammersleyTable<n> hammersley_table() {
    HammersleyTable<n> h;
    h.one = 1.0f;
    for (uint32_t i = 0; i < n; i++) {
        uint32_t bits = i;
        bits = (bits << 16) | (bits >> 16);
        bits = ((bits & 0x55555555u) << 1) | ((bits & 0xAAAAAAAAu) >> 1);
        bits = ((bits & 0x33333333u) << 2) | ((bits & 0xCCCCCCCCu) >> 2);
        bits = ((bits & 0x0F0F0F0Fu) << 4) | ((bits & 0xF0F0F0F0u) >> 4);
        bits = ((bits & 0x00FF00FFu) << 8) | ((bits & 0xFF00FF00u) >> 8);
        const float xiX = (float)i / (float)n;
        const float xiY = (float)(bits * (1.0 / 4294967295.0));
        const float phi = (float)(2.0 * (double)kPi * (double)xiX);
        float s, c;
        sincos_2pi(phi * 0.15915494309189535f, s, c);
        h.t[3 * i] = xiY, h.t[3 * i + 1] = c, h.t[3 * i + 2] = s;
    }
    return h;
}

// The phi / theta steps of PrefilterDiffuseIrradiance (release build: 360 x 90) with their cosf / sinf.
IrradianceTables irradiance_tables() {
    IrradianceTables t = {};
    const float halfPi = (float)((double)kPi * 0.5);
    const float deltaPhi = (float)((double)kTau / 360.0), deltaTheta = (float)((double)halfPi / 90.0);
    for (float phi = 0.0f; phi < kTau && t.numPhi < kMaxPhi; phi += deltaPhi, t.numPhi++)
        t.cosPhi[t.numPhi] = cosf(phi), t.sinPhi[t.numPhi] = sinf(phi);
    for (float theta = 0.0f; theta < halfPi && t.numTheta < kMaxTheta; theta += deltaTheta, t.numTheta++)
        t.cosTheta[t.numTheta] = cosf(theta), t.sinTheta[t.numTheta] = sinf(theta);
    t.scale = kPi * 1.0f / (float)(t.numPhi * t.numTheta);
    t.one = 1.0f;
    return t;
}

swr_status check_env(swr_texture env, const char* what) {
    if (!env) return swr_internal_fail(SWR_EINVAL, what);
    if (env->format != SWR_FORMAT_R11G11B10F || env->d.num_layers < 1)
        return swr_internal_fail(SWR_EINVAL, "swr_ibl: the environment map must be an R11G11B10 octahedral texture");
    return SWR_OK;
}

}  // namespace
}  // namespace swr

using namespace swr;

extern "C" {

swr_status swr_ibl_irradiance_map(swr_texture env, swr_texture out) {
    swr_status s = check_env(env, "swr_ibl_irradiance_map: NULL environment map");
    if (s != SWR_OK) return s;
    if (!out || out->format != SWR_FORMAT_R11G11B10F)
        return swr_internal_fail(SWR_EINVAL, "swr_ibl_irradiance_map: the output must be an R11G11B10 texture");
    static const IrradianceTables tb = irradiance_tables();
    cudaStream_t st = swr_internal_stream();
    const uint32_t n = out->d.width * out->d.height, blocks = (n + kIrrTexels - 1) / kIrrTexels;
    // Every sample reads one level. Up to kSkyScratchTexels texels (4 MB unpacked, which the caches hold) level 2 is
    // unpacked first; a larger one, and the last level of a map without a level 2, is read as it is. Calls on several
    // streams may unpack one map at once: each writes the same words, made of texels that no caller may change
    // before all of them have read them.
    if (env->skyScratch) {
        uint4* texels = (uint4*)env->skyScratch;
        const uint32_t count = ((env->d.width >> 2) + 1) * (env->d.height >> 2);
        {
            LaunchScope ls("k_unpack_env", st);
            k_unpack_env<<<(count + 255) / 256, 256, 0, st>>>(env->d, texels);
        }
        LaunchScope ls("k_ibl_irradiance", st);
        k_ibl_irradiance<true><<<blocks, (kIrrWarps + 1) * 32, 0, st>>>(env->d, texels, out->d, (uint32_t*)out->d.data, tb);
    } else {
        LaunchScope ls("k_ibl_irradiance", st);
        k_ibl_irradiance<false><<<blocks, (kIrrWarps + 1) * 32, 0, st>>>(env->d, nullptr, out->d, (uint32_t*)out->d.data, tb);
    }
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? SWR_OK : swr_internal_cuda_fail(e, "swr_ibl_irradiance_map");
}

swr_status swr_ibl_radiance_map(swr_texture env, swr_texture out) {
    swr_status s = check_env(env, "swr_ibl_radiance_map: NULL environment map");
    if (s != SWR_OK) return s;
    if (!out || out->format != SWR_FORMAT_R11G11B10F || out->d.mip_levels < 2)
        return swr_internal_fail(SWR_EINVAL, "swr_ibl_radiance_map: the output must be an R11G11B10 texture with mips");
    static const HammersleyTable<128> ham = hammersley_table<128>();
    cudaStream_t st = swr_internal_stream();
    uint32_t total = 0;
    for (uint32_t l = 0; l < out->d.mip_levels; l++) total += (out->d.width >> l) * (out->d.height >> l);
    {
        LaunchScope ls("k_ibl_radiance", st);
        k_ibl_radiance<<<(total + 31) / 32, (kRadWarps + 1) * 32, 0, st>>>(env->d, out->d, (uint32_t*)out->d.data,
                                                                                              ham, total);
    }
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? SWR_OK : swr_internal_cuda_fail(e, "swr_ibl_radiance_map");
}

swr_status swr_ibl_env_brdf_lut(swr_texture out) {
    if (!out || out->format != SWR_FORMAT_RG16F)
        return swr_internal_fail(SWR_EINVAL, "swr_ibl_env_brdf_lut: the output must be an RG16f texture");
    static const HammersleyTable<1024> ham = hammersley_table<1024>();
    cudaStream_t st = swr_internal_stream();
    const uint32_t n = out->d.width * out->d.height;
    {
        LaunchScope ls("k_ibl_env_brdf", st);
        k_ibl_env_brdf<<<(n + 31) / 32, (kBrdfWarps + 1) * 32, 0, st>>>(out->d, (uint32_t*)out->d.data, ham);
    }
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? SWR_OK : swr_internal_cuda_fail(e, "swr_ibl_env_brdf_lut");
}

}  // extern "C"
