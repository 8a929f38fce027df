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
};
template <uint32_t N>
struct HammersleyTable {
    float t[3 * N];  // Hammersley(i, N): Xi.y, cos(phi), sin(phi) with phi = 2 pi Xi.x
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

// Two values at a time with the packed FP32 instructions (sm_100): the same IEEE operations on each.
// a + (b - a) f, rounded after each operation (b - a as the exact product's fma).
__device__ __forceinline__ float2 lerp2(float2 a, float2 b, float f) {
    const float2 d = __ffma2_rn(a, make_float2(-1.0f, -1.0f), b);
    return __fadd2_rn(a, __fmul2_rn(d, make_float2(f, f)));
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
__device__ __forceinline__ F3 sample_env_level(const DevTexture& t, const EnvLevel& e, float u, float v) {
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
    const float2 ra = lerp2(make_float2(c00.x, c00.y), make_float2(c10.x, c10.y), fx);
    const float2 rb = lerp2(make_float2(c01.x, c01.y), make_float2(c11.x, c11.y), fx);
    const float2 rz = lerp2(make_float2(c00.z, c01.z), make_float2(c10.z, c11.z), fx);
    const float2 r = lerp2(ra, rb, fy);
    return { r.x, r.y, rz.x + (rz.y - rz.x) * fy };
}

// A texel's channels have at most 6 mantissa bits, so the top half of each float holds it: x and y in one word,
// z as a float, row by row.
__global__ void k_unpack_env(const __grid_constant__ DevTexture env, uint2* __restrict__ texels) {
    const EnvLevel e = env_level(env, 2);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (uint32_t)(e.width * e.height)) return;
    const F3 c = unpack_r11g11b10(e.base[texel_offset((int32_t)(i % e.width), (int32_t)(i / e.width), e.stride)]);
    texels[i] = make_uint2((__float_as_uint(c.x) >> 16) | __float_as_uint(c.y), __float_as_uint(c.z));
}
__device__ __forceinline__ float2 unpacked_xy(uint2 p) { return make_float2(__uint_as_float(p.x << 16), __uint_as_float(p.x & 0xFFFF0000u)); }
// sample_env_level from them: 8 operations unpack the four texels instead of 36, and the sample is bound by
// integer and logic operations (half rate).
__device__ __forceinline__ F3 sample_env_unpacked(const DevTexture& t, const EnvLevel& e, const uint2* __restrict__ texels, float u, float v) {
    const int32_t ix = min(max(__float2int_rn(u * t.scale_lerp_u), 0), t.mask_lerp_u) >> e.m;
    const int32_t iy = min(max(__float2int_rn(v * t.scale_lerp_v), 0), t.mask_lerp_v) >> e.m;
    const int32_t xf = max(ix - 127, 0), yf = max(iy - 127, 0);
    const int32_t tx = xf >> 8, ty = yf >> 8;
    const bool inX = tx + 1 < e.width, inY = ty + 1 < e.height;
    const uint2* p = texels + ty * e.width + tx;
    const uint2* q = p + (inY ? e.width : 0);
    const int32_t right = inX ? 1 : 0;
    const uint2 c00 = p[0], c10 = p[right], c01 = q[0], c11 = q[right];
    const float fs = 1.0f / 256;
    const float fx = inX ? (float)(xf & 255) * fs : 0.0f, fy = (float)(yf & 255) * fs;
    const float2 ra = lerp2(unpacked_xy(c00), unpacked_xy(c10), fx), rb = lerp2(unpacked_xy(c01), unpacked_xy(c11), fx);
    const float2 rz = lerp2(make_float2(__uint_as_float(c00.y), __uint_as_float(c01.y)),
                            make_float2(__uint_as_float(c10.y), __uint_as_float(c11.y)), fx);
    const float2 r = lerp2(ra, rb, fy);
    return { r.x, r.y, rz.x + (rz.y - rz.x) * fy };
}

// SampleOctLevel<EnvSampler> (Texture.h:467-480): between mips trunc(level) and trunc(level) + 1.
__device__ __forceinline__ F3 sample_oct_level(const DevTexture& t, F3 dir, float level) {
    float u, v;
    map_oct(dir, u, v);
    const int32_t baseMip = trunc2i(level);
    const F3 b = sample_env_level(t, env_level(t, baseMip), u, v);
    const float frac = level - (float)baseMip;
    if (frac > 0.0f && baseMip < (int32_t)t.mip_levels - 1) {
        const F3 l = sample_env_level(t, env_level(t, baseMip + 1), u, v);
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

// ImportanceSampleGGX (Shading.cpp:56-70) with the sample's Xi.y and simd::cos / sin of its azimuth.
__device__ __forceinline__ F3 importance_sample_ggx(float xiY, float cphi, float sphi, float roughness, F3 N, F3 tx, F3 ty) {
    const float a = roughness * roughness;
    const float cosTheta = __fsqrt_rn((1.0f - xiY) / (1.0f + (a * a - 1.0f) * xiY));
    const float sinTheta = __fsqrt_rn(1.0f - cosTheta * cosTheta);
    const F3 H = { cphi * sinTheta, sphi * sinTheta, cosTheta };
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
template <int W, int T, int C, int K, class ChunkFn, class TermFn>
__device__ __forceinline__ void ordered_sum(float* buf, float (&sum)[lane_sums<T, C>()], ChunkFn chunk, TermFn term) {
    constexpr uint32_t kStep = 32 / T;
    constexpr int kSums = lane_sums<T, C>();
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, texel = lane % T;
#pragma unroll
    for (int j = 0; j < kSums; j++) sum[j] = 0.0f;
    uint32_t before = 0;
    for (uint32_t c = 0;; c++) {
        const uint32_t n = chunk(c);
        float* b = buf + (c & 1) * (K * C * T) + texel;
        if (warp > 0) {
            for (uint32_t k = (warp - 1) * kStep + lane / T; k < n; k += W * kStep) {
                float t[C];
                term(k, t);
#pragma unroll
                for (int j = 0; j < C; j++) b[(k * C + j) * T] = t[j];
            }
        } else if (before && lane < (kSums == 1 ? T * C : T)) {  // the chunk of the last barrier
            const float* q = buf + ((c + 1) & 1) * (K * C * T) + (kSums == 1 ? lane / T : 0) * T + texel;
#pragma unroll 8
            for (uint32_t k = 0; k < before; k++)
#pragma unroll
                for (int j = 0; j < kSums; j++) sum[j] = sum[j] + q[(k * C + j) * T];
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
// SMs, each with a barrier every two samples of a warp). Bound by instruction issue (about 200 operations a
// sample, 133 M samples): 1.47 -> 1.01 ms. 3 to 6 compute warps 1.34 to 1.12 ms, 12 1.06; 8 texels a block
// 1.07 or more; packed texels (a larger map) 1.09.
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
__global__ void __launch_bounds__((kIrrWarps + 1) * 32) k_ibl_irradiance(const __grid_constant__ DevTexture env, const uint2* __restrict__ texels, const __grid_constant__ DevTexture out,
                                                                          uint32_t* outData, const __grid_constant__ IrradianceTables tb) {
    __shared__ float buf[2 * kIrrRows * kMaxTheta * 3 * kIrrTexels];
    __shared__ float2 theta[kMaxTheta], phi[kMaxPhi];  // cos, sin
    for (uint32_t i = threadIdx.x; i < tb.numTheta; i += blockDim.x) theta[i] = make_float2(tb.cosTheta[i], tb.sinTheta[i]);
    for (uint32_t i = threadIdx.x; i < tb.numPhi; i += blockDim.x) phi[i] = make_float2(tb.cosPhi[i], tb.sinPhi[i]);
    __syncthreads();
    const uint32_t n = out.width * out.height;
    const uint32_t i = min(blockIdx.x * kIrrTexels + (threadIdx.x & 31) % kIrrTexels, n - 1);  // lanes past the end repeat the last texel
    const uint32_t x = i % out.width, y = i / out.width;
    const float u = ((float)x + 0.5f) * (1.0f / (float)out.width), v = ((float)y + 0.5f) * (1.0f / (float)out.height);
    const F3 N = unmap_oct(u, v);
    F3 right, up;
    tangent_frame(N, right, up);
    const EnvLevel level = env_level(env, 2);  // SampleOctLevel at level 2: no second mip
    F3 tmp[kIrrRows] = {};
    float acc[1];
    ordered_sum<kIrrWarps, kIrrTexels, 3, kIrrRows * (int)kMaxTheta>(buf, acc,
        [&](uint32_t c) -> uint32_t {
            uint32_t rows = 0;
#pragma unroll
            for (int r = 0; r < kIrrRows; r++) {
                if (c * kIrrRows + r >= tb.numPhi) break;
                const float cp = phi[c * kIrrRows + r].x, sp = phi[c * kIrrRows + r].y;
                tmp[r] = { cp * right.x + sp * up.x, cp * right.y + sp * up.y, cp * right.z + sp * up.z };
                rows++;
            }
            return rows * tb.numTheta;
        },
        [&](uint32_t k, float (&t)[3]) {
            const bool second = k >= tb.numTheta;
            const F3 a = second ? tmp[1] : tmp[0];
            const float2 cs = theta[second ? k - tb.numTheta : k];
            const float ct = cs.x, st = cs.y;
            const float2 d = __fadd2_rn(__fmul2_rn(make_float2(ct, ct), make_float2(N.x, N.y)),
                                        __fmul2_rn(make_float2(st, st), make_float2(a.x, a.y)));
            const F3 dir = { d.x, d.y, ct * N.z + st * a.z };
            float su, sv;
            map_oct(dir, su, sv);
            const F3 s = tonemap_sample(kUnpacked ? sample_env_unpacked(env, level, texels, su, sv) : sample_env_level(env, level, su, sv), 1.0f);
            t[0] = s.x * ct * st, t[1] = s.y * ct * st, t[2] = s.z * ct * st;
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
    __shared__ float buf[2 * kRadChunk * 4 * 32];
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
            const float* q = ham.t + 3 * (first + k);
            const F3 H = importance_sample_ggx(q[0], q[1], q[2], roughness, R, tx, ty);
            const float VoH = dot3(R, H);
            const float NoH = vmax(VoH, 0.0f);
            const F3 L = { 2.0f * VoH * H.x - R.x, 2.0f * VoH * H.y - R.y, 2.0f * VoH * H.z - R.z };
            const float NoL = vmax(dot3(R, L), 0.0f);
            t[0] = 0.0f, t[1] = 0.0f, t[2] = 0.0f, t[3] = 0.0f;
            if (NoL > 0.0f) {
                const float pdf = d_ggx(NoH, roughness) / 4.0f + 0.001f;
                const float omegaS = 1.0f / ((float)numSamples * pdf);
                const float mip = vmax(0.5f * approx_log2(omegaS / omegaP), 0.0f);
                const F3 c = tonemap_sample(sample_oct_level(env, L, mip), 1.0f);
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
    __shared__ float buf[2 * kBrdfChunk * 2 * 32];
    const uint32_t n = out.width * out.height;
    const uint32_t i = min(blockIdx.x * 32 + (threadIdx.x & 31), n - 1);
    const uint32_t x = i % out.width, y = i / out.width;
    const float NoV = ((float)x + 0.5f) * (1.0f / (float)out.width), roughness = ((float)y + 0.5f) * (1.0f / (float)out.height);
    const F3 N = { 0.0f, 0.0f, 1.0f };
    const F3 V = { __fsqrt_rn(1.0f - NoV * NoV), 0.0f, NoV };
    F3 tx, ty;
    tangent_frame(N, tx, ty);
    uint32_t first = 0;
    float acc[2];
    ordered_sum<kBrdfWarps, 32, 2, kBrdfChunk>(buf, acc,
        [&](uint32_t c) -> uint32_t {
            first = c * kBrdfChunk;
            return first < sampleCount ? min((uint32_t)kBrdfChunk, sampleCount - first) : 0u;
        },
        [&](uint32_t k, float (&t)[2]) {
            const float* q = ham.t + 3 * (first + k);
            const F3 H = importance_sample_ggx(q[0], q[1], q[2], roughness, N, tx, ty);
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
    // Every sample reads one level. Up to kSkyScratchTexels texels (2 MB unpacked, which the caches hold) it is
    // unpacked first; a larger one is read as it is.
    if (env->skyScratch) {
        uint2* texels = (uint2*)env->skyScratch;
        const uint32_t level = std::min(2u, env->d.mip_levels - 1), count = (env->d.width >> level) * (env->d.height >> level);
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
