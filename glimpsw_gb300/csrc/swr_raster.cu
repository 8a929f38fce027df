// Meshlet rasterizer kernels: mesh shader (ShadeMeshlet), clip codes, triangle setup, clipping and
// vis-buffer rasterization (FS_EncodeSurfaceId<false> and, for alpha-tested materials,
// FS_EncodeSurfaceId<true>) for sm_103a.
//
// Work decomposition:
//   k_draw_meshlets  one warp per meshlet (dynamic fetch, a block's warps sharing fetched groups), or several
//                    in small draws. Lanes transform the 64 vertices into shared memory and test the
//                    faces, then own one of the remaining triangles each: setup and edge equations
//                    in registers. Triangles whose 4-aligned box covers at most kSmallTiles 4x4
//                    tiles are rasterized by the whole warp, four tiles (64 pixels) per step, those
//                    of at most two samples by their lane; larger and clipped triangles go to a device
//                    queue. Alpha-tested meshlets are drawn by a pass of their own.
//   k_raster_big     warps take runs of 32x32-pixel chunks of queued triangles (flattened by a prefix of
//                    chunk counts kept in the queue), reject empty and hidden chunks one per lane
//                    and rasterize the rest four tiles per step.
//   k_finalize       converts per-pixel keys to the reference's depth and surfaceId layers, for readers of
//                    the layers that do not take the keys themselves.
// The depth test is a 64-bit atomicMax on (ordered depth, 0xFFFFFFFE - rank); the result is
// independent of execution order and equals the single-threaded reference. The alpha test is a
// function of the triangle and the fragment alone, so it only removes fragments and keeps that
// property.
//
// Tile depth culling: tileMin holds, per 4x4 tile, a lower bound of the depth words of its 16
// keys (keys only grow, and tileMin only takes minima of values its pixels had reached). Before a
// tile is shaded, an upper bound of the triangle's depth over the tile is compared with it; a tile
// the triangle cannot win anywhere is skipped. The vis-buffer is unchanged (only fragments that
// would fail the depth test are skipped), while the dense scenes' overdraw mostly disappears.
//
// Figures of the form a -> b beside a choice are of that choice alone, on the kernels as they were then: later
// choices moved both. The kernels as they are (us, SM at 2070 MHz):
//   1080p frame of 100k meshlets: mesh stage 333, chunk stage 151; 24 views of 100k meshlets in a batch: 1231, 221
//   inside a 50k-meshlet scene, half of the materials alpha-tested, 1916x1036: mesh stage 103, opaque chunks 122,
//   alpha pass 53, its chunks 193; G-buffer draw of 30k, 1600x900: 113, 81, 110, 133
//   overdraw draw of 20k, 1280x720: 160, 148; 150k meshlets culled against the Hi-Z, 2560x1440: 40, 81
//   1024 meshlets at 1280x720: 30, 15; 60 at 252x140: 9.2, 7.5
#include <algorithm>
#include <cfloat>
#include <mutex>
#include <numeric>
#include <type_traits>

#include "../../include/swr/approx14.h"
#include "../../include/swr/raster_math.cuh"
#include "swr_device.cuh"
#include "swr_internal.h"
#include "swr_sample.cuh"

namespace swr {

constexpr int kWarpsPerBlock = 8;
constexpr int kSmallTiles = 16;
static_assert(kSmallTiles <= 16, "the small triangles' tile -> row multiply-shift is exact for at most 16 tiles");
constexpr int kPacketTiles = 128, kPacketTilesAlpha = 64;  // in-warp tile budget of a 32-triangle step
constexpr int kSpreadTiles = 4;    // over budget, triangles above this many tiles are queued
constexpr int kChunkTiles = 8;  // chunk = 8x8 tiles = 32x32 pixels

// A record in a warp's shared memory padded to 80 bytes. TriRec and AlphaExt are 64 bytes; with a
// 64-byte stride the 16-byte loads of one field by lanes holding different triangles (the tile
// tests) fall into two of the eight 16-byte bank groups of a quarter warp, with an 80-byte stride
// into eight. The loads stay 16-byte vectors.
template <class T>
struct __align__(16) Padded {
    T v;
    uint4 pad;
};

// A draw's chunk shape as passed to the queue and chunk stage: width | height << 8, in tiles.
__host__ __device__ __forceinline__ uint32_t chunk_shape(const DrawArgs& a) {
    const uint32_t w = a.chunkTiles ? a.chunkTiles : (uint32_t)kChunkTiles;
    return w | ((a.chunkTilesY ? a.chunkTilesY : w) << 8);
}

// ShadeMeshlet's vertex transform (Shading.cpp:295-298): the clip position of a vertex slot; slots
// past the 16-vertex chunks up to NumVertices are zero.
__device__ __forceinline__ float4 clip_position(float x, float y, float z, bool live, const ViewParams& vp) {
    return live ? clip_transform(x, y, z, vp.m) : make_float4(0.f, 0.f, 0.f, 0.f);
}

// TriangleEdgeVars::Setup (Rasterizer.cpp:296-329) into a TriRec with its rank (the opaque
// vis-buffer shader does not read the perspective-correct barycentrics; alpha_ext adds them from
// *rcpAreaOut). Returns the fixed-point determinant (> 0, or 0 for a triangle degenerate in fixed
// point).
__device__ __forceinline__ int32_t edge_setup(const Setup& t, int halfW, int halfH, uint32_t bbMin, uint32_t bbMax,
                                              uint32_t rank, TriRec& r, float* rcpAreaOut = nullptr) {
    const Edges e = edge_vars(t, halfW, halfH);
    r.E0 = e.E0, r.E1 = e.E1, r.E2 = e.E2;
    r.A12 = e.A12, r.B12 = e.B12, r.A20 = e.A20, r.B20 = e.B20, r.A01 = e.A01, r.B01 = e.B01;
    r.Z0 = e.Z0, r.Z10 = e.Z10, r.Z20 = e.Z20;
    r.bbMin = bbMin, r.bbMax = bbMax;
    r.lowword = 0xFFFFFFFEu - rank;
    r.pad = 0;
    if (rcpAreaOut) *rcpAreaOut = e.rcpArea;
    return e.det;
}


// ------------------------------------------------------------------ fragments
// DrawTriangle inner loop (Rasterizer.h:287-323) + FS_EncodeSurfaceId<false> (Shading.cpp:309-331)
// for one pixel inside the triangle's render box.
__device__ __forceinline__ void shade_fragment(const TriRec& r, uint32_t px, uint32_t py, unsigned long long* keys,
                                               uint32_t width) {
    int32_t e0 = (int32_t)((uint32_t)r.E0 + (uint32_t)r.A12 * px + (uint32_t)r.B12 * py);
    int32_t e1 = (int32_t)((uint32_t)r.E1 + (uint32_t)r.A20 * px + (uint32_t)r.B20 * py);
    int32_t e2 = (int32_t)((uint32_t)r.E2 + (uint32_t)r.A01 * px + (uint32_t)r.B01 * py);
    if ((e0 | e1 | e2) < 0) return;
    float depth = ffma(__int2float_rn(e1), r.Z10, ffma(__int2float_rn(e2), r.Z20, r.Z0));
    if (depth != depth) return;  // NaN never passes `Depth > old`
    unsigned long long key = ((unsigned long long)float_order(depth) << 32) | r.lowword;
    unsigned long long* p = keys + pixel_offset(px, py, width);
    if (key > *(volatile unsigned long long*)p) atomicMax(p, key);
}

// Tiny triangles, drawn by their own lane. A sample passes the edge tests only inside the closed
// fixed-point triangle (the tests are exact: floor(F / 16) >= 0 iff F >= 0, and the top-left
// biases only remove boundary samples), so its pixel p satisfies 16 (p - half) + 8 in
// [min, max] of the vertices, i.e. p in [(min + 7) >> 4, (max - 8) >> 4] + half, computed per
// 16-bit half (the render box's single 32-bit add can carry from x into y). The tile walk visits
// [bbMin, bbMax). The lane evaluates the pixels of both ranges' intersection: exactly the walk's
// covered pixels. A triangle degenerate in fixed point (det 0) can pass samples on its whole line
// and keeps the walk.
constexpr uint32_t kTinyPixels = 2;
// A meshlet is drawn in the single-view draw's first pass when its bounding sphere's radius exceeds
// this share of the clip w of its centre (about 94 pixels at 1920 pixels across and 60 degrees).
constexpr float kLargeMeshlet = 0.1f;
struct TinyBox { uint32_t x0, y0, x1, y1; };  // inclusive pixel range
__device__ __forceinline__ bool tiny_box(const Setup& t, int halfW, int halfH, uint32_t bbMin, uint32_t bbMax,
                                         TinyBox& b) {
    const uint32_t vp = (uint32_t)halfW | ((uint32_t)halfH << 16);
    const uint32_t lo = srai16_4(__vadd2(__vmins2(__vmins2(t.Pos0, t.Pos1), t.Pos2), 0x00070007u));
    const uint32_t hi = srai16_4(__vsub2(__vmaxs2(__vmaxs2(t.Pos0, t.Pos1), t.Pos2), 0x00080008u));
    const uint32_t x = __vmaxs2(__vadd2(lo, vp), bbMin);
    const uint32_t y = __vmins2(__vadd2(hi, vp), bbMax - 0x00010001u);
    b.x0 = x & 0xFFFF, b.y0 = x >> 16, b.x1 = y & 0xFFFF, b.y1 = y >> 16;
    const int w = (int)(int16_t)(y & 0xFFFF) - (int)(int16_t)(x & 0xFFFF) + 1;
    const int h = (int)(int16_t)(y >> 16) - (int)(int16_t)(x >> 16) + 1;
    return w <= 0 || h <= 0 || w * h <= (int)kTinyPixels;
}

__device__ __forceinline__ void shade_tiny(const TriRec& r, const TinyBox& b, unsigned long long* keys, uint32_t width) {
    for (int y = (int16_t)b.y0; y <= (int16_t)b.y1; y++)
        for (int x = (int16_t)b.x0; x <= (int16_t)b.x1; x++) {
            const uint32_t px = (uint32_t)x, py = (uint32_t)y;
            const int32_t e0 = (int32_t)((uint32_t)r.E0 + (uint32_t)r.A12 * px + (uint32_t)r.B12 * py);
            const int32_t e1 = (int32_t)((uint32_t)r.E1 + (uint32_t)r.A20 * px + (uint32_t)r.B20 * py);
            const int32_t e2 = (int32_t)((uint32_t)r.E2 + (uint32_t)r.A01 * px + (uint32_t)r.B01 * py);
            if ((e0 | e1 | e2) < 0) continue;
            const float depth = ffma(__int2float_rn(e1), r.Z10, ffma(__int2float_rn(e2), r.Z20, r.Z0));
            if (depth != depth) continue;
            atomicMax(keys + pixel_offset(px, py, width), ((unsigned long long)float_order(depth) << 32) | r.lowword);
        }
}

// ceil(256 / n) for n = 1..16, the multiplier of the small triangles' tile -> row multiply-shift:
// ceil(256 / n) - 1 packed 8 bits per entry in two words (an integer divide per triangle costs more
// than the rest of its tile bookkeeping).
__device__ __forceinline__ uint32_t row_magic(int n) {
    const unsigned long long t = n <= 8 ? 0x1f242a333f557fffull : 0xf1112131517191cull;
    return (uint32_t)((t >> (8 * ((n - 1) & 7))) & 0xFF) + 1u;
}

// The terms of a triangle's tile tests that do not depend on the tile, computed once per triangle (in
// the mesh stage by the lane that sets it up, in the chunk stage before a chunk's tiles): with them a tile costs six
// multiply-adds, one sign test, two conversions and two fmas (alpha-tested chunks 629 -> 608 us of a
// 1916x1036 frame, 24-view batched mesh stage 1.47 -> 1.45 ms; opaque chunk stage no change).
//
// F is the edge value at pixel (0, 0) plus the edge's largest increase over a 4x4 tile, so the tile at
// (px, py) holds a sample inside the edge only if F + A px + B py >= 0 (wrapping as the shading's).
//
// zc gives an upper bound of the depth tile_pixel_key computes for any sample of a tile:
// zc + Z10 F1(px, py) + Z20 F2(px, py). The exact depth Z0 + Z10 e1 + Z20 e2 is affine in the pixel: the
// first sample's plus i Gx + j Gy at sample (i, j), Gx = Z10 A20 + Z20 A01, Gy = Z10 B20 + Z20 B01, so
// its maximum over the tile is the first sample's plus 3 max(Gx, 0) + 3 max(Gy, 0), and the first
// sample's edge values are F - s with s the tile increases above. With u = 2^-24 and
// S = |Z0| + |Z10| m1 + |Z20| m2, where m = |E| + |A| X + |B| Y bounds every |e| and |F| in the box and
// eight steps more, a computed sample depth is within 4u S of the exact one and the bound's evaluation
// within 20u S of its own; 2^-18 S = 64u S covers both. A NaN bound never culls (tile_live).
struct __align__(16) TileTest {
    int32_t F0, F1, F2;
    float zc;
};
__device__ __forceinline__ int32_t tile_step(int32_t A, int32_t B) { return 3 * (max(A, 0) + max(B, 0)); }
__device__ __forceinline__ TileTest tile_test(const TriRec& r) {
    const int32_t s1 = tile_step(r.A20, r.B20), s2 = tile_step(r.A01, r.B01);
    TileTest t;
    t.F0 = (int32_t)((uint32_t)r.E0 + (uint32_t)tile_step(r.A12, r.B12));
    t.F1 = (int32_t)((uint32_t)r.E1 + (uint32_t)s1);
    t.F2 = (int32_t)((uint32_t)r.E2 + (uint32_t)s2);
    const float X = (float)((r.bbMax & 0xFFFF) + 8), Y = (float)((r.bbMax >> 16) + 8);
    const float a20 = (float)r.A20, b20 = (float)r.B20, a01 = (float)r.A01, b01 = (float)r.B01;
    const float m1 = ffma(fabsf(a20), X, ffma(fabsf(b20), Y, fabsf((float)r.E1)));
    const float m2 = ffma(fabsf(a01), X, ffma(fabsf(b01), Y, fabsf((float)r.E2)));
    const float S = ffma(fabsf(r.Z10), m1, ffma(fabsf(r.Z20), m2, fabsf(r.Z0)));
    const float gx = ffma(r.Z10, a20, fmul(r.Z20, a01)), gy = ffma(r.Z10, b20, fmul(r.Z20, b01));
    float z = ffma(3.0f, fadd(fmaxf(gx, 0.0f), fmaxf(gy, 0.0f)), r.Z0);
    z = ffma(-r.Z10, (float)s1, ffma(-r.Z20, (float)s2, z));
    t.zc = ffma(S, 0x1p-18f, z);
    return t;
}

// Raises the tile's depth bound to the minimum of the values its 16 pixels reported (the two
// halves of the warp shade one tile each). A bound rises only if every pixel's value is above it, which a
// ballot tells for both halves; the two whole-warp reductions, each over one half's values, run only then.
__device__ __forceinline__ void update_tile_min(uint32_t obs, uint32_t* tileMin, uint32_t tileIdx, uint32_t known,
                                                bool active, int lane) {
    const unsigned above = __ballot_sync(0xFFFFFFFFu, active && obs > known);
    if ((above & 0xFFFFu) != 0xFFFFu && (above >> 16) != 0xFFFFu) return;
    const bool upper = lane & 16;
    const uint32_t lo = __reduce_min_sync(0xFFFFFFFFu, upper ? 0xFFFFFFFFu : obs);
    const uint32_t hi = __reduce_min_sync(0xFFFFFFFFu, upper ? obs : 0xFFFFFFFFu);
    obs = upper ? hi : lo;
    if (active && (lane & 15) == 0 && obs > known) atomicMax(&tileMin[tileIdx], obs);
}

// One lane rasterizes a whole triangle (fallback of the rare clipped triangle that finds the
// queue full; slow but exact).
__device__ __noinline__ void raster_serial(const TriRec& r, unsigned long long* keys, uint32_t width) {
    uint32_t minX = r.bbMin & 0xFFFF, minY = r.bbMin >> 16, maxX = r.bbMax & 0xFFFF, maxY = r.bbMax >> 16;
    for (uint32_t y = minY; y < maxY; y++)
        for (uint32_t x = minX; x < maxX; x++) shade_fragment(r, x, y, keys, width);
}

// Takes back a claim of the chunk queue that has no room (swr_queue.h).
__device__ __forceinline__ void queue_release(const DrawArgs& a, unsigned long long claim) {
    atomicAdd(&a.s.control[1], 0ull - claim);
    atomicOr(&a.s.control[2], kStatusBigOverflow);
}

// The chunks (chunk_shape) of a triangle's render box.
__device__ __forceinline__ uint32_t triangle_chunks(const TriRec& r, uint32_t chunk) {
    const uint32_t tilesX = ((r.bbMax & 0xFFFF) - (r.bbMin & 0xFFFF)) >> 2, tilesY = ((r.bbMax >> 16) - (r.bbMin >> 16)) >> 2;
    const uint32_t cw = chunk & 0xFF, ch = chunk >> 8;
    return ((tilesX + cw - 1) / cw) * ((tilesY + ch - 1) / ch);
}

// Appends a triangle (its view index in r.pad) to the chunk queue; false when the queue is full
// (the caller rasterizes it).
__device__ __forceinline__ bool enqueue_big(const TriRec& r, const DrawArgs& a, uint32_t chunk) {
    const unsigned long long claim = queue_claim(1, triangle_chunks(r, chunk));
    const unsigned long long old = atomicAdd(&a.s.control[1], claim);
    const uint32_t slot = queue_slots(old);
    if (!queue_fits(slot, queue_chunks(old), 1, a.s.bigCapacity)) {
        queue_release(a, claim);
        return false;
    }
    a.s.big[slot] = r;
    a.s.bigBase[slot] = queue_chunks(old);
    return true;
}

// ------------------------------------------------------------------ alpha test
// FS_EncodeSurfaceId<true> (Shading.cpp:309-331): after the depth test, the fragment's
// perspective-correct barycentrics (Rasterizer.h:300-317, rcp14 reproduced exactly) interpolate the
// vertices' texcoords (FragmentVars::Interpolate = BaryLerp, Rasterizer.h:101-104), the material's
// texture is sampled at the implicit LOD of the 4x4 tile (SampleImplicitLod, Texture.h:403-410,
// with the 2x2 finite differences texutil::dFdx/dFdy, Texture.h:258-275) and the fragment survives
// if the texel is >= AlphaCutoff << 24. Every sample of a visited tile takes part in the
// differences and in the tile's filter choice, covered or not, as the reference's 16 lanes do.

// Mesh::TexCoords[VertexId]. The index byte is not bounded by the reference, whose record holds
// NormalTangents and Indices after the 64 texcoords: indices below 224 read that word of the
// record, larger ones (the next record in the reference) read 0.
__device__ __forceinline__ uint32_t texcoord_word(const uint8_t* mp, uint32_t idx) {
    return idx < 224 ? *(const uint32_t*)(mp + kOffTexCoords + 4 * idx) : 0u;
}

// Alpha-test terms of a triangle from its setup (TriangleEdgeVars W terms, Rasterizer.cpp:320-328).
__device__ __forceinline__ AlphaExt alpha_ext(const Setup& t, float rcpArea, uint32_t tc0, uint32_t tc1, uint32_t tc2,
                                              uint32_t material) {
    AlphaExt x;
    x.W0 = t.W0;
    x.W0S = fmul(t.W0, rcpArea), x.W1S = fmul(t.W1, rcpArea), x.W2S = fmul(t.W2, rcpArea);
#pragma unroll
    for (int k = 0; k < 3; k++) x.ru[k] = 0.0f, x.rv[k] = 0.0f;
    x.tc0 = tc0, x.tc1 = tc1, x.tc2 = tc2;
    x.zero0 = 0, x.zero1 = 0;
    x.material = material;
    return x;
}

struct TexCoord { float u, v; };

// Interpolated texcoord of the sample whose edge values are (u, v) (as floats).
__device__ __forceinline__ TexCoord alpha_texcoord(const AlphaExt& x, float u, float v) {
    float bu, bv;  // clipped (kTriAlpha): barycentrics of the source triangle
    perspective_bary(u, v, x.W0, x.W0S, x.W1S, x.W2S, (x.material & kTriAlpha) != 0, x.ru, x.rv, bu, bv);
    const float b0 = fsub(fsub(1.0f, bu), bv);
    TexCoord s;
    s.u = ffma(h2f(x.tc0 & 0xFFFF), b0, ffma(h2f(x.tc1 & 0xFFFF), bu, fmul(h2f(x.tc2 & 0xFFFF), bv)));
    s.v = ffma(h2f(x.tc0 >> 16), b0, ffma(h2f(x.tc1 >> 16), bu, fmul(h2f(x.tc2 >> 16), bv)));
    return s;
}

// CalcMipLevel(grad) - LerpFracBits (Texture.h:271-275, 408) from the differences of the scaled
// sample positions (d/dx su, d/dx sv, d/dy su, d/dy sv).
__device__ __forceinline__ int32_t alpha_mip(float gx, float gy, float gz, float gw) {
    const float dx = ffma(gx, gx, fmul(gy, gy)), dy = ffma(gz, gz, fmul(gw, gw));
    return (ilog2_x86(vmax(dx, dy)) >> 1) - 8;
}

// The opaque tile shading of shade_live_tiles with the alpha test, for pixel (tx + l % 4,
// ty + l / 4), l = lane % 16, called by all 32 lanes: each half-warp shades one tile
// (valid is false on a half without one); cur is the pixel's key, read before (0: no tile). The x and y
// differences pair lanes l ^ 1 and l ^ 4 of a half. Returns a lower bound of the pixel's depth word.
__device__ __forceinline__ uint32_t shade_tile_pixel_alpha(const TriRec& r, const AlphaExt& x, const DevTexture& tex,
                                                           uint32_t cutoff, uint32_t tx, uint32_t ty, bool valid, int lane,
                                                           unsigned long long* p, unsigned long long cur) {
    const uint32_t l = lane & 15;
    const uint32_t px = tx + (l & 3), py = ty + (l >> 2);
    const int32_t e0 = (int32_t)((uint32_t)r.E0 + (uint32_t)r.A12 * px + (uint32_t)r.B12 * py);
    const int32_t e1 = (int32_t)((uint32_t)r.E1 + (uint32_t)r.A20 * px + (uint32_t)r.B20 * py);
    const int32_t e2 = (int32_t)((uint32_t)r.E2 + (uint32_t)r.A01 * px + (uint32_t)r.B01 * py);
    const float u = __int2float_rn(e1), v = __int2float_rn(e2);
    const float depth = ffma(u, r.Z10, ffma(v, r.Z20, r.Z0));
    const unsigned long long key = ((unsigned long long)float_order(depth) << 32) | r.lowword;
    bool pass = valid && (e0 | e1 | e2) >= 0 && depth == depth && key > cur;
    if (__any_sync(0xFFFFFFFFu, pass)) {
        const TexCoord s = alpha_texcoord(x, u, v);
        const float su = fmul(s.u, tex.scale_lerp_u), sv = fmul(s.v, tex.scale_lerp_v);
        const float sux = __shfl_xor_sync(0xFFFFFFFFu, su, 1), svx = __shfl_xor_sync(0xFFFFFFFFu, sv, 1);
        const float suy = __shfl_xor_sync(0xFFFFFFFFu, su, 4), svy = __shfl_xor_sync(0xFFFFFFFFu, sv, 4);
        // dFdx = p[l | 1] - p[l & ~1], dFdy = p[l | 4] - p[l & ~4]; alpha_mip squares them, so their sign is free
        const int32_t mip = alpha_mip(fsub(su, sux), fsub(sv, svx), fsub(su, suy), fsub(sv, svy));
        const bool nearest = (__ballot_sync(0xFFFFFFFFu, mip > 0) & (0xFFFFu << (lane & 16))) != 0;
        if (pass) pass = sample_alpha8(tex, s.u, s.v, mip, nearest) >= cutoff;
    }
    if (!pass) return (uint32_t)(cur >> 32);
    atomicMax(p, key);
    return (uint32_t)(key >> 32);
}

// One lane rasterizes a whole alpha-tested triangle, the 16 samples of each tile in turn
// (fallback of a triangle that finds the queue full; slow but exact).
__device__ __noinline__ void raster_serial_alpha(const TriRec& r, const AlphaExt& x, const DevMaterial* materials,
                                                 unsigned long long* keys, uint32_t width) {
    const DevMaterial& mt = materials[x.material & ~kTriAlpha];
    const uint32_t cutoff = mt.alpha_cutoff;
    const uint32_t minX = r.bbMin & 0xFFFF, minY = r.bbMin >> 16, maxX = r.bbMax & 0xFFFF, maxY = r.bbMax >> 16;
    for (uint32_t ty = minY; ty < maxY; ty += 4) {
        for (uint32_t tx = minX; tx < maxX; tx += 4) {
            float su[16], sv[16], tu[16], tv[16];
            unsigned pass = 0;
            for (uint32_t l = 0; l < 16; l++) {
                const uint32_t px = tx + (l & 3), py = ty + (l >> 2);
                const int32_t e0 = (int32_t)((uint32_t)r.E0 + (uint32_t)r.A12 * px + (uint32_t)r.B12 * py);
                const int32_t e1 = (int32_t)((uint32_t)r.E1 + (uint32_t)r.A20 * px + (uint32_t)r.B20 * py);
                const int32_t e2 = (int32_t)((uint32_t)r.E2 + (uint32_t)r.A01 * px + (uint32_t)r.B01 * py);
                const float u = __int2float_rn(e1), v = __int2float_rn(e2);
                const float depth = ffma(u, r.Z10, ffma(v, r.Z20, r.Z0));
                const unsigned long long key = ((unsigned long long)float_order(depth) << 32) | r.lowword;
                if ((e0 | e1 | e2) >= 0 && depth == depth && key > *(volatile unsigned long long*)(keys + (tx << 2) + ty * width + l))
                    pass |= 1u << l;
                const TexCoord s = alpha_texcoord(x, u, v);
                tu[l] = s.u, tv[l] = s.v;
                su[l] = fmul(s.u, mt.tex.scale_lerp_u), sv[l] = fmul(s.v, mt.tex.scale_lerp_v);
            }
            if (!pass) continue;
            int32_t mip[16];
            bool nearest = false;
            for (uint32_t l = 0; l < 16; l++) {
                const uint32_t lx = l & ~1u, hx = l | 1u, ly = l & ~4u, hy = l | 4u;
                mip[l] = alpha_mip(fsub(su[hx], su[lx]), fsub(sv[hx], sv[lx]), fsub(su[hy], su[ly]), fsub(sv[hy], sv[ly]));
                nearest |= mip[l] > 0;
            }
            for (uint32_t l = 0; l < 16; l++) {
                if (!((pass >> l) & 1) || sample_alpha8(mt.tex, tu[l], tv[l], mip[l], nearest) < cutoff) continue;
                const uint32_t px = tx + (l & 3), py = ty + (l >> 2);
                const int32_t e1 = (int32_t)((uint32_t)r.E1 + (uint32_t)r.A20 * px + (uint32_t)r.B20 * py);
                const int32_t e2 = (int32_t)((uint32_t)r.E2 + (uint32_t)r.A01 * px + (uint32_t)r.B01 * py);
                const float depth = ffma(__int2float_rn(e1), r.Z10, ffma(__int2float_rn(e2), r.Z20, r.Z0));
                atomicMax(keys + (tx << 2) + ty * width + l, ((unsigned long long)float_order(depth) << 32) | r.lowword);
            }
        }
    }
}

// Appends an alpha-tested triangle and its AlphaExt (in the next slot, which owns no chunks) to
// the chunk queue; false when the queue is full (the caller rasterizes it).
__device__ __forceinline__ bool enqueue_alpha(const TriRec& r, const AlphaExt& x, const DrawArgs& a, uint32_t chunk) {
    const uint32_t chunks = triangle_chunks(r, chunk);
    const unsigned long long claim = queue_claim(2, chunks);
    const unsigned long long old = atomicAdd(&a.s.control[1], claim);
    const uint32_t slot = queue_slots(old);
    const unsigned long long base = queue_chunks(old);
    if (!queue_fits(slot, base, 2, a.s.bigCapacity)) {
        queue_release(a, claim);
        return false;
    }
    a.s.big[slot] = r;
    a.s.big[slot + 1] = *(const TriRec*)&x;
    a.s.bigBase[slot] = base;
    a.s.bigBase[slot + 1] = base + chunks;
    return true;
}

// Appends the records of the lanes with `want` (rec, its view index in pad; alpha-tested ones with their
// terms x in the next slot) to the chunk queue, called by all 32 lanes of a packet; false on a lane whose
// triangle found the queue full. One atomic serves the warp: the queue's tail is one word, and an atomic
// per triangle (488k in the 1080p frame of 100k meshlets, about one a clock) kept every warp waiting:
// mesh stage 645 -> 408 us there, 282 -> 220 us for a 20k-meshlet overdraw draw, 428 -> 265 us from inside a
// 60k-meshlet scene.
template <bool kAlpha>
__device__ __forceinline__ bool enqueue_warp(bool want, const TriRec& rec, const AlphaExt* x, const DrawArgs& a, uint32_t chunk,
                                             int lane) {
    const unsigned m = __ballot_sync(0xFFFFFFFFu, want);
    if (m == 0) return true;
    constexpr uint32_t kSlots = kAlpha ? 2 : 1;
    const uint32_t chunks = want ? triangle_chunks(rec, chunk) : 0u;
    uint32_t incl = chunks;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += v;
    }
    unsigned long long old = 0;
    if (lane == 31) old = atomicAdd(&a.s.control[1], queue_claim(__popc(m) * kSlots, incl));
    old = __shfl_sync(0xFFFFFFFFu, old, 31);
    const uint32_t slot = queue_slots(old) + __popc(m & ((1u << lane) - 1u)) * kSlots;
    const unsigned long long base = queue_chunks(old) + (incl - chunks);
    const bool fits = queue_fits(slot, base, kSlots, a.s.bigCapacity);
    if (want && fits) {
        a.s.big[slot] = rec;
        a.s.bigBase[slot] = base;
        if constexpr (kAlpha) {
            a.s.big[slot + 1] = *(const TriRec*)x;
            a.s.bigBase[slot + 1] = base + chunks;
        }
    }
    const unsigned full = __ballot_sync(0xFFFFFFFFu, want && !fits);
    if (full) {  // the last lanes' claims: one addition for all
        const uint32_t all = __shfl_sync(0xFFFFFFFFu, incl, 31);
        if (lane == __ffs(full) - 1) queue_release(a, queue_claim(__popc(full) * kSlots, all - (incl - chunks)));
    }
    return !want || fits;
}

// A small triangle's record (the mesh stage's tile walk): pad = tilesX | row_magic << 8 | kPadReadKey.
// A triangle of more tiles has kPadWide instead of the first two.
constexpr uint32_t kPadReadKey = 1u << 24, kPadWide = 1u << 25;
// The 4x4 tiles of a triangle's render box.
__device__ __forceinline__ uint32_t triangle_tiles(const TriRec& r) {
    return (((r.bbMax & 0xFFFF) - (r.bbMin & 0xFFFF)) >> 2) * (((r.bbMax >> 16) - (r.bbMin >> 16)) >> 2);
}

// Upper bound of any fragment depth of a triangle from its vertex depths: a fragment's depth is its
// edge functions' interpolation of Z0, Z1, Z2 inside the triangle, so at most their maximum, plus the
// roundings of the plane terms and of the evaluation, within 16 ulp of the largest |Z| (2^-20);
// 2^-16 of it is kept. For a small triangle this is much tighter than the plane's value at the tile
// corners, which lie outside it. NaN vertex depths give a NaN, which never beats a fragment's.
__device__ __forceinline__ float triangle_depth_bound(const Setup& t) {
    const float m = fmaxf(fmaxf(fabsf(t.Z0), fabsf(t.Z1)), fabsf(t.Z2));
    const bool nan = t.Z0 != t.Z0 || t.Z1 != t.Z1 || t.Z2 != t.Z2;
    return nan ? __int_as_float(0x7F800000) : fadd(fmaxf(fmaxf(t.Z0, t.Z1), t.Z2), fmul(m, 0x1p-16f));
}

// True if the tile at (px, py) (4-aligned) can be shaded for r: some sample may pass the edges
// and, when a depth bound is kept, r may beat the tile's depth bound somewhere. *known receives
// the bound read (for the later update). zmax is a second bound of the triangle's depth
// (triangle_depth_bound; +inf: none). The bound compares as an ordered word: a negative one counts as
// 0, which only culls less; the NaN the fmas give is the positive 0x7FFFFFFF, above every depth.
__device__ __forceinline__ bool tile_live(const TriRec& r, const TileTest& t, uint32_t px, uint32_t py,
                                          const uint32_t* tileMin, uint32_t tilesPerRow, uint32_t* known, float zmax) {
    const int32_t f0 = (int32_t)((uint32_t)t.F0 + (uint32_t)r.A12 * px + (uint32_t)r.B12 * py);
    const int32_t f1 = (int32_t)((uint32_t)t.F1 + (uint32_t)r.A20 * px + (uint32_t)r.B20 * py);
    const int32_t f2 = (int32_t)((uint32_t)t.F2 + (uint32_t)r.A01 * px + (uint32_t)r.B01 * py);
    if ((f0 | f1 | f2) < 0) return false;
    if (!tileMin) return true;
    *known = tileMin[(py >> 2) * tilesPerRow + (px >> 2)];
    const float b = ffma(__int2float_rn(f1), r.Z10, ffma(__int2float_rn(f2), r.Z20, t.zc));
    return ((uint32_t)max(__float_as_int(fminf(b, zmax)), 0) | 0x80000000u) >= *known;
}

// The key DrawTriangle + FS_EncodeSurfaceId<false> (Rasterizer.h:287-323, Shading.cpp:309-331)
// offers for pixel (tx + l % 4, ty + l / 4) of the 4x4 tile at the 4-aligned (tx, ty), 0 if the
// sample is outside the triangle or its depth is NaN. The tiled key offset is the tile's base
// plus l, so a tile's 16 keys are one 128-byte line.
__device__ __forceinline__ unsigned long long tile_pixel_key(const TriRec& r, uint32_t tx, uint32_t ty, uint32_t l) {
    const uint32_t px = tx + (l & 3), py = ty + (l >> 2);
    const int32_t e0 = (int32_t)((uint32_t)r.E0 + (uint32_t)r.A12 * px + (uint32_t)r.B12 * py);
    const int32_t e1 = (int32_t)((uint32_t)r.E1 + (uint32_t)r.A20 * px + (uint32_t)r.B20 * py);
    const int32_t e2 = (int32_t)((uint32_t)r.E2 + (uint32_t)r.A01 * px + (uint32_t)r.B01 * py);
    if ((e0 | e1 | e2) < 0) return 0ull;
    const float depth = ffma(__int2float_rn(e1), r.Z10, ffma(__int2float_rn(e2), r.Z20, r.Z0));
    if (depth != depth) return 0ull;  // NaN never passes `Depth > old`
    return ((unsigned long long)float_order(depth) << 32) | r.lowword;
}

// Shades the live tiles of the warp-wide candidate set (the lanes in `mask` hold a tile origin
// tpx/tpy, its depth bound tmin and a triangle selector rsel for rec()) and raises the tiles' depth
// bounds (each pixel reports a lower bound of its depth word afterwards). The live tiles are first packed
// into `list` (32 entries of shared memory): a step then reads its tiles' entries instead of searching the
// mask and shuffling every field. Four tiles per step: each half-warp takes two, and a lane's two key loads
// are issued together (the walk is bound by instruction issue and by their latency). With the packed list
// and update_tile_min's ballot: 1080p mesh stage of 100k meshlets 408 -> 379 us, 60k meshlets from inside
// 265 -> 237 us. Loading the next step's keys ahead cost spills: 443 us.
template <class Rec, class ReadKey>
__device__ __forceinline__ void shade_live_tiles(Rec&& rec, ReadKey&& readKey, uint32_t rsel, unsigned mask, uint32_t tpx,
                                                 uint32_t tpy, uint32_t tmin, unsigned long long* keys, uint32_t* tileMin,
                                                 uint32_t width, int lane, uint4* list) {
    const uint32_t half = lane >> 4, l = lane & 15, m = __popc(mask);
    if ((mask >> lane) & 1)  // key offset of the tile, its origin (below 2896), depth bound and triangle
        list[__popc(mask & ((1u << lane) - 1u))] = make_uint4((tpx << 2) + tpy * width, tpx | (tpy << 16), tmin, rsel);
    __syncwarp();
    unsigned long long* k = keys + l;
    // The key read filters losing atomics and gives the tile bound each pixel's new depth. For
    // triangles whose readKey(selector) is false (above the draw's keyReadTiles tiles) it is
    // skipped: the atomic is unconditional and a pixel's bound is max(new depth, old tile
    // bound), still a lower bound of its final key.
    auto fetch = [&](uint32_t i, uint4& e, bool& valid, bool& read, unsigned long long& cur) {
        e = list[i & 31];
        valid = i < m;
        read = valid && readKey(valid ? e.w : 0u);
        cur = read ? *(volatile unsigned long long*)(k + e.x) : 0ull;
    };
    auto shade = [&](const uint4& e, bool valid, bool read, unsigned long long cur) {
        const unsigned long long key = valid ? tile_pixel_key(rec(e.w), e.y & 0xFFFF, e.y >> 16, l) : 0ull;
        if (key > cur) atomicMax(k + e.x, key);
        if (tileMin) {
            const uint32_t obs = read ? (uint32_t)((key > cur ? key : cur) >> 32) : max((uint32_t)(key >> 32), e.z);
            update_tile_min(obs, tileMin, e.x >> 4, e.z, valid, lane);
        }
    };
    for (uint32_t i = 0; i < m; i += 4) {
        uint4 a, b;
        bool va, vb, ra, rb;
        unsigned long long ca, cb;
        fetch(i + half, a, va, ra, ca);
        fetch(i + 2 + half, b, vb, rb, cb);
        shade(a, va, ra, ca);
        shade(b, vb, rb, cb);
    }
    __syncwarp();
}

// shade_live_tiles for alpha-tested triangles of one material (texture tex, alpha cutoff): a
// candidate's triangle is rec(rsel), its alpha terms ext(rsel) (the tiles of a step may belong
// to different triangles). The keys of both tiles of a half-warp are loaded first (alpha pass of a G-buffer
// draw 431 -> 385 us).
template <class Rec, class Ext>
__device__ __forceinline__ void shade_live_tiles_alpha(Rec&& rec, Ext&& ext, uint32_t rsel,
                                                       const DevTexture& tex, uint32_t cutoff, unsigned mask,
                                                       uint32_t tpx, uint32_t tpy, uint32_t tmin,
                                                       unsigned long long* keys, uint32_t* tileMin, uint32_t width,
                                                       int lane, uint4* list) {
    const uint32_t half = lane >> 4, l = lane & 15, m = __popc(mask);
    if ((mask >> lane) & 1)
        list[__popc(mask & ((1u << lane) - 1u))] = make_uint4((tpx << 2) + tpy * width, tpx | (tpy << 16), tmin, rsel);
    __syncwarp();
    unsigned long long* k = keys + l;
    for (uint32_t i = half; i - half < m; i += 4) {
        unsigned long long cur[2];
#pragma unroll
        for (int j = 0; j < 2; j++) cur[j] = i + 2 * j < m ? *(volatile unsigned long long*)(k + list[(i + 2 * j) & 31].x) : 0ull;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            if (i - half + 2 * j >= m) break;  // neither half has a tile
            const uint32_t n = i + 2 * j;
            const bool valid = n < m;
            const uint4 e = list[valid ? n : 0];
            const uint32_t obs = shade_tile_pixel_alpha(rec(e.w), ext(e.w), tex, cutoff, e.y & 0xFFFF, e.y >> 16, valid, lane,
                                                        k + e.x, cur[j]);
            if (tileMin) update_tile_min(obs, tileMin, e.x >> 4, e.z, valid, lane);
        }
    }
    __syncwarp();
}

// ceil(2^16 / n) for n = 1..16: t / n == (t * kDiv16[n]) >> 16 for every t < 256 (checked
// exhaustively), the tile index division of a chunk of at most 16 x 16 tiles.
__constant__ uint32_t kDiv16[17] = { 0, 65536, 32768, 21846, 16384, 13108, 10923, 9363, 8192,
                                     7282, 6554, 5958, 5462, 5042, 4682, 4370, 4096 };

// Rasterizes the tiles of [x0, x0 + 4*tilesX) x [y0, y0 + 4*tilesY) that are not provably empty
// or hidden: 32 tiles are tested at a time (one per lane), then shade(mask, tpx, tpy, tmin) shades
// the surviving ones. Returns whether there were any. divMagic: kDiv16[tilesX] for a chunk (tilesX, tilesY <= 16), 0 otherwise.
template <class Shade>
__device__ __forceinline__ bool raster_region_with(const TriRec& r, const TileTest& tt, uint32_t x0, uint32_t y0, int tilesX, int tilesY,
                                                   const uint32_t* tileMin, uint32_t width, int lane, Shade&& shade,
                                                   uint32_t divMagic) {
    const int T = tilesX * tilesY;
    const uint32_t tw = width >> 2;
    bool any = false;
    for (int tb = 0; tb < T; tb += 32) {
        const int t = tb + lane;
        bool live = false;
        uint32_t tpx = 0, tpy = 0, tmin = 0;
        if (t < T) {
            int ty = divMagic ? (int)(((uint32_t)t * divMagic) >> 16) : t / tilesX, tx = t - ty * tilesX;
            tpx = x0 + tx * 4, tpy = y0 + ty * 4;
            live = tile_live(r, tt, tpx, tpy, tileMin, tw, &tmin, __int_as_float(0x7F800000));
        }
        const unsigned mask = __ballot_sync(0xFFFFFFFFu, live);
        if (mask) shade(mask, tpx, tpy, tmin);
        any = any || mask;
    }
    return any;
}

// raster_region_with for an opaque triangle, four tiles per step.
__device__ __forceinline__ bool raster_region(const TriRec& r, const TileTest& tt, uint32_t x0, uint32_t y0, int tilesX, int tilesY,
                                              unsigned long long* keys, uint32_t* tileMin, uint32_t width, int lane, uint32_t readTiles,
                                              uint4* list, uint32_t divMagic = 0) {
    const bool readKey = readTiles == 0 || triangle_tiles(r) <= readTiles;
    return raster_region_with(r, tt, x0, y0, tilesX, tilesY, tileMin, width, lane,
                       [&](unsigned mask, uint32_t tpx, uint32_t tpy, uint32_t tmin) {
                           shade_live_tiles([&](uint32_t) -> const TriRec& { return r; }, [&](uint32_t) { return readKey; }, 0,
                                            mask, tpx, tpy, tmin, keys, tileMin, width, lane, list);
                       }, divMagic);
}

// The same for the alpha-tested triangle *rp with alpha terms *xp (material texture tex, alpha cutoff).
__device__ __forceinline__ bool raster_region_alpha(const TriRec* rp, const TileTest& tt, const AlphaExt* xp, const DevTexture& tex,
                                                    uint32_t cutoff, uint32_t x0, uint32_t y0, int tilesX, int tilesY,
                                                    unsigned long long* keys, uint32_t* tileMin, uint32_t width, int lane,
                                                    uint4* list, uint32_t divMagic = 0) {
    return raster_region_with(*rp, tt, x0, y0, tilesX, tilesY, tileMin, width, lane,
                       [&](unsigned mask, uint32_t tpx, uint32_t tpy, uint32_t tmin) {
                           shade_live_tiles_alpha([&](uint32_t) -> const TriRec& { return *rp; },
                                                  [&](uint32_t) -> const AlphaExt& { return *xp; }, 0, tex, cutoff, mask, tpx,
                                                  tpy, tmin, keys, tileMin, width, lane, list);
                       }, divMagic);
}

// ------------------------------------------------------------------ overdraw shader
// FS_Overdraw (Shading.cpp:333-342) over the live tiles of the warp-wide candidate set, packed and stepped as
// shade_live_tiles does (no depth bounds: every tile a triangle covers counts). DrawTriangle visits a tile
// only if a sample is covered; then every sample counts, covered ones in the high word of the pixel's counter and
// the others in the low word, and the tile's 16 depths feed a maximum kept in the key's high word (NaN never
// replaces: vmaxps keeps the old value). The keys of both tiles of a half-warp are loaded ahead: mesh stage of 20,000
// meshlets at 1280x720 209 -> 160 us (one tile a half-warp and step 196, a mask walked with shuffles 209), chunk stage
// 164 -> 146 us with 64 registers (171 with 48, which spill).
template <class Rec>
__device__ __forceinline__ void shade_live_tiles_overdraw(Rec&& rec, uint32_t rsel, unsigned mask, uint32_t tpx, uint32_t tpy,
                                                          unsigned long long* keys, unsigned long long* counts,
                                                          uint32_t width, int lane, uint4* list) {
    const uint32_t half = lane >> 4, l = lane & 15, m = __popc(mask);
    if ((mask >> lane) & 1) list[__popc(mask & ((1u << lane) - 1u))] = make_uint4((tpx << 2) + tpy * width, tpx | (tpy << 16), rsel, 0);
    __syncwarp();
    auto fetch = [&](uint32_t i, uint4& e, unsigned long long& cur) {
        e = list[i & 31];
        cur = i < m ? *(volatile unsigned long long*)&keys[e.x + l] : 0ull;
    };
    auto shade = [&](uint32_t i, const uint4& e, unsigned long long cur) {
        const bool valid = i < m;
        const TriRec& r = rec(valid ? e.z : 0u);
        const uint32_t px = (e.y & 0xFFFF) + (l & 3), py = (e.y >> 16) + (l >> 2);
        const int32_t e0 = (int32_t)((uint32_t)r.E0 + (uint32_t)r.A12 * px + (uint32_t)r.B12 * py);
        const int32_t e1 = (int32_t)((uint32_t)r.E1 + (uint32_t)r.A20 * px + (uint32_t)r.B20 * py);
        const int32_t e2 = (int32_t)((uint32_t)r.E2 + (uint32_t)r.A01 * px + (uint32_t)r.B01 * py);
        const bool covered = valid && (e0 | e1 | e2) >= 0;
        if (!((__ballot_sync(0xFFFFFFFFu, covered) >> (lane & 16)) & 0xFFFFu)) return;
        atomicAdd(&counts[e.x + l], covered ? (1ull << 32) : 1ull);
        const float depth = ffma(__int2float_rn(e1), r.Z10, ffma(__int2float_rn(e2), r.Z20, r.Z0));
        const unsigned long long key = (unsigned long long)float_order(depth) << 32;
        if (depth == depth && key > cur) atomicMax(&keys[e.x + l], key);
    };
    for (uint32_t i = half; i - half < m; i += 4) {
        uint4 a, b;
        unsigned long long ca, cb;
        fetch(i, a, ca);
        fetch(i + 2, b, cb);
        shade(i, a, ca);
        __syncwarp();
        shade(i + 2, b, cb);
        __syncwarp();
    }
}

__device__ __forceinline__ bool raster_region_overdraw(const TriRec& r, const TileTest& tt, uint32_t x0, uint32_t y0, int tilesX, int tilesY,
                                                       unsigned long long* keys, unsigned long long* counts,
                                                       uint32_t width, int lane, uint4* list, uint32_t divMagic = 0) {
    return raster_region_with(r, tt, x0, y0, tilesX, tilesY, nullptr, width, lane,
                       [&](unsigned mask, uint32_t tpx, uint32_t tpy, uint32_t) {
                           shade_live_tiles_overdraw([&](uint32_t) -> const TriRec& { return r; }, 0, mask, tpx, tpy, keys,
                                                     counts, width, lane, list);
                       }, divMagic);
}

// One lane draws a whole triangle with the overdraw shader (the full-queue fallback of a clipped
// triangle).
__device__ __noinline__ void raster_serial_overdraw(const TriRec& r, unsigned long long* keys, unsigned long long* counts,
                                                    uint32_t width) {
    const uint32_t minX = r.bbMin & 0xFFFF, minY = r.bbMin >> 16, maxX = r.bbMax & 0xFFFF, maxY = r.bbMax >> 16;
    for (uint32_t ty = minY; ty < maxY; ty += 4) {
        for (uint32_t tx = minX; tx < maxX; tx += 4) {
            unsigned cov = 0;
            for (uint32_t l = 0; l < 16; l++) {
                const uint32_t px = tx + (l & 3), py = ty + (l >> 2);
                const int32_t e0 = (int32_t)((uint32_t)r.E0 + (uint32_t)r.A12 * px + (uint32_t)r.B12 * py);
                const int32_t e1 = (int32_t)((uint32_t)r.E1 + (uint32_t)r.A20 * px + (uint32_t)r.B20 * py);
                const int32_t e2 = (int32_t)((uint32_t)r.E2 + (uint32_t)r.A01 * px + (uint32_t)r.B01 * py);
                if ((e0 | e1 | e2) >= 0) cov |= 1u << l;
            }
            if (!cov) continue;
            for (uint32_t l = 0; l < 16; l++) {
                const uint32_t px = tx + (l & 3), py = ty + (l >> 2), off = (tx << 2) + ty * width + l;
                atomicAdd(&counts[off], ((cov >> l) & 1) ? (1ull << 32) : 1ull);
                const int32_t e1 = (int32_t)((uint32_t)r.E1 + (uint32_t)r.A20 * px + (uint32_t)r.B20 * py);
                const int32_t e2 = (int32_t)((uint32_t)r.E2 + (uint32_t)r.A01 * px + (uint32_t)r.B01 * py);
                const float depth = ffma(__int2float_rn(e1), r.Z10, ffma(__int2float_rn(e2), r.Z20, r.Z0));
                if (depth == depth) atomicMax(&keys[off], (unsigned long long)float_order(depth) << 32);
            }
        }
    }
}

// Clipper::ClipTriangles + FlushPacket (Rasterizer.cpp:398-491) for this lane's triangle; the
// lanes of a packet are independent (each prim restarts its new-vertex slots). Fan outputs are
// set up with TrianglePacket::Setup and queued with rank (packet, clipped, lane, fan index).
// For an alpha-tested material (alphaMat != ~0u) the barycentric rows are clipped too and become
// the outputs' TriangleClipData; the texcoords are those of the source triangle (record mp, index
// bytes idxBytes).
__device__ __noinline__ void clip_and_queue(Vtx v0, Vtx v1, Vtx v2, uint32_t outcodes, const DrawArgs& a,
                                            const ViewParams& vp, uint32_t viewIndex, uint32_t chunk, int cullMode,
                                            uint32_t gMeshlet, uint32_t prim, uint32_t& nRaster,
                                            uint32_t alphaMat, const uint8_t* mp, const uint8_t* idxBytes) {
    const bool alpha = alphaMat != ~0u;
    ClipPoly P;
    if (!clip_polygon(v0, v1, v2, outcodes, vp.bx, vp.by, alpha ? 6 : 4, P)) {
        atomicOr(&a.s.control[2], kStatusClipOverflow);
        return;
    }
    const uint32_t vertCount = P.count;
    if (vertCount < 2) return;
    for (uint32_t vi = 0; vi + 2 < vertCount; vi++) {
        Vtx a0, a1, a2;
        float ru[3], rv[3];
        clip_fan(P, vi, a0, a1, a2, alpha ? ru : nullptr, rv);
        Setup t;
        uint32_t bbMin, bbMax;
        if (!tri_setup(a0, a1, a2, vp.halfW, vp.halfH, cullMode, t, bbMin, bbMax)) continue;
        TriRec r;
        float rcpArea;
        edge_setup(t, vp.halfW, vp.halfH, bbMin, bbMax, make_rank(gMeshlet, prim, 1, vi), r, &rcpArea);
        r.pad = viewIndex;
        nRaster++;
        if (alpha) {
            AlphaExt x = alpha_ext(t, rcpArea, texcoord_word(mp, idxBytes[prim]), texcoord_word(mp, idxBytes[128 + prim]),
                                   texcoord_word(mp, idxBytes[256 + prim]), alphaMat | kTriAlpha);
            for (int k = 0; k < 3; k++) x.ru[k] = ru[k], x.rv[k] = rv[k];  // TriangleClipData, Rasterizer.cpp:455-458
            r.pad = viewIndex | kTriAlpha;
            if (!enqueue_alpha(r, x, a, chunk)) raster_serial_alpha(r, x, a.materials, vp.keys, vp.width);
            continue;
        }
        if (enqueue_big(r, a, chunk)) continue;
        if (a.counts) raster_serial_overdraw(r, vp.keys, a.counts, vp.width);
        else raster_serial(r, vp.keys, vp.width);
    }
}

// simd::gather_preload64's index mapping (preload64_index) of four packed index bytes: i < 32 stays, others
// read 32 + (i & 31).
__device__ __forceinline__ uint32_t preload64_index4(uint32_t w) {
    return (w & 0x1F1F1F1Fu) | ((w | (w >> 1) | (w >> 2)) & 0x20202020u);
}

// ------------------------------------------------------------------ kernels
// Per-warp shared memory: transformed vertices, index bytes, triangle records and the view. The alpha
// pass also keeps each small triangle's alpha terms.
struct WarpSmem {
    float2 xy[64];       // projected vertices: x/w, y/w (the face test reads these alone); then 32 live tiles
    uint2 pz[64];        // snapped position (packed as TrianglePacket's) and z/w
    uint32_t idx[96];    // index bytes, mapped by preload64_index4
    Padded<TriRec> tris[32];  // the padding holds the triangle's TileTest
    ViewParams view;
    uint8_t order[32];   // the lanes with small triangles, in order
    uint8_t code[64];    // vertex_code
    uint32_t live[128];  // the meshlet's triangles that survive the face test or need clipping: mapped
                         // index bytes 0-2, then the triangle, with bit 31 set if it needs clipping
    float zmax[32];      // each small triangle's depth bound (triangle_depth_bound)
};
struct WarpSmemAlpha : WarpSmem {
    float rw[64];        // 1/w of the vertices
    Padded<AlphaExt> exts[32];
};

// True if a meshlet of material mat goes to the alpha pass. Out of line: it is run once per 32 positions of
// scenes with alpha-tested materials, and inline it slowed draws without any (24 batched views: mesh stage
// 1281 us out of line, 1492 inline).
__device__ __noinline__ bool takes_alpha_pass(const DevMaterial* materials, uint32_t numMaterials, uint32_t mat, bool all) {
    if (mat == 0xFFFFFFFFu || mat >= numMaterials) return false;
    const DevMaterial& m = materials[mat];
    return (all ? material_alpha_tested_all(m) : material_alpha_tested(m)) && !material_alpha_passes(m);
}

// True if no triangle of a meshlet can change a pixel: its vertices (slots below `slots` of pz, all of them inside
// the view) lie in a box of tiles whose depth bounds are all above the nearest vertex (triangle_depth_bound of
// the meshlet). The alpha pass finds 41 to 46 % of its meshlets hidden by the opaque pass and by each other: 94 ->
// 77 us of a 1916x1036 frame from inside, 175 -> 144 us of a 1600x900 G-buffer. The box is read four rows of tiles
// at a time and left at the first rows that are not nearer, mostly the first ones: five meshlets that fill 1280x720
// 112.7 -> 100 us. Larger boxes are not tested. Alpha pass + the chunk stage after it, us, by the limit in tiles:
//                                               512          2048          8192          none
//   50,000 meshlets, inside, 1916x1036       71 + 229      57 + 211      54 + 197      55 + 191
//   30,000, G-buffer, 1600x900              127 + 171     112 + 157     111 + 132     111 + 131
//   18,960, outside, 836x688                 90 + 111      83 +  90      85 +  90      84 +  89
//   61,025, outside, 1188x1104               34 +  94      34 +  93      34 +  92      34 +  99
//    1,960, inside, 2516x1168                27 + 173      27 + 170      28 + 167      56 + 140
//   53,291, inside, 1160x1104                20 + 105      20 + 105      20 + 105      20 + 105
constexpr uint32_t kHiddenTiles = 8192;
__device__ __forceinline__ bool meshlet_hidden(const uint2* pz, uint32_t slots, const ViewParams& vp, int lane) {
    uint32_t lo = 0x7FFF7FFFu, hi = 0x80008000u, z = 0;
#pragma unroll
    for (int j = 0; j < 2; j++) {
        if (32 * j + lane < slots) {
            const uint2 q = pz[32 * j + lane];
            lo = __vmins2(lo, q.x), hi = __vmaxs2(hi, q.x), z = max(z, q.y);
        }
    }
    z = __reduce_max_sync(0xFFFFFFFFu, z);
    const int32_t x0 = __reduce_min_sync(0xFFFFFFFFu, (int32_t)(int16_t)(lo & 0xFFFF)), y0 = __reduce_min_sync(0xFFFFFFFFu, (int32_t)lo >> 16);
    const int32_t x1 = __reduce_max_sync(0xFFFFFFFFu, (int32_t)(int16_t)(hi & 0xFFFF)), y1 = __reduce_max_sync(0xFFFFFFFFu, (int32_t)hi >> 16);
    // render_bbox of the whole; a triangle's 32-bit add may carry 1 into y, which the 8 covers
    const int32_t tx0 = max(((x0 + 7) >> 4) + vp.halfW, 0) >> 2, ty0 = max(((y0 + 7) >> 4) + vp.halfH, 0) >> 2;
    const int32_t tx1 = (min(((x1 + 7) >> 4) + vp.halfW, 2 * vp.halfW) + 3) >> 2, ty1 = (min(((y1 + 8) >> 4) + vp.halfH, 2 * vp.halfH) + 3) >> 2;
    if (tx1 <= tx0 || ty1 <= ty0 || (uint32_t)((tx1 - tx0) * (ty1 - ty0)) > kHiddenTiles) return false;
    const int32_t tw = vp.width >> 2;
    const float zf = __uint_as_float(z), bound = fadd(zf, fmul(zf, 0x1p-16f));
    if ((int32_t)z < 0) return false;
    for (int32_t top = ty0; top < ty1; top += 4) {  // the first rows mostly tell that a meshlet is not hidden
        const int32_t y = top + (lane >> 3);
        uint32_t known = 0xFFFFFFFFu;
        for (int32_t x = tx0 + (lane & 7); x < tx1 && y < ty1; x += 8) known = min(known, vp.tileMin[y * tw + x]);
        if (!__all_sync(0xFFFFFFFFu, (__float_as_uint(bound) | 0x80000000u) < known)) return false;
    }
    return true;
}

// Mesh stage. A work item is one meshlet of one view: a single-view draw numbers its meshlets
// 0..count-1; a batched draw concatenates the meshlet ranges of its views (viewStart is their
// prefix), so one launch serves views of any size.
// Vis-buffer draws take two passes: the opaque pass draws every opaque meshlet and appends the
// work items of alpha-tested meshlets to alphaList; the alpha pass draws those with
// FS_EncodeSurfaceId<true>. The order of the passes does not change the keys. OverdrawShader draws
// take one pass over every meshlet.
// View of batched work position p: the largest v with viewStart[v] <= p.
__device__ __forceinline__ uint32_t view_of(const uint32_t* viewStart, uint32_t numViews, uint32_t p) {
    uint32_t lo = 0, hi = numViews - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (viewStart[mid] <= p) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// A block's pool of meshlets that a fetched group held beyond the one its warp draws next: any warp of the block
// takes them before it fetches another group, and a warp that gives takes until the pool is empty before it ends, so
// none is left. Where groups hold several visible meshlets some warps used to draw three or four in a row, 20,000 to
// 100,000 cycles each, while the median warp was done (at 0.27 of the kernel's time inside a 50k-meshlet scene, 0.35
// in a G-buffer draw of 30k): mesh stage 160 -> 124 us and 184 -> 142 us there, 234 -> 185 in a draw of 60k meshlets
// at 2560x1440, 357 -> 342 of 100k at 1920x1080, 1281 -> 1244 for 24 batched views (all but the first meshlet of a
// group given; all but three 1250, all but eight 1290).
constexpr uint32_t kPoolSlots = 64, kPoolFree = 0xFFFFFFFFu;
static_assert(SWR_MAX_MESHLETS <= 1u << 21, "a pool's word");
__device__ __forceinline__ uint32_t pool_take(uint32_t* pool, int lane) {
    const uint32_t s0 = ((volatile uint32_t*)pool)[lane], s1 = ((volatile uint32_t*)pool)[32 + lane];
    uint32_t taken = kPoolFree;
    for (unsigned any = __ballot_sync(0xFFFFFFFFu, s0 != kPoolFree || s1 != kPoolFree); any && taken == kPoolFree; any &= any - 1) {
        const int src = __ffs(any) - 1;
        if (lane == src) taken = atomicExch(&pool[s0 != kPoolFree ? lane : 32 + lane], kPoolFree);
        taken = __shfl_sync(0xFFFFFFFFu, taken, src);
    }
    return taken;
}
// Gives the lanes of mask but the first, as far as their slots are free; returns the lanes kept.
__device__ __forceinline__ unsigned pool_give(uint32_t* pool, unsigned mask, uint32_t item, int lane, int warp) {
    bool given = false;
    if (((mask & (mask - 1)) >> lane) & 1) {
        const uint32_t slot = (lane + 8 * warp) & (kPoolSlots - 1);
        given = atomicCAS(&pool[slot], kPoolFree, item) == kPoolFree || atomicCAS(&pool[slot ^ 32], kPoolFree, item) == kPoolFree;
    }
    return mask & ~__ballot_sync(0xFFFFFFFFu, given);
}

enum : int { kPassOpaque = 0, kPassAlpha = 1, kPassOverdraw = 2 };
// kShaded: the meshlets come shaded by a user mesh shader (a.shaded, swr_shaded_meshlet records):
// clip positions, indices, PrimCount, CullMode and FragmentShaderId are read from the record
// instead of ShadeMeshlet's transform of the Meshlet (whose texcoords and material the alpha test
// still reads).
// kSmall: a single-view draw of at most as many meshlets as the grid has warps. 2^a.partShift warps take a meshlet
// each, chosen by their index: all of them transform it and test its faces, and each draws its share of the
// triangles that are left. A warp alone is a serial chain (a step of four tiles takes 1,300 cycles): 60 meshlets at
// 252x140 56 -> 8.7 us (at most 8 warps a meshlet 13.8, 16 10.9), 1024 at 1280x720 66 -> 31 us, and with the
// tail gone fewer triangles are queued: chunk stage 39 -> 18 us. Two items a warp: 33 us.
template <int kPass, bool kShaded = false, bool kSmall = false>
__global__ void __launch_bounds__(512, 2) k_draw_meshlets(DrawArgs a) {
    constexpr bool kAlpha = kPass == kPassAlpha, kOver = kPass == kPassOverdraw;
    using Smem = typename std::conditional<kAlpha, WarpSmemAlpha, WarpSmem>::type;
    extern __shared__ __align__(16) unsigned char smemRaw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    Smem& S = ((Smem*)smemRaw)[warp];
    const uint8_t* idxBytes = (const uint8_t*)S.idx;
    Padded<TriRec>* tris = S.tris;
    uint4* const list = (uint4*)S.xy;  // live tiles being shaded (shade_live_tiles): the face test is done with xy then
    const ViewParams& vp = S.view;
    const uint32_t chunk = chunk_shape(a);
    const bool multi = a.views != nullptr;
    // Work positions. Position p of a view draws its meshlet draw_order(p) (order_stride); a batched
    // draw concatenates its views' positions, padded to multiples of kBatchGroup (viewStart); the
    // alpha pass walks its list of work items.
    const uint32_t totalItems = kAlpha ? (uint32_t)a.s.control[9] : (multi ? a.viewStart[a.numViews] : a.count);
    unsigned long long* const cursor = &a.s.control[kAlpha ? 10 : 0];
    unsigned long long* const idleWarps = &a.s.control[kAlpha ? 12 : 11];  // warps past their last item
    const uint32_t numWarps = gridDim.x * (blockDim.x >> 5);
    uint32_t curView = 0xFFFFFFFFu;
    if (!multi) {
        if (lane == 0) {
            ViewParams v = {};
            for (int k = 0; k < 16; k++) v.m[k] = a.m[k];
            v.halfW = a.halfW, v.halfH = a.halfH, v.width = a.width, v.height = a.height;
            v.bx = a.bx, v.by = a.by, v.meshletOffset = a.meshletOffset, v.count = a.count;
            v.keys = a.keys, v.tileMin = a.tileMin;
            S.view = v;
        }
        curView = 0;
        __syncwarp();
    }
    // per warp, within 32 bits: less than 2^21 meshlets x 128 in a view; thousands of warps share the less than 2^32
    // positions x 128 of a batch, whose blocks add theirs in 64 bits
    uint32_t nProcessed = 0, nRaster = 0, nClipped = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) a.s.control[8] = 0;  // the cursor of the chunk stage after this pass

    // Work items are fetched a group at a time: one contended atomic per group. A group's cull
    // bits are tested at once (one position per lane), then the warp walks the visible ones.
    // Batched draws, most of whose (view, meshlet) items are culled, fetch groups of 32. A work
    // item is viewStart[view] + m (m alone in single-view draws), as the alpha list records it.
    uint32_t laneMeshlet = 0;              // the meshlet of this lane's position in the group
    uint32_t fetchView = 0;                // batched draws: the view of the fetched group
    unsigned fetchMask = 0;                // lanes of the fetched group whose meshlet is visible
    // Single view: positions per fetch. A draw of fewer meshlets than groups for every warp starts with
    // smaller groups, so that no warp draws several meshlets in a row while others have none.
    const uint32_t leastGroup = totalItems < 2 * numWarps ? 1u : 2u;
    // Sparse: of 1024 positions sampled from the cull bitmap few are visible. Groups start at 32 then, so that the
    // warps' own first groups take 150,000 positions without a cursor (its contended atomics kept the warps from their
    // first meshlet for 25,000 cycles and more), and every triangle above kSpreadTiles tiles is queued, as no other
    // meshlets hide the few visible ones' serial steps: 213 of 150,000 visible, mesh stage 67.6 -> 42.7 us.
    // "Few" depends on the positions a warp has: where the first groups take them all, nothing balances the visible
    // ones between the blocks, and what is saved is soon lost; where most groups come from the cursor, it pays longer.
    // Whole draws at 1280x720 and 2560x1440, mean us, sparse / not, by meshlets and visible share:
    //             0.05 %      0.3 %       0.5 %       1 %         2 %         3 %
    //    20,000   66 /  71    86 /  85    91 /  89   112 /  98   137 / 112   139 / 122
    //   150,000   89 / 103   119 / 126   139 / 133   160 / 154   186 / 164   196 / 170
    //   220,000   90 / 107   121 / 134   134 / 144   155 / 159   191 / 174   198 / 191
    //   400,000  107 / 123   144 / 156   160 / 172   178 / 189   207 / 219   229 / 233
    uint32_t firstGroup = min(kDrawGroup, max(totalItems / numWarps, leastGroup));
    bool sparse = false;
    if (!kSmall && !kAlpha && !multi && a.cullBitmap && totalItems >= 1024) {
        const unsigned long long words = totalItems >> 4;
        unsigned seen = 0;
        for (uint32_t k = 2 * lane; k < 2u * lane + 2; k++) seen += __popc(a.cullBitmap[(uint32_t)((words * k) >> 6)]);
        const unsigned few = totalItems > 64 * numWarps ? 32u : totalItems > 40 * numWarps ? 12u : 4u;
        sparse = __reduce_add_sync(0xFFFFFFFFu, seen) < few;
        if (sparse) firstGroup = 32;
    }
    uint32_t fetchGroup = firstGroup;
    // Single-view draws walk their positions twice: meshlets large on screen first, then the rest
    // (a second cursor, control[7]), so the costliest work items start early and the last ones
    // are small: a cheaper tail, and near geometry raises the tile depth bounds before the far.
    const bool twoPass = !multi && !kAlpha && !kShaded;
    uint32_t pass = twoPass ? 0u : 1u;
    // 2^partShift warps share a meshlet: small draws, and an alpha pass of few meshlets for its warps (a G-buffer draw's
    // 10,000 by two: 143 -> 128 us; by four 128, and 7,200 of another 84 instead of 72 us).
    constexpr bool kParts = kSmall || kAlpha;
    const uint32_t partShift = kSmall ? a.partShift : kAlpha ? (totalItems < numWarps ? 2u : totalItems < 4 * numWarps ? 1u : 0u) : 0u;
    // A pass's first group is the warp's own, later ones come from the cursor, where those first groups take at most a
    // quarter of the positions (or the draw is sparse; the overdraw shader's pass gains by it at any size). In smaller
    // draws all come from the cursor: own groups of 4 hand out 20,000 positions at once, and the warps with costly
    // ones end last (20,000 meshlets at 64x36 84 us with own groups, 68 without, 16x8 80 and 62, 320x180 125 and 113;
    // 50,000 at 64x36 116 and 106; 60,000 at 2560x1440 860 and 837 of a frame; 100,000 at 1920x1080 618 and 623).
    const bool ownFirst = kAlpha || kOver || sparse || totalItems >= 4 * numWarps * firstGroup;
    bool ownTaken = !ownFirst;
    // Opaque pass of a scene with alpha-tested materials: a fetched group's alpha-tested meshlets go to the
    // alpha pass's list with one atomic, before their records are read (a draw of alpha-tested meshlets alone:
    // 45 -> 27 us). A shaded meshlet's FragmentShaderId is only known from its record, and is looked at
    // later. Returns the lanes left to draw.
    constexpr bool kSplitAlpha = kPass == kPassOpaque && !kShaded;
    auto split_alpha = [&](unsigned mask, uint32_t meshlet, uint32_t item) -> unsigned {
        bool alpha = false;
        if ((mask >> lane) & 1) {
            const uint32_t mat = *(const uint32_t*)(a.meshlets + (size_t)meshlet * kMeshletSize + kOffMaterialId);
            alpha = takes_alpha_pass(a.materials, a.numMaterials, mat, a.alphaAll != 0);
        }
        const unsigned am = __ballot_sync(0xFFFFFFFFu, alpha);
        if (am == 0) return mask;
        uint32_t at = 0;
        if (lane == 0) at = (uint32_t)atomicAdd(&a.s.control[9], (unsigned long long)__popc(am));
        at = __shfl_sync(0xFFFFFFFFu, at, 0);
        if (alpha) a.s.alphaList[at + __popc(am & ((1u << lane) - 1u))] = item;
        return mask & ~am;
    };
    constexpr bool kPool = !kAlpha && !kSmall && !kOver;  // (the overdraw shader's pass loses by it, 159 -> 169 us)
    __shared__ uint32_t pool[kPool ? kPoolSlots : 1];
    __shared__ unsigned long long blockSums[kPool ? 4 : 1];  // the warps' counters, and how many have added theirs
    if constexpr (kPool) {
        if (threadIdx.x < 4) blockSums[threadIdx.x] = 0;
        for (uint32_t k = threadIdx.x; k < kPoolSlots; k += blockDim.x) pool[k] = kPoolFree;
        __syncthreads();
    }
    uint32_t nextItem = warp * gridDim.x + blockIdx.x;  // kSmall: blocks first, so that all SMs get some
    while (true) {
        uint32_t m, view = 0, item, part = 0;
        if constexpr (kSmall) {
            if (nextItem >= totalItems << partShift) break;
            m = item = nextItem >> partShift, part = nextItem & ((1u << partShift) - 1u);
            nextItem += numWarps;
            if (a.cullBitmap && !((a.cullBitmap[m >> 4] >> (m & 15)) & 1)) continue;
            if (a.s.alphaList) {
                const uint32_t mat = *(const uint32_t*)(a.meshlets + (size_t)(a.meshletOffset + m) * kMeshletSize + kOffMaterialId);
                if (takes_alpha_pass(a.materials, a.numMaterials, mat, a.alphaAll != 0)) {
                    if (part == 0 && lane == 0) a.s.alphaList[atomicAdd(&a.s.control[9], 1ull)] = item;
                    continue;
                }
            }
        } else if constexpr (kAlpha) {
            // one item per atomic: alpha-tested meshlets are few and costly (taken four at a time, 12,600 of them
            // left most warps with none: 525 -> 306 us)
            uint32_t idx = warp * gridDim.x + blockIdx.x;  // the first by the warp's index
            if (ownTaken) {
                if (lane == 0) idx = numWarps + (uint32_t)atomicAdd(cursor, 1ull);
                idx = __shfl_sync(0xFFFFFFFFu, idx, 0);
            }
            ownTaken = true;
            if (idx >= totalItems << partShift) break;
            part = idx & ((1u << partShift) - 1u);
            item = a.s.alphaList[idx >> partShift];
            m = item;
            if (multi) {
                view = view_of(a.viewStart, a.numViews, item);
                m = item - a.viewStart[view];
            }
        } else {
            if (multi) {
                uint32_t taken = kPoolFree;
                if (kPool && fetchMask == 0) {
                    taken = pool_take(pool, lane);
                }
                if (taken == kPoolFree && fetchMask == 0) {
                    uint32_t b = 0;
                    if (lane == 0) b = (uint32_t)atomicAdd(cursor, (unsigned long long)kBatchGroup);
                    const uint32_t base = __shfl_sync(0xFFFFFFFFu, b, 0);
                    if (base >= totalItems) break;
                    // groups interleave the views: group G is group G / numViews of view G % numViews
                    const uint32_t G = base / kBatchGroup;
                    fetchView = G % a.numViews;
                    const ViewParams& fv = a.views[fetchView];
                    // the cull wrote the group's 32 results as one word, in draw order
                    const uint32_t g = G / a.numViews, q = g * kBatchGroup + lane;
                    const uint32_t n = fv.count - g * kBatchGroup;  // positions of the group in the view (> 0)
                    const unsigned inView = n >= 32 ? 0xFFFFFFFFu : (1u << n) - 1u;
                    fetchMask = (fv.groupMasks ? fv.groupMasks[g] : 0xFFFFFFFFu) & inView;
                    if (fetchMask == 0) continue;
                    laneMeshlet = q < fv.count ? draw_order(q, fv.count, fv.orderStride) : 0u;
                    if (kSplitAlpha && a.s.alphaList) {
                        fetchMask = split_alpha(fetchMask, fv.meshletOffset + laneMeshlet, a.viewStart[fetchView] + laneMeshlet);
                        if (fetchMask == 0) continue;
                    }
                    // as a pool's word holds a view of up to 2046 and a meshlet
                    if (kPool && a.numViews < 2047) fetchMask = pool_give(pool, fetchMask, fetchView << 21 | laneMeshlet, lane, warp);
                }
                if (taken != kPoolFree) {
                    view = taken >> 21, m = taken & 0x1FFFFFu;
                } else {
                    view = fetchView;
                    m = __shfl_sync(0xFFFFFFFFu, laneMeshlet, __ffs(fetchMask) - 1);
                    fetchMask &= fetchMask - 1;
                }
                item = a.viewStart[view] + m;
            } else {
                // Single view: groups of fetchGroup positions (2 to 32), their cull bits tested at
                // once (one position per lane). The group grows while groups come back empty (a
                // sparse view fetches 32 positions per atomic) and shrinks while they hold more than
                // one visible meshlet (a dense view fetches about one visible meshlet at a time, so
                // the last work items spread evenly over the warps).
                uint32_t taken = kPoolFree;
                if (kPool && fetchMask == 0) {
                    taken = pool_take(pool, lane);
                }
                if (taken == kPoolFree && fetchMask == 0) {
                    uint32_t b = 0;
                    if (!ownTaken) {
                        b = (warp * gridDim.x + blockIdx.x) * firstGroup;
                        ownTaken = true;
                    } else if (lane == 0) {
                        b = (ownFirst ? numWarps * firstGroup : 0u) +
                            (uint32_t)atomicAdd(twoPass && pass == 1 ? &a.s.control[7] : cursor, (unsigned long long)fetchGroup);
                    }
                    const uint32_t base = __shfl_sync(0xFFFFFFFFu, b, 0);
                    if (base >= totalItems) {
                        if (pass == 0) {  // the large meshlets are all taken: the rest from position 0
                            pass = 1, fetchGroup = firstGroup, ownTaken = !ownFirst;
                            continue;
                        }
                        break;
                    }
                    const uint32_t q = base + lane;
                    bool vis = false;
                    if (lane < fetchGroup && q < totalItems) {
                        laneMeshlet = draw_order(q, a.count, a.orderStride);
                        vis = a.cullBitmap == nullptr || ((a.cullBitmap[laneMeshlet >> 4] >> (laneMeshlet & 15)) & 1);
                        if (vis && twoPass) {  // bounding sphere radius against the clip w of its centre
                            const float4 sp = *(const float4*)(a.meshlets + (size_t)(a.meshletOffset + laneMeshlet) * kMeshletSize);
                            const float w = fmaf(sp.x, a.m[3], fmaf(sp.y, a.m[7], fmaf(sp.z, a.m[11], a.m[15])));
                            vis = (sp.w > kLargeMeshlet * w) == (pass == 0);
                        }
                    }
                    fetchMask = __ballot_sync(0xFFFFFFFFu, vis);
                    if (kSplitAlpha && a.s.alphaList) fetchMask = split_alpha(fetchMask, a.meshletOffset + laneMeshlet, laneMeshlet);
                    const int got = __popc(fetchMask);
                    fetchGroup = got == 0 ? min(fetchGroup * 2, 32u) : (got > 1 ? max(fetchGroup / 2, leastGroup) : fetchGroup);
                    if (fetchMask == 0) continue;
                    if constexpr (kPool) fetchMask = pool_give(pool, fetchMask, laneMeshlet, lane, warp);
                }
                if (taken != kPoolFree) {
                    m = taken;
                } else {
                    m = __shfl_sync(0xFFFFFFFFu, laneMeshlet, __ffs(fetchMask) - 1);
                    fetchMask &= fetchMask - 1;
                }
                item = m;
            }
        }
        if (multi && view != curView) {
            __syncwarp();
            ((uint32_t*)&S.view)[lane] = ((const uint32_t*)&a.views[view])[lane];
            __syncwarp();
            curView = view;
        }
        // (the fetch skipped meshlets whose cull bit is clear, Shading.cpp:282-289; the alpha list
        // holds visible ones only)

        const uint32_t g = vp.meshletOffset + m;
        const uint8_t* mp = a.meshlets + (size_t)g * kMeshletSize;
        // The record's positions (all 64 slots) and index bytes are loaded together with its header,
        // not after it: one memory round trip per meshlet instead of two.
        const uint8_t* sp = kShaded ? a.shaded + (size_t)m * kShadedSize : nullptr;
        const float* P = (const float*)(kShaded ? sp + kShadedPositions : mp + kOffPositions);
        const float px0 = P[lane], py0 = P[64 + lane], pz0 = P[128 + lane];
        const float px1 = P[32 + lane], py1 = P[96 + lane], pz1 = P[160 + lane];
        float pw0 = 1.0f, pw1 = 1.0f;
        if constexpr (kShaded) pw0 = P[192 + lane], pw1 = P[224 + lane];
        const uint32_t* I = (const uint32_t*)(kShaded ? sp + kShadedIndices : mp + kOffIndices);
        const uint8_t* rawIdx = (const uint8_t*)I;  // the record's index bytes (the texcoords' are not mapped)
        const uint32_t ix0 = I[lane], ix1 = I[32 + lane], ix2 = I[64 + lane];
        const uint32_t hdr = *(const uint32_t*)(kShaded ? sp : mp + kOffNumVertices);
        const uint32_t matId = *(const uint32_t*)(mp + kOffMaterialId);
        // record arrays hold 64 / 128; a shaded meshlet defines all 64 vertex slots
        const uint32_t nv = kShaded ? 64u : hdr & 0xFF, nt = min((kShaded ? hdr : hdr >> 8) & 0xFF, 128u);
        int cullMode = kCullFrontCCW;
        bool alphaTested = false;  // FragmentShaderId 1
        if (matId != 0xFFFFFFFFu && matId < a.numMaterials) {  // Shading.cpp:302-306
            const DevMaterial& mt = a.materials[matId];
            cullMode = mt.is_double_sided ? kCullNone : kCullFrontCCW;
            alphaTested = a.alphaAll ? material_alpha_tested_all(mt) : material_alpha_tested(mt);
            if constexpr (kShaded) alphaTested = alphaTested && ((hdr >> 16) & 0xFF) == 1;
        }
        if constexpr (kShaded) cullMode = (int)((hdr >> 8) & 0xFF);
        if (kPass == kPassOpaque && kShaded && alphaTested) {  // drawn by the alpha pass
            if (lane == 0) a.s.alphaList[atomicAdd(&a.s.control[9], 1ull)] = item;
            continue;
        }
        if (nt == 0) continue;
        if (!kParts || part == 0) nProcessed += nt;

        // ShadeMeshlet vertex loop (Shading.cpp:295-298): 16-vertex chunks up to NumVertices; the
        // slots past them are zero. What the triangles need of a vertex alone is computed here, once
        // instead of in about six triangles: the projection, the snapped position and the clip codes.
        // The stage is bound by instruction issue (68 % of the slots, 263 M instructions in the 1080p frame
        // of 100k meshlets): with the positions snapped per vertex, packed index bytes, the clip codes
        // skipped for a meshlet inside the view and the tile owners found by ballots, 379 -> 355 us there,
        // 24 batched views 1.44 -> 1.31 ms.
        const uint32_t nvr = min((nv + 15) & ~15u, 64u);
        const float fsx = (float)(vp.halfW * 16), fsy = (float)(vp.halfH * 16);
        auto xform = [&](uint32_t v, float x, float y, float z, float w) {
            const float4 c = kShaded ? make_float4(x, y, z, w) : clip_position(x, y, z, v < nvr, vp);
            const Ndc n = project(c.x, c.y, c.z, c.w);
            S.xy[v] = make_float2(n.x, n.y);
            const uint32_t pos = ((uint32_t)round2i(fmul(n.x, fsx)) & 0xFFFF) | ((uint32_t)round2i(fmul(n.y, fsy)) << 16);
            S.pz[v] = make_uint2(pos, __float_as_uint(n.z));
            if constexpr (kAlpha) S.rw[v] = n.rw;
            const uint32_t code = vertex_code(c, vp.bx, vp.by);
            S.code[v] = (uint8_t)code;
            return code == kCodeInBand;
        };
        const bool in0 = xform(lane, px0, py0, pz0, pw0), in1 = xform(32 + lane, px1, py1, pz1, pw1);
        const uint32_t mx0 = preload64_index4(ix0), mx1 = preload64_index4(ix1), mx2 = preload64_index4(ix2);
        S.idx[lane] = mx0, S.idx[32 + lane] = mx1, S.idx[64 + lane] = mx2;
        // vertex slots that count: all, or (alpha pass) the meshlet's vertices if its triangles use no others
        uint32_t slots = 64;
        if (kAlpha && nv < 64) {
            const uint32_t first = 4 * lane, used = first >= nt ? 0u : 0xFFFFFFFFu >> (8 * (4 - min(nt - first, 4u)));
            const uint32_t past = (__vcmpgeu4(mx0, nv * 0x01010101u) | __vcmpgeu4(mx1, nv * 0x01010101u) | __vcmpgeu4(mx2, nv * 0x01010101u)) & used;
            if (!__any_sync(0xFFFFFFFFu, past != 0)) slots = nv;
        }
        // every such vertex inside the viewport and the depth range: every triangle is trivially accepted
        const bool allInside = __all_sync(0xFFFFFFFFu, (in0 || (kAlpha && lane >= slots)) && (in1 || (kAlpha && 32 + lane >= slots)));
        __syncwarp();

        // About half of a closed meshlet's triangles face away. The face test runs first for all of
        // them and compacts the rest into S.live, so the setup and binning below run on full
        // 32-triangle steps. Each triangle keeps its index p (its rank), so the keys do not change.
        // Alpha pass: a meshlet behind what is drawn is only counted (its box of tiles takes fewer instructions than
        // its triangles). The opaque pass, where a smaller part is hidden, loses by the test: 354 -> 364 us at
        // 1080p, 1.27 -> 1.38 ms for 24 batched views.
        const bool hidden = kAlpha && allInside && vp.tileMin && meshlet_hidden(S.pz, slots, vp, lane);
        uint32_t nLive = 0;
        for (uint32_t base = 0; base < nt; base += 32) {
            const uint32_t p = base + lane;
            const uint32_t i0 = idxBytes[p], i1 = idxBytes[128 + p], i2 = idxBytes[256 + p];
            bool accepted = p < nt, clip = false;
            if (!allInside) {  // Clipper::ComputeClipCodes (Rasterizer.cpp:353-397) from the vertices' codes
                const uint32_t c0 = S.code[i0], c1 = S.code[i1], c2 = S.code[i2];
                const uint32_t partial = (c0 | c1 | c2) & 0x3Fu, combined = c0 & c1 & c2 & 0x3Fu;
                const bool trivial = (c0 & c1 & c2 & kCodeInBand) != 0 && !(partial & 0x30u);
                const bool accept = accepted && combined == 0, nontriv = accept && !trivial;
                if (a.countClipped && (!kParts || part == 0)) nClipped += __popc(__ballot_sync(0xFFFFFFFFu, nontriv)) * (lane == 0);
                clip = nontriv && a.clipMode;
                accepted = accept && trivial;
            }
            const float2 q0 = S.xy[i0], q1 = S.xy[i1], q2 = S.xy[i2];
            const bool live = clip || (accepted && front_facing({ q0.x, q0.y, 0.0f, 0.0f }, { q1.x, q1.y, 0.0f, 0.0f },
                                                                { q2.x, q2.y, 0.0f, 0.0f }, cullMode));
            const unsigned liveMask = __ballot_sync(0xFFFFFFFFu, live);
            if (kAlpha && hidden) {  // counted alone: the warp's share, as another warp of the meshlet may not find it hidden
                const uint32_t at = nLive + __popc(liveMask & ((1u << lane) - 1u));
                nLive += __popc(liveMask);
                if (live && (at & ((1u << partShift) - 1u)) == part) {
                    Setup t;
                    t.Pos0 = S.pz[i0].x, t.Pos1 = S.pz[i1].x, t.Pos2 = S.pz[i2].x;
                    uint32_t bbMin, bbMax;
                    render_bbox(t, vp.halfW, vp.halfH, bbMin, bbMax);
                    nRaster += lo16(bbMin) < lo16(bbMax) && hi16(bbMin) < hi16(bbMax);
                }
                continue;
            }
            if (live) S.live[nLive + __popc(liveMask & ((1u << lane) - 1u))] = i0 | (i1 << 8) | (i2 << 16) | (p << 24) | (clip ? 0x80000000u : 0u);
            nLive += __popc(liveMask);
        }
        __syncwarp();

        if (kAlpha && hidden) continue;
        const uint32_t nMine = kParts ? (nLive + (1u << partShift) - 1u - part) >> partShift : nLive;
        for (uint32_t base = 0; base < nMine; base += 32) {
            const bool valid = base + lane < nMine;
            const uint32_t e = valid ? S.live[kParts ? ((base + lane) << partShift) + part : base + lane] : 0u;
            const uint32_t i0 = e & 0xFF, i1 = (e >> 8) & 0xFF, i2 = (e >> 16) & 0xFF, p = (e >> 24) & 127u;
            const bool accepted = valid && !(e & 0x80000000u), clipped = valid && (e & 0x80000000u);

            int myTiles = 0;     // tiles of this lane's small triangle (0 if none)
            bool queue = false;  // this lane's triangle goes to the chunk queue
            if (accepted) {  // trivially accepted and front-facing (the first pass's face test)
                const uint2 v0 = S.pz[i0], v1 = S.pz[i1], v2 = S.pz[i2];
                Setup t;
                t.Pos0 = v0.x, t.Pos1 = v1.x, t.Pos2 = v2.x;
                t.Z0 = __uint_as_float(v0.y), t.Z1 = __uint_as_float(v1.y), t.Z2 = __uint_as_float(v2.y);
                if constexpr (kAlpha) t.W0 = S.rw[i0], t.W1 = S.rw[i1], t.W2 = S.rw[i2];
                uint32_t bbMin, bbMax;
                render_bbox(t, vp.halfW, vp.halfH, bbMin, bbMax);
                if (lo16(bbMin) < lo16(bbMax) && hi16(bbMin) < hi16(bbMax)) {
                    TriRec r;
                    float rcpArea;
                    const int32_t det = edge_setup(t, vp.halfW, vp.halfH, bbMin, bbMax, make_rank(g, p, 0, 0), r, &rcpArea);
                    nRaster++;
                    AlphaExt x;
                    if constexpr (kAlpha)
                        x = alpha_ext(t, rcpArea, texcoord_word(mp, rawIdx[p]), texcoord_word(mp, rawIdx[128 + p]),
                                      texcoord_word(mp, rawIdx[256 + p]), matId);
                    const int tilesX = ((bbMax & 0xFFFF) - (bbMin & 0xFFFF)) >> 2;
                    const int tilesY = ((bbMax >> 16) - (bbMin >> 16)) >> 2;
                    TinyBox tb;
                    if (kPass == kPassOpaque && det > 0 && tiny_box(t, vp.halfW, vp.halfH, bbMin, bbMax, tb)) {
                        shade_tiny(r, tb, vp.keys, vp.width);
                    } else if (tilesX * tilesY <= kSmallTiles) {
                        // tile index -> row by a multiply-shift (exact for tile < 16, tilesX <= 16), and
                        // whether the shading reads the keys before its atomics (keyReadTiles)
                        r.pad = (uint32_t)tilesX | (row_magic(tilesX) << 8) |
                                (a.keyReadTiles == 0 || (uint32_t)(tilesX * tilesY) <= a.keyReadTiles ? kPadReadKey : 0u);
                        tris[lane].v = r;
                        *(TileTest*)&tris[lane].pad = tile_test(r);
                        if constexpr (kAlpha) S.exts[lane].v = x;
                        myTiles = tilesX * tilesY;
                        S.zmax[lane] = triangle_depth_bound(t);
                    } else {
                        r.pad = kAlpha ? view | kTriAlpha : view;
                        tris[lane].v = r;
                        if constexpr (kAlpha) S.exts[lane].v = x;
                        queue = true;
                    }
                }
            }
            if (clipped) {  // rare: the clip-space vertices are transformed again
                const uint32_t partial = (S.code[i0] | S.code[i1] | S.code[i2]) & 0x3Fu;
                auto clip_vertex = [&](uint32_t v) {
                    const float4 c = kShaded ? make_float4(P[v], P[64 + v], P[128 + v], P[192 + v])
                                             : clip_position(P[v], P[64 + v], P[128 + v], v < nvr, vp);
                    return Vtx{ c.x, c.y, c.z, c.w };
                };
                clip_and_queue(clip_vertex(i0), clip_vertex(i1), clip_vertex(i2), partial, a, vp, view, chunk, cullMode, g, p,
                               nRaster, kAlpha ? matId : ~0u, mp, rawIdx);
            }
            __syncwarp();

            // Once half of the warps have run out of work items, the warps still busy are the
            // kernel's tail (in a sparse frame, a few visible meshlets are all of it). A packet whose
            // small triangles cover more than kPacketTiles tiles would then keep this warp busy for
            // many steps while the others idle: its triangles of more than kSpreadTiles tiles go to
            // the queue, whose chunks spread over all warps of the chunk stage. (Sparser budgets, or
            // a second level once 90 % of the warps are idle, cost the dense frame more than they
            // gain in the sparse one.)
            bool spread = sparse;
            if (!spread && __reduce_add_sync(0xFFFFFFFFu, (unsigned)myTiles) > (kAlpha ? kPacketTilesAlpha : kPacketTiles)) {
                unsigned long long idle = 0;
                if (lane == 0) idle = *(volatile unsigned long long*)idleWarps;
                spread = __shfl_sync(0xFFFFFFFFu, idle, 0) * 2 >= numWarps;
            }
            if (spread && myTiles > kSpreadTiles) {
                tris[lane].v.pad = kAlpha ? view | kTriAlpha : view;
                myTiles = 0;
                queue = true;
            }
            const AlphaExt* ext = nullptr;
            if constexpr (kAlpha) ext = &S.exts[lane].v;
            if (!enqueue_warp<kAlpha>(queue, tris[lane].v, ext, a, chunk, lane)) {
                // The full queue turned it away: its tiles join the warp's list, however many they are. (With a second
                // copy of the tile loop for it the batched mesh stage took 1281 us instead of 1276.)
                TriRec& r = tris[lane].v;
                myTiles = (int)triangle_tiles(r);
                r.pad = kPadWide | kPadReadKey;
                *(TileTest*)&tris[lane].pad = tile_test(r);
                S.zmax[lane] = __int_as_float(0x7F800000);
            }

            // Small triangles: the warp walks the concatenated tile lists of all of them, four
            // tiles (64 pixels) per step, so tiny triangles share steps.
            int incl = myTiles;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                int v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= o) incl += v;
            }
            const int excl = incl - myTiles;
            const int total = __shfl_sync(0xFFFFFFFFu, incl, 31);
            const unsigned owners = __ballot_sync(0xFFFFFFFFu, myTiles > 0);
            if (myTiles > 0) S.order[__popc(owners & ((1u << lane) - 1u))] = (uint8_t)lane;
            __syncwarp();
            // 32 tiles at a time: lane j tests tile b + j of the list (empty or hidden tiles are
            // dropped), then the live ones are shaded four per step.
            const uint32_t tw = vp.width >> 2;
            for (int b = 0; b < total; b += 32) {
                const int t = b + lane;
                // tile t's owner: the last triangle whose list starts at or before it
                const bool starts = myTiles > 0 && (uint32_t)(excl - b) < 32u;
                const unsigned startMask = __reduce_or_sync(0xFFFFFFFFu, starts ? 1u << (excl - b) : 0u);
                const int before = __popc(__ballot_sync(0xFFFFFFFFu, myTiles > 0 && excl < b));
                const uint32_t own = t < total ? S.order[before + __popc(startMask & (0xFFFFFFFFu >> (31 - lane))) - 1] : 0u;
                const int ownerExcl = __shfl_sync(0xFFFFFFFFu, excl, own);
                bool live = false;
                uint32_t tpx = 0, tpy = 0, tmin = 0;
                if (t < total) {
                    const TriRec& r = tris[own].v;
                    const int tile = t - ownerExcl;
                    int tilesX = r.pad & 0xFF, ty = (tile * (int)((r.pad >> 8) & 0x1FF)) >> 8;
                    if (r.pad & kPadWide) {
                        tilesX = (int)(((r.bbMax & 0xFFFF) - (r.bbMin & 0xFFFF)) >> 2);
                        ty = tile / tilesX;
                    }
                    const int tx = tile - ty * tilesX;
                    tpx = (r.bbMin & 0xFFFF) + tx * 4, tpy = (r.bbMin >> 16) + ty * 4;
                    live = tile_live(r, *(const TileTest*)&tris[own].pad, tpx, tpy, vp.tileMin, tw, &tmin, S.zmax[own]);
                }
                const unsigned liveMask = __ballot_sync(0xFFFFFFFFu, live);
                if constexpr (kAlpha) {
                    const DevMaterial& mt = a.materials[matId];
                    shade_live_tiles_alpha([&](uint32_t q) -> const TriRec& { return tris[q].v; },
                                           [&](uint32_t q) -> const AlphaExt& { return S.exts[q].v; }, own, mt.tex,
                                           mt.alpha_cutoff, liveMask, tpx, tpy, tmin, vp.keys, vp.tileMin, vp.width,
                                           lane, list);
                } else if constexpr (kOver) {
                    shade_live_tiles_overdraw([&](uint32_t q) -> const TriRec& { return tris[q].v; }, own, liveMask, tpx, tpy,
                                              vp.keys, a.counts, vp.width, lane, list);
                } else {
                    shade_live_tiles([&](uint32_t q) -> const TriRec& { return tris[q].v; },
                                     [&](uint32_t q) { return (tris[q].v.pad & kPadReadKey) != 0u; }, own, liveMask, tpx, tpy,
                                     tmin, vp.keys, vp.tileMin, vp.width, lane, list);
                }
            }
            __syncwarp();
        }
        __syncwarp();
    }
    // perf counters (Rasterizer.h:366-370)
    nRaster = __reduce_add_sync(0xFFFFFFFFu, nRaster);
    if (lane == 0) {
        atomicAdd(idleWarps, 1ull);
        if constexpr (!kPool) {
            if (nProcessed) atomicAdd(&a.s.control[3], (unsigned long long)nProcessed);
            if (nRaster) atomicAdd(&a.s.control[4], (unsigned long long)nRaster);
            if (nClipped) atomicAdd(&a.s.control[5], (unsigned long long)nClipped);
        } else {
            // one addition a block, by its last warp: the words share a line, which takes one at a time (1080p mesh
            // stage 340 -> 333 us)
            if (nProcessed) atomicAdd(&blockSums[0], (unsigned long long)nProcessed);
            if (nRaster) atomicAdd(&blockSums[1], (unsigned long long)nRaster);
            if (nClipped) atomicAdd(&blockSums[2], (unsigned long long)nClipped);
            __threadfence_block();
            if (atomicAdd(&blockSums[3], 1ull) == (blockDim.x >> 5) - 1) {
                __threadfence_block();
                const volatile unsigned long long* sums = blockSums;
                for (int k = 0; k < 3; k++)
                    if (const unsigned long long n = sums[k]) atomicAdd(&a.s.control[3 + k], n);
            }
        }
    }
}

// Chunk stage: warps take runs of up to kChunkRun consecutive chunks (chunk_shape: w x h tiles) of the queued
// triangles from a global cursor (control[8], zeroed by the mesh stage), locate the run's first
// chunk by a 32-way search over the queue's chunk prefix, test the run's chunks one per lane
// (chunk_live) and rasterize the surviving ones together. A queued triangle carries its view in pad
// (batched draws) or belongs to the single view; an alpha-tested one (kTriAlpha) has its AlphaExt in the
// next slot, which owns no chunks and is never selected.
//
// The stage is bound by instruction issue, and most of what it is given is hidden or empty: in the
// 1080p frame of 100k meshlets 758k chunks of 24 M tiles hold 0.73 M live tiles, and 93 % of the chunks
// none. A warp that tested each chunk's tiles spent about 340 instructions on such a chunk; a lane's
// test shares its instructions with the run's others: chunk stage 279 -> 158 us (133 M instructions
// instead of 293 M), 629 -> 466 us in an alpha-tested frame from inside the scene. Runs of 4, 16 and 32
// chunks: 198, 184 and 193 us (the queue starts with near geometry, whose chunks survive together, so long
// runs leave some warps with all of it; in the alpha-tested frame 385, 685 and 867 us).
// With alpha-tested materials runs of 4: their live chunks cost about five times more (2, 4 and 8: 405, 363 and
// 432 us of chunk stage inside a 50k-meshlet scene).
constexpr uint32_t kChunkRun = 8, kChunkRunAlpha = 4;
// A shorter run when the queue holds fewer chunks than this many runs a warp, but two chunks while it holds one run a
// warp of them: the queue's first chunks, those of the nearest triangles, cost the most (runs by 4 / 6 / 8 a warp:
// 142 / 137 / 123 us of opaque chunk stage inside a 50k-meshlet scene; one chunk a run instead of two 93 against
// 80 us in a sparse 2560x1440 draw, by the cursor's atomics).
constexpr uint32_t kRunsPerWarp = 8;

// Per 32x32-pixel block, a lower bound of the tile depth bounds inside it, in the words after the tile
// bounds (tile_blocks): one load tells a chunk's lane that the whole block is nearer. The bounds are
// only refreshed where they proved too loose: a chunk that passed them and then had no live tile raises
// the blocks it touches to the minimum of their 64 tiles (tile bounds only grow, so a stale block
// bound stays a bound).
__device__ __forceinline__ void refresh_blocks(uint32_t x0, uint32_t y0, uint32_t x1, uint32_t y1, uint32_t* tileMin,
                                               uint32_t width, uint32_t height, int lane) {
    const uint32_t tw = width >> 2, th = height >> 2, bw = (width + 31) >> 5;
    uint32_t* blockMin = tileMin + tw * th;
    for (uint32_t by = y0 >> 5; by <= (y1 - 1) >> 5; by++)
        for (uint32_t bx = x0 >> 5; bx <= (x1 - 1) >> 5; bx++) {
            const uint32_t tx = bx * 8 + (lane & 7), ty = by * 8 + (lane >> 3);
            uint32_t m = 0xFFFFFFFFu;
            if (tx < tw && ty < th) m = tileMin[ty * tw + tx];
            if (tx < tw && ty + 4 < th) m = min(m, tileMin[(ty + 4) * tw + tx]);
            m = __reduce_min_sync(0xFFFFFFFFu, m);
            if (lane == 0 && m > blockMin[by * bw + bx]) atomicMax(&blockMin[by * bw + bx], m);
        }
}

// False if no sample of r in [x0, x1) x [y0, y1) can pass its edges or beat the depth bounds of the blocks
// there (tileMin null: edges alone). The depth bound is the smaller of the plane's maximum over the
// rectangle (tile_test's argument with the rectangle's size in place of the tile's) and the
// triangle's own maximum: the three edge values sum to the same E = E0 + E1 + E2 everywhere, so where all
// are >= 0, e1 + e2 <= E and no depth exceeds Z0 + max(0, Z10 E, Z20 E) by more than the roundings,
// 2^-16 of the terms' magnitudes being kept. (E is det / 16 up to the floors, except where a guard-band
// triangle's edge values wrapped.) A NaN bound counts as above every depth.
__device__ __forceinline__ bool chunk_live(const TriRec& r, uint32_t x0, uint32_t y0, uint32_t x1, uint32_t y1,
                                           const uint32_t* tileMin, uint32_t width, uint32_t height) {
    const int32_t w = (int32_t)(x1 - x0) - 1, h = (int32_t)(y1 - y0) - 1;
    const uint32_t e0 = (uint32_t)r.E0 + (uint32_t)r.A12 * x0 + (uint32_t)r.B12 * y0;
    const uint32_t e1 = (uint32_t)r.E1 + (uint32_t)r.A20 * x0 + (uint32_t)r.B20 * y0;
    const uint32_t e2 = (uint32_t)r.E2 + (uint32_t)r.A01 * x0 + (uint32_t)r.B01 * y0;
    const int32_t f0 = (int32_t)(e0 + (uint32_t)(max(r.A12, 0) * w + max(r.B12, 0) * h));
    const int32_t f1 = (int32_t)(e1 + (uint32_t)(max(r.A20, 0) * w + max(r.B20, 0) * h));
    const int32_t f2 = (int32_t)(e2 + (uint32_t)(max(r.A01, 0) * w + max(r.B01, 0) * h));
    if ((f0 | f1 | f2) < 0) return false;
    if (!tileMin) return true;
    const uint32_t bw = (width + 31) >> 5;
    const uint32_t* blockMin = tileMin + (width >> 2) * (height >> 2);
    // a chunk of at most 32 pixels a side touches at most 2 x 2 blocks, one of 64 at most 3 x 3
    const uint32_t bx0 = x0 >> 5, by0 = y0 >> 5, bx1 = (x1 - 1) >> 5, by1 = (y1 - 1) >> 5;
    uint32_t known = min(min(blockMin[by0 * bw + bx0], blockMin[by0 * bw + bx1]), min(blockMin[by1 * bw + bx0], blockMin[by1 * bw + bx1]));
    if (bx1 - bx0 > 1 || by1 - by0 > 1)
        for (uint32_t by = by0; by <= by1; by++)
            for (uint32_t bx = bx0; bx <= bx1; bx++) known = min(known, blockMin[by * bw + bx]);
    const float u = __int2float_rn((int32_t)e1), v = __int2float_rn((int32_t)e2);
    const float a20 = (float)r.A20, b20 = (float)r.B20, a01 = (float)r.A01, b01 = (float)r.B01;
    const float W = (float)(w + 2), H = (float)(h + 2);
    const float gx = ffma(r.Z10, a20, fmul(r.Z20, a01)), gy = ffma(r.Z10, b20, fmul(r.Z20, b01));
    const float m1 = ffma(fabsf(a20), W, ffma(fabsf(b20), H, fabsf(u))), m2 = ffma(fabsf(a01), W, ffma(fabsf(b01), H, fabsf(v)));
    const float S = ffma(fabsf(r.Z10), m1, ffma(fabsf(r.Z20), m2, fabsf(r.Z0)));
    float plane = ffma(u, r.Z10, ffma(v, r.Z20, r.Z0));
    plane = ffma(fmaxf(gx, 0.0f), (float)w, ffma(fmaxf(gy, 0.0f), (float)h, plane));
    plane = ffma(S, 0x1p-18f, plane);
    const float sum = __int2float_rn((int32_t)((uint32_t)r.E0 + (uint32_t)r.E1 + (uint32_t)r.E2));
    const float z1 = fmul(r.Z10, sum), z2 = fmul(r.Z20, sum);
    const float top = ffma(fadd(fabsf(r.Z0), fadd(fabsf(z1), fabsf(z2))), 0x1p-16f, fadd(r.Z0, fmaxf(fmaxf(z1, z2), 0.0f)));
    const float bound = z1 == z1 && z2 == z2 ? fminf(plane, top) : __int_as_float(0x7F800000);
    return ((uint32_t)max(__float_as_int(bound), 0) | 0x80000000u) >= known;
}

// A chunk of the alpha-tested triangle whose record (and AlphaExt after it) is at q.
__device__ __forceinline__ bool raster_chunk_alpha(const TriRec* q, const DevMaterial* materials, uint32_t x0, uint32_t y0,
                                                int tilesX, int tilesY, unsigned long long* keys, uint32_t* tileMin,
                                                uint32_t width, int lane, uint4* list) {
    const AlphaExt* xp = (const AlphaExt*)&q[1];
    const DevMaterial& mt = materials[xp->material & ~kTriAlpha];
    return raster_region_alpha(q, tile_test(*q), xp, mt.tex, mt.alpha_cutoff, x0, y0, tilesX, tilesY, keys, tileMin, width,
                               lane, list, kDiv16[tilesX]);
}

// kAlpha: the scene has alpha-tested materials (a build of its own with more registers, so that neither keeps
// the other's; 48 and 64 registers hold 40 and 32 warps per SM: chunk stages of the alpha-tested frame 459 ->
// 404 us).
template <bool kOver, bool kAlpha>
__global__ void __launch_bounds__(256, kAlpha || kOver ? 4 : 5) k_raster_big(const TriRec* __restrict__ big, const unsigned long long* __restrict__ bigBase,
                                                    unsigned long long* control, uint32_t capacity,
                                                    unsigned long long* keys, uint32_t* tileMin, uint32_t width, uint32_t height,
                                                    const ViewParams* __restrict__ views, uint32_t chunk,
                                                    const DevMaterial* __restrict__ materials, unsigned long long* counts,
                                                    uint32_t readTiles, uint32_t maxRun, bool lastStage) {
    __shared__ uint4 list[8][32];  // per warp: the live tiles being shaded
    const unsigned long long q = control[1];
    if (lastStage && blockIdx.x == 0 && threadIdx.x == 0)  // the next draw's second cursor, alpha list and idle-warp counts
        control[7] = control[9] = control[10] = control[11] = control[12] = 0;
    const uint32_t n = min(capacity, queue_slots(q));
    if (n == 0) return;
    const int lane = threadIdx.x & 31;
    const TriRec& last = big[n - 1];
    const int lastTX = (int)(((last.bbMax & 0xFFFF) - (last.bbMin & 0xFFFF)) >> 2);
    const int lastTY = (int)(((last.bbMax >> 16) - (last.bbMin >> 16)) >> 2);
    const uint32_t cw = chunk & 0xFF, ch = chunk >> 8, cwShift = 31 - __clz(cw);  // powers of two
    const unsigned long long total = bigBase[n - 1] + (unsigned long long)((lastTX + cw - 1) / cw) * ((lastTY + ch - 1) / ch);
    // a sparse queue (few big triangles) is spread with shorter runs so that every warp gets work
    const unsigned long long warps = (unsigned long long)gridDim.x * (blockDim.x >> 5);
    const unsigned long long share = total / (warps * kRunsPerWarp);
    const uint32_t run = (uint32_t)max(share ? 2ull : 1ull, min((unsigned long long)maxRun, share));
    // The warp's first run is its own by its index (blocks first: the queue starts with near geometry), later ones
    // come from the cursor; every warp of the grid is resident. (All warps at the cursor at once: 17.5 -> 15.2 us at
    // 1280x720, 93 -> 80 us in the sparse draw, with the run rule 233 -> 223 us for 24 batched views.)
    unsigned long long w0 = ((unsigned long long)(threadIdx.x >> 5) * gridDim.x + blockIdx.x) * run;
    for (bool own = true;; own = false) {
        if (!own) {
            if (lane == 0) w0 = warps * run + atomicAdd(&control[8], (unsigned long long)run);
            w0 = __shfl_sync(0xFFFFFFFFu, w0, 0);
        }
        if (w0 >= total) break;
        // the largest slot with bigBase[slot] <= w0: 32 probes a step
        uint32_t slot = 0, hi = n - 1;
        while (slot < hi) {
            const uint32_t step = (hi - slot + 31) / 32, probe = slot + step * (lane + 1);
            const uint32_t below = __popc(__ballot_sync(0xFFFFFFFFu, probe <= hi && bigBase[min(probe, hi)] <= w0));
            slot += below * step;
            hi = min(hi, slot + step - 1);
        }
        const unsigned long long w = w0 + lane;
        bool live = lane < run && w < total;
        uint32_t xy0 = 0, xy1 = 0, k = (uint32_t)(w - bigBase[slot]);  // the lane's chunk of its triangle
        if constexpr (!kAlpha) {
            // Every slot owns chunks: the triangles that start within the run set a bit each, and a lane's
            // triangle is as many slots on as bits are set up to it.
            const uint32_t next = slot + 1 + lane;
            const unsigned long long start = next < n ? bigBase[next] - w0 : 32ull;
            const unsigned starts = __reduce_or_sync(0xFFFFFFFFu, start < 32 ? 1u << start : 0u) & (0xFFFFFFFFu >> (31 - lane));
            slot += __popc(starts);
            if (starts) k = lane - (31 - __clz(starts));
        } else if (live) {  // at most 64 slots on (32 chunks, each of another triangle and its AlphaExt)
            uint32_t end = min(n - 1, slot + 2 * (uint32_t)lane);
            while (slot < end) {
                const uint32_t mid = (slot + end + 1) >> 1;
                if (bigBase[mid] <= w) slot = mid; else end = mid - 1;
            }
            k = (uint32_t)(w - bigBase[slot]);
        }
        if (live) {
            const TriRec r = big[slot];
            const uint32_t minX = r.bbMin & 0xFFFF, minY = r.bbMin >> 16, maxX = r.bbMax & 0xFFFF, maxY = r.bbMax >> 16;
            // k / chunksX by a reciprocal: (k + 1/2) / chunksX is at least 1 / 724 from an integer (chunksX <= 362,
            // k < 2^17), the rounding errors below 2^-12
            const uint32_t chunksX = (((maxX - minX) >> 2) + cw - 1) >> cwShift;
            const uint32_t cy = (uint32_t)__fdividef((float)k + 0.5f, (float)chunksX), cx = k - cy * chunksX;
            const uint32_t x0 = minX + cx * (cw * 4), y0 = minY + cy * (ch * 4);
            const uint32_t x1 = min(x0 + cw * 4, maxX), y1 = min(y0 + ch * 4, maxY);
            const uint32_t* vtiles = tileMin;
            uint32_t vw = width, vh = height;
            if (views) {
                const ViewParams& v = views[r.pad & ~kTriAlpha];
                vtiles = v.tileMin, vw = v.width, vh = v.height;
            }
            live = chunk_live(r, x0, y0, x1, y1, vtiles, vw, vh);
            xy0 = x0 | (y0 << 16), xy1 = x1 | (y1 << 16);
        }
        unsigned mask = __ballot_sync(0xFFFFFFFFu, live);
        while (mask) {
            const int src = __ffs(mask) - 1;
            mask &= mask - 1;
            const uint32_t s = __shfl_sync(0xFFFFFFFFu, slot, src);
            const uint32_t a = __shfl_sync(0xFFFFFFFFu, xy0, src), b = __shfl_sync(0xFFFFFFFFu, xy1, src);
            const uint32_t x0 = a & 0xFFFF, y0 = a >> 16, x1 = b & 0xFFFF, y1 = b >> 16;
            const int tilesX = (int)((x1 - x0) >> 2), tilesY = (int)((y1 - y0) >> 2);
            const TriRec r = big[s];
            unsigned long long* vkeys = keys;
            uint32_t* vtiles = tileMin;
            uint32_t vw = width, vh = height;
            if (views) {
                const ViewParams& v = views[r.pad & ~kTriAlpha];
                vkeys = v.keys, vtiles = v.tileMin, vw = v.width, vh = v.height;
            }
            if constexpr (kOver) {
                raster_region_overdraw(r, tile_test(r), x0, y0, tilesX, tilesY, vkeys, counts, vw, lane, list[threadIdx.x >> 5], kDiv16[tilesX]);
            } else {
                bool any;
                if (kAlpha && (r.pad & kTriAlpha))
                    any = raster_chunk_alpha(big + s, materials, x0, y0, tilesX, tilesY, vkeys, vtiles, vw, lane,
                                             list[threadIdx.x >> 5]);
                else
                    any = raster_region(r, tile_test(r), x0, y0, tilesX, tilesY, vkeys, vtiles, vw, lane, readTiles, list[threadIdx.x >> 5], kDiv16[tilesX]);
                if (!any && vtiles) refresh_blocks(x0, y0, x1, y1, vtiles, vw, vh, lane);
            }
        }
    }
}

// Keys from a depth layer (pre-existing depth: low word kKeyEmptyLow) and, when kept, each tile's
// depth bound as the minimum over its 16 pixels (a tile is 16 consecutive words; the grid stride
// is a multiple of 16, so a half-warp always covers one tile).
__global__ void k_init_keys(const uint32_t* __restrict__ depth, unsigned long long* __restrict__ keys,
                            uint32_t* __restrict__ tileMin, uint32_t n, uint32_t blocks) {
    if (tileMin)  // no bound yet: the chunk stage raises the blocks it finds hidden
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < blocks; i += gridDim.x * blockDim.x) tileMin[(n >> 4) + i] = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint32_t hi = float_order(__uint_as_float(depth[i]));
        keys[i] = ((unsigned long long)hi << 32) | kKeyEmptyLow;
        if (tileMin) {
            const unsigned half = 0xFFFFu << (threadIdx.x & 16);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) hi = min(hi, __shfl_xor_sync(half, hi, o));
            if ((i & 15) == 0) tileMin[i >> 4] = hi;
        }
    }
}

__global__ void k_clear(uint32_t* __restrict__ l0, uint32_t* __restrict__ l1, unsigned long long* __restrict__ keys,
                        uint32_t* __restrict__ tileMin, uint32_t n, uint32_t blocks, uint32_t color, uint32_t depthBits) {
    const uint32_t hi = float_order(__uint_as_float(depthBits));
    if (tileMin)
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < blocks; i += gridDim.x * blockDim.x) tileMin[(n >> 4) + i] = hi;
    const unsigned long long key = ((unsigned long long)hi << 32) | kKeyEmptyLow;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) * 4; i < n; i += gridDim.x * blockDim.x * 4) {
        // n is a multiple of 16 (4x4 tiles), so the 16-byte vectors never straddle the end
        *(uint4*)&l0[i] = make_uint4(color, color, color, color);
        if (l1) *(uint4*)&l1[i] = make_uint4(depthBits, depthBits, depthBits, depthBits);
        if (keys) {
            *(ulonglong2*)&keys[i] = make_ulonglong2(key, key);
            *(ulonglong2*)&keys[i + 2] = make_ulonglong2(key, key);
        }
        if (tileMin && (i & 15) == 0) tileMin[i >> 4] = hi;
    }
}

__global__ void k_fill(uint32_t* __restrict__ dst, uint32_t n, uint32_t v) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) dst[i] = v;
}

__global__ void k_finalize(const unsigned long long* __restrict__ keys, uint32_t* __restrict__ l0,
                           uint32_t* __restrict__ l1, uint32_t n) {
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) * 2; i < n; i += gridDim.x * blockDim.x * 2) {
        const ulonglong2 k = *(const ulonglong2*)&keys[i];
        const unsigned long long kk[2] = { k.x, k.y };
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const uint32_t low = (uint32_t)kk[j];
            if (low == kKeyEmptyLow) continue;
            l1[i + j] = __float_as_uint(float_unorder((uint32_t)(kk[j] >> 32)));
            if (l0) l0[i + j] = rank_surface_id(0xFFFFFFFEu - low);  // l0 null: depth only
        }
    }
}

// OverdrawShader results: layer 0 += the counters (two saturating 16-bit halves, as the
// reference's _mm512_adds_epu16 accumulate them), layer 1 = the maximum depth where a sample
// raised it.
__global__ void k_finalize_overdraw(const unsigned long long* __restrict__ keys, const unsigned long long* __restrict__ counts,
                                    uint32_t* __restrict__ l0, uint32_t* __restrict__ l1, uint32_t n) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned long long c = counts[i];
        const uint32_t old = l0[i];
        const unsigned long long lo = (old & 0xFFFFu) + (c & 0xFFFFFFFFull), hi = (old >> 16) + (c >> 32);
        l0[i] = (uint32_t)min(lo, 0xFFFFull) | ((uint32_t)min(hi, 0xFFFFull) << 16);
        const unsigned long long k = keys[i];
        if ((uint32_t)k != kKeyEmptyLow) l1[i] = __float_as_uint(float_unorder((uint32_t)(k >> 32)));
    }
}

// Framebuffer::GetPixels de-tiling (ImageHelpers.cpp:109-147) into a row-major buffer, a thread per row of
// a 4x4 tile: a 16-byte load, and a 16-byte store where the rows of dst are aligned (vec). kKeys: pending draws are
// read from the keys, which the layer's words (layer 0: surface ids, 1: depths) only fill in for, instead of
// being written to the layers first: 12 bytes a pixel instead of 24. Bound by bandwidth: two 2560x1440 layers
// 14.9 -> 9.2 us (a thread per pixel before); the ids of 24 views of 256x256 to 2560x1440 from their keys
// 164 -> 90 us, the pass over their layers included (a thread per tile: 157).
template <bool kKeys>
__global__ void __launch_bounds__(256) k_detile(const uint32_t* __restrict__ src, const unsigned long long* __restrict__ keys, uint32_t* dst,
                                                uint32_t width, uint32_t height, uint32_t stride, uint32_t layer, uint32_t vec) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, t = i >> 2, tw = width >> 2;
    if (t >= tw * (height >> 2)) return;
    const uint32_t ty = t / tw, tx = t - ty * tw;
    uint32_t v[4];
    if constexpr (kKeys) {
        const ulonglong2 p = ((const ulonglong2*)keys)[2 * i], q = ((const ulonglong2*)keys)[2 * i + 1];
        const unsigned long long k[4] = { p.x, p.y, q.x, q.y };
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const uint32_t low = (uint32_t)k[j];
            if (low == kKeyEmptyLow) v[j] = src[4 * i + j];
            else v[j] = layer == 0 ? rank_surface_id(0xFFFFFFFEu - low) : __float_as_uint(float_unorder((uint32_t)(k[j] >> 32)));
        }
    } else {
        const uint4 p = ((const uint4*)src)[i];
        v[0] = p.x, v[1] = p.y, v[2] = p.z, v[3] = p.w;
    }
    uint32_t* row = dst + (size_t)(ty * 4 + (i & 3)) * stride + tx * 4;
    if (vec) {
        *(uint4*)row = make_uint4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++) row[j] = v[j];
    }
}

static int grid_for(uint32_t n, int perThread, int block) {
    long long g = ((long long)n / perThread + block - 1) / block;
    return (int)max(1ll, min(g, 152ll * 16));
}

uint32_t order_stride(uint32_t count) {
    if (count <= 2) return 1;
    uint32_t s = (uint32_t)((double)count * 0.6180339887498949) | 1u;
    while (std::gcd(s, count) != 1u) s += 2;
    return s % count;
}

// The dynamic shared memory limit of a mesh-stage pass is an attribute of the kernel in one
// device's context: it is raised per device (and only when a larger size is needed), under a lock
// because draws may come from several host threads.
static void raise_smem_limit(int pass, const void* kernel, size_t bytes) {
    static std::mutex mu;
    static size_t setSize[64][6] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
    std::lock_guard<std::mutex> lock(mu);
    if (bytes <= setSize[dev][pass]) return;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess)
        setSize[dev][pass] = bytes;
}

constexpr uint32_t kMaxPartShift = 5;  // a share of two to four triangles
void launch_draw(const DrawArgs& args, cudaStream_t st, int numSMs) {
    DrawArgs a = args;
    if (!a.views) {
        a.orderStride = order_stride(a.count);
        // Single-view draws skip the key read for triangles above 4 tiles (1080p, 100k meshlets:
        // 1.378 -> 1.320 ms); batched draws of many small views lose by it (64 views 5.93 -> 6.34
        // ms), because their tiles are mostly covered partially, and keep every read.
        a.keyReadTiles = 4;
    }
    const uint32_t warps = a.warpsPerBlock ? a.warpsPerBlock : kWarpsPerBlock;
    const size_t smem = warps * sizeof(WarpSmem), smemAlpha = warps * sizeof(WarpSmemAlpha);
    if (smem > 48 * 1024)
        raise_smem_limit(a.counts ? kPassOverdraw : kPassOpaque,
                         a.counts ? (const void*)k_draw_meshlets<kPassOverdraw> : (const void*)k_draw_meshlets<kPassOpaque>,
                         smem);
    if (a.s.alphaList && smemAlpha > 48 * 1024) raise_smem_limit(kPassAlpha, (const void*)k_draw_meshlets<kPassAlpha>, smemAlpha);
    const uint32_t chunk = chunk_shape(a);
    const int grid = numSMs * (32 / warps);  // 64 registers a thread leave room for 32 resident warps per SM
    if (a.counts) {  // OverdrawShader: one pass, every meshlet
        {
            LaunchScope ls("k_draw_meshlets_overdraw", st);
            k_draw_meshlets<kPassOverdraw><<<grid, warps * 32, smem, st>>>(a);
        }
        LaunchScope ls("k_raster_big_overdraw", st);
        k_raster_big<true, false><<<numSMs * 4, 256, 0, st>>>(a.s.big, a.s.bigBase, a.s.control, a.s.bigCapacity, a.keys, nullptr,
                                                       a.width, a.height, a.views, chunk, a.materials, a.counts, 0u, kChunkRun,
                                                              true);
        return;
    }
    auto chunks = [&](bool last) {
        LaunchScope ls("k_raster_big", st);
        if (a.s.alphaList && last)
            k_raster_big<false, true><<<numSMs * 4, 256, 0, st>>>(a.s.big, a.s.bigBase, a.s.control, a.s.bigCapacity, a.keys,
                                                                  a.tileMin, a.width, a.height, a.views, chunk, a.materials,
                                                                  nullptr, a.keyReadTiles, kChunkRunAlpha, true);
        else
            k_raster_big<false, false><<<numSMs * 5, 256, 0, st>>>(a.s.big, a.s.bigBase, a.s.control, a.s.bigCapacity, a.keys,
                                                                   a.tileMin, a.width, a.height, a.views, chunk, a.materials,
                                                                   nullptr, a.keyReadTiles, kChunkRun, last);
    };
    // Before the alpha pass, which then meets the depth bounds of the opaque pass's large triangles (inside a
    // 50k-meshlet scene, half of the materials alpha-tested: alpha pass 239 -> 109 us, chunk stages 383 -> 429 us).
    auto opaque_chunks = [&] {
        chunks(false);
        cudaMemsetAsync(&a.s.control[1], 0, sizeof(unsigned long long), st);  // an empty queue
    };
    // The alpha pass's grid: as many blocks as its larger shared memory lets an SM hold.
    const int gridAlpha = numSMs * (int)std::max<size_t>(1, std::min<size_t>(32 / warps, 227 * 1024 / (smemAlpha + 1024)));
    if (a.shaded) {  // meshlets shaded by a user mesh shader
        if (smem > 48 * 1024) raise_smem_limit(3, (const void*)k_draw_meshlets<kPassOpaque, true>, smem);
        if (a.s.alphaList && smemAlpha > 48 * 1024) raise_smem_limit(4, (const void*)k_draw_meshlets<kPassAlpha, true>, smemAlpha);
        {
            LaunchScope ls("k_draw_meshlets_shaded", st);
            k_draw_meshlets<kPassOpaque, true><<<grid, warps * 32, smem, st>>>(a);
        }
        if (a.s.alphaList) {
            opaque_chunks();
            LaunchScope ls("k_draw_meshlets_shaded_alpha", st);
            k_draw_meshlets<kPassAlpha, true><<<gridAlpha, warps * 32, smemAlpha, st>>>(a);
        }
    } else {
        {
            LaunchScope ls("k_draw_meshlets", st);
            if (a.views == nullptr && a.count <= (uint32_t)grid * warps) {
                if (smem > 48 * 1024) raise_smem_limit(5, (const void*)k_draw_meshlets<kPassOpaque, false, true>, smem);
                while (a.partShift < kMaxPartShift && (uint64_t)a.count << (a.partShift + 1) <= (uint64_t)grid * warps) a.partShift++;
                k_draw_meshlets<kPassOpaque, false, true><<<grid, warps * 32, smem, st>>>(a);
            } else {
                k_draw_meshlets<kPassOpaque><<<grid, warps * 32, smem, st>>>(a);
            }
        }
        if (a.s.alphaList) {  // the scene has alpha-tested materials
            opaque_chunks();
            LaunchScope ls("k_draw_meshlets_alpha", st);
            k_draw_meshlets<kPassAlpha><<<gridAlpha, warps * 32, smemAlpha, st>>>(a);
        }
    }
    chunks(true);
}

void launch_init_keys(const uint32_t* depthLayer, unsigned long long* keys, uint32_t* tileMin, uint32_t width, uint32_t height,
                      cudaStream_t st) {
    LaunchScope ls("k_init_keys", st);
    const uint32_t n = width * height;
    k_init_keys<<<grid_for(n, 1, 256), 256, 0, st>>>(depthLayer, keys, tileMin, n, tile_blocks(width, height));
}

void launch_clear(uint32_t* l0, uint32_t* l1, unsigned long long* keys, uint32_t* tileMin, uint32_t width, uint32_t height,
                  uint32_t color, uint32_t depthBits, cudaStream_t st) {
    LaunchScope ls("k_clear", st);
    const uint32_t n = width * height;
    k_clear<<<grid_for(n, 4, 256), 256, 0, st>>>(l0, l1, keys, tileMin, n, tile_blocks(width, height), color, depthBits);
}

void launch_fill(uint32_t* dst, uint32_t n, uint32_t value, cudaStream_t st) {
    LaunchScope ls("k_fill", st);
    k_fill<<<grid_for(n, 1, 256), 256, 0, st>>>(dst, n, value);
}

void launch_finalize(const unsigned long long* keys, uint32_t* l0, uint32_t* l1, uint32_t n, cudaStream_t st) {
    LaunchScope ls("k_finalize", st);
    k_finalize<<<grid_for(n, 2, 256), 256, 0, st>>>(keys, l0, l1, n);
}

void launch_finalize_overdraw(const unsigned long long* keys, const unsigned long long* counts, uint32_t* l0, uint32_t* l1,
                              uint32_t n, cudaStream_t st) {
    LaunchScope ls("k_finalize_overdraw", st);
    k_finalize_overdraw<<<grid_for(n, 1, 256), 256, 0, st>>>(keys, counts, l0, l1, n);
}

void launch_detile(const uint32_t* src, const unsigned long long* keys, uint32_t* dst, uint32_t width, uint32_t height,
                   uint32_t stride, uint32_t layer, cudaStream_t st) {
    LaunchScope ls("k_detile", st);
    const uint32_t blocks = (width * (height >> 2) + 255) / 256, vec = ((uintptr_t)dst & 15) == 0 && stride % 4 == 0;
    if (keys) k_detile<true><<<blocks, 256, 0, st>>>(src, keys, dst, width, height, stride, layer, vec);
    else k_detile<false><<<blocks, 256, 0, st>>>(src, nullptr, dst, width, height, stride, layer, vec);
}

}  // namespace swr
