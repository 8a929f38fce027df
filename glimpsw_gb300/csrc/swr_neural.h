// Learned texture decoder shared definitions: the per-material parameter block, the BF16 operand
// image the tensor-core kernels copy into shared memory, the per-material latent pyramid, and the
// kernels' argument blocks. The decoder has no counterpart in the reference; the plain sampler
// (SampleLevel<SurfaceSampler>, Texture.h:412-459) produces its training targets and stays the
// fallback for texture levels the latents do not cover.
#pragma once
#include <atomic>
#include <cstdint>

#include "swr_internal.h"

namespace swr {

constexpr uint32_t kNeuralChannels = 8;     // latent channels
constexpr uint32_t kNeuralHidden = 64;      // two hidden layers of 64 (GELU)
constexpr uint32_t kNeuralOutputs = 8;      // albedo RGB, normal XY, metallic, roughness, AO
constexpr uint32_t kNeuralMaxLevels = 4;    // latent levels; latent level k has texture level k+2's size
constexpr uint32_t kNeuralMaxDecoded = kNeuralMaxLevels + 2;  // decoded texture levels 0 .. levels+1
constexpr uint32_t kNeuralDownscale = 4;    // texture level 0 texels per latent level 0 texel, per axis
constexpr uint32_t kNeuralMaxStepMaterials = 64;

// FP32 parameter block of one material (padded layout; 5384 live parameters):
//   W1[64][16]: columns 0-7 weigh the latent channels, column 8 is b1 (the input vector carries a
//               constant 1 there), columns 9 and 10 weigh the level-0 / level-1 flags, columns
//               11-15 are zero and stay zero;
//   W2[64][64], b2[64], W3[8][64], b3[8].
constexpr uint32_t kPW1 = 0, kPW2 = 1024, kPB2 = 5120, kPW3 = 5184, kPB3 = 5696, kNeuralParams = 5704;

// BF16 operand image of one material (slab layout of swr_tc.cuh, K-major B operands):
//   W1 [64 n][16 k], W2 [64][64], W3 [16][64] (rows 8-15 zero), b2 f32[64], b3 f32[16]   forward part
//   W3t [64][16] (= W3^T), W2t [64][64] (= W2^T), W1t [16][64] (= W1^T)                    backward part
constexpr uint32_t kIW1 = 0, kIW2 = 2048, kIW3 = 10240, kIB2 = 12288, kIB3 = 12544, kNeuralFwdImage = 12800;
constexpr uint32_t kIW3t = 12800, kIW2t = 14848, kIW1t = 23040, kNeuralImage = 25088;

// Kernel view of a model.
struct NeuralDev {
    uint32_t numMaterials, levels;
    uint32_t texelsPerMaterial;                 // latent texels over all levels
    uint32_t levelOffset[kNeuralMaxLevels];     // first texel of each level inside a material block
    uint32_t levelW[kNeuralMaxLevels], levelH[kNeuralMaxLevels];
    const DevTexture* tex;                      // per material (layer 0 RGBA, layer 1 NX NY M R)
    const uint16_t* latentHalf;                 // FP16 [material][texel][8]
    const uint8_t* image;                       // [material][kNeuralImage]
    uint64_t waitNs;                            // limit of each bounded tensor-core / copy wait
};

struct NeuralTrainArgs {
    NeuralDev n;
    const float* latent;        // FP32 master [material][texel][8]
    float* latentGrad;          // same shape, accumulated by the step
    float* partial;             // [block][kNeuralParams] parameter gradients of each block
    const uint32_t* samples;    // optional explicit samples [slot][samplesPerMaterial]: level<<28 | ty<<14 | tx
    const uint32_t* invalid;    // with explicit samples: nonzero if one lies outside the texture (nothing runs)
    float* loss;                // [0] += squared error, [1] += samples
    uint32_t* status;           // bit 0: a tensor-core wait timed out
    uint32_t materials[kNeuralMaxStepMaterials];
    uint32_t numSlots, samplesPerMaterial, ctasPerMaterial;
    uint32_t seedLo, seedHi, step;
    uint32_t levelShift;        // level l drawn with weight 2^(levelShift (levels-1-l))
};

struct NeuralAdamArgs {
    float* params;              // [material][kNeuralParams]
    float* m;
    float* v;
    const float* partial;
    uint8_t* image;
    float* latent;
    float* latentM;
    float* latentV;
    float* latentGrad;
    uint32_t texelsPerMaterial;
    uint32_t ctasPerMaterial, numSlots;
    float lr, beta1, beta2, eps;
    uint32_t materials[kNeuralMaxStepMaterials];
    float lrm[kNeuralMaxStepMaterials];   // lr / (1 - beta1^t) per slot (t: the material's step count)
    float s2[kNeuralMaxStepMaterials];    // 1 / sqrt(1 - beta2^t) per slot
};

struct NeuralDecodeArgs {
    NeuralDev n;
    const unsigned long long* sorted;   // requests grouped by material: slot<<32 | level<<28 | ty<<14 | tx
    const uint32_t* reqOffset;          // [numMaterials + 1] first request of each material
    const uint32_t* tileOffset;         // [numMaterials + 1] first 128-request tile of each material
    uint2* out;                         // [slot] decoded (layer 0 RGBA8 with AO in alpha, layer 1 RGBA8)
    uint32_t* status;
    // without lists (sorted == nullptr): the count texels of one material, decoded to slots 0, 1, ...
    const uint32_t* texels;
    const uint32_t* invalid;            // nonzero if one of them lies outside the texture (nothing runs)
    uint32_t material, count;
};

// Sets *invalid if one of the packed texels (level<<28 | ty<<14 | tx) is outside the decoded levels of a width x
// height texture.
void launch_neural_check(const uint32_t* texels, uint32_t count, uint32_t decodedLevels, uint32_t width, uint32_t height,
                         uint32_t* invalid, cudaStream_t st);
// out[i] = the sum of partial[c][i] over the c < ctas gradients, in that order.
void launch_neural_sum(const float* partial, uint32_t ctas, float* out, cudaStream_t st);
void launch_neural_train(const NeuralTrainArgs& a, uint32_t blocks, cudaStream_t st);
void launch_neural_adam(const NeuralAdamArgs& a, cudaStream_t st);
void launch_neural_decode(const NeuralDecodeArgs& a, uint32_t blocks, cudaStream_t st);
uint32_t neural_decode_blocks_per_sm();  // resident decode CTAs per SM (shared memory and TMEM bound)
void launch_neural_image(float* params, uint8_t* image, uint32_t numMaterials, cudaStream_t st);
void launch_neural_latent_init(const NeuralDev& n, float* latent, cudaStream_t st);
void launch_neural_export(const float* latent, uint16_t* half, size_t count, cudaStream_t st);
// One CTA announces a 16-byte copy on an mbarrier and issues none, waits at most limitNs with TMEM
// allocated, then frees the TMEM and sets status bit 0 if the wait gave up.
void launch_wait_selftest(uint32_t* status, uint64_t limitNs, cudaStream_t st);
void launch_neural_offsets(const uint32_t* counts, uint32_t* reqOffset, uint32_t* tileOffset, uint32_t numMaterials,
                           cudaStream_t st);
// The emit pass counts requests per material in kCountCopies copies on lines of their own, a block in copy block %
// kCountCopies (one word per material, all on a line, took 230,000 atomics a frame: emit pass 162 -> 94 us).
constexpr uint32_t kCountCopies = 16;
__host__ __device__ inline uint32_t count_stride(uint32_t numMaterials) { return (numMaterials + 32u) & ~31u; }
// Flags of the neural resolve's pixel records (swr_shade.cu); the filter weights are in bits 8 to 23.
enum : uint32_t {
    kSurfFast = 1u,        // sampled from decoded texels, or untextured (albedo and NMR 0)
    kSurfDecoded = 2u,     // a decoded material sample: fetch it
    kSurfNearest = 4u, kSurfInX = 8u, kSurfInY = 16u, kSurfTwoLayers = 32u,
    kSurfHand = 1u << 31,  // the bitangent's sign bit
};
// Whether a decoded sample needs the texel of slot k (00 10 01 11), and which it is.
__host__ __device__ inline bool surf_has_slot(uint32_t flags, uint32_t k) {
    return k == 0 || (!(flags & kSurfNearest) && (!(k & 1) || (flags & kSurfInX)) && (!(k & 2) || (flags & kSurfInY)));
}
__host__ __device__ inline uint32_t surf_slot_texel(uint32_t first, uint32_t k) { return first + (k & 1) + ((k >> 1) << 14); }
// records: the second plane of the pixels' records.
void launch_neural_scatter(const uint4* records, uint32_t pixels, const uint32_t* reqOffset, uint32_t* cursor,
                           unsigned long long* sorted, uint32_t* levelCount, uint32_t numMaterials, cudaStream_t st);

}  // namespace swr

struct swr_neural_t;
namespace swr {
void neural_sync_half(swr_neural_t* n, cudaStream_t st);  // FP16 latents up to date with the master copy
int neural_num_sms();
}  // namespace swr

struct swr_neural_t {
    swr::NeuralDev d;                        // device view (pointers below)
    std::vector<swr::DevTexture> texHost;
    swr::DevTexture* tex;
    float *latent, *latentM, *latentV, *latentGrad;
    uint16_t* latentHalf;
    float *params, *paramM, *paramV;
    uint8_t* image;
    float* partial;
    size_t partialFloats;
    float* loss;                             // device: squared error, samples, the status word, then the check flags
    uint32_t* status;                        // device: loss + 2
    std::atomic<uint64_t> flagsInUse{0};     // check flags (kCheckFlags words after loss[3]; 0 when free) held by calls
    std::vector<uint32_t> steps;             // Adam step count per material
    uint64_t seed;
    uint32_t trainCalls;
    bool halfStale;                          // latentHalf behind the master copy
    // neural resolve scratch (grow-only)
    unsigned long long* sorted;
    uint2* decoded;
    uint4* surf;                             // two planes of a word per pixel: the emit pass's surface records
    size_t scratchSlots;
    uint32_t* counters;                      // kCountCopies counts | cursors | reqOffset | tileOffset, numMaterials+1 each,
                                             // then 4 per-level request counts
};
