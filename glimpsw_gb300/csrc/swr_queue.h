// The tail of the chunk queue: one 64-bit word, the slots taken in its high 24 bits and their chunks in its low 40,
// so that one addition claims both. A claim without room is taken back at once, so the word never holds more than
// the queue's capacity plus the claims in flight, and neither field reaches its end: slots carried out of the word
// (or chunks into the slots) would hand out slots that other triangles hold. Plain integer code, for host tests too.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define SWR_QUEUE_FN inline __host__ __device__
#else
#define SWR_QUEUE_FN inline
#endif

namespace swr {

constexpr uint32_t kQueueChunkBits = 40, kQueueSlotBits = 64 - kQueueChunkBits;
// In flight at once: 32 claims of a warp, of at most two slots (an alpha-tested triangle) and 2^17 chunks (362 x 362
// of 2 x 2 tiles at 2896 x 2896), of the 64 warps of each of at most 256 SMs.
constexpr uint32_t kQueueWarps = 256 * 64;
constexpr unsigned long long kQueueSlotsInFlight = kQueueWarps * 32ull * 2, kQueueChunksInFlight = kQueueWarps * 32ull << 17;
constexpr uint32_t kQueueMaxCapacity = (1u << kQueueSlotBits) - 1 - (uint32_t)kQueueSlotsInFlight;
// Claims from here on have no room either, whatever the capacity.
constexpr unsigned long long kQueueChunkLimit = 1ull << (kQueueChunkBits - 1);
static_assert(kQueueMaxCapacity + kQueueSlotsInFlight < 1ull << kQueueSlotBits, "slots");
static_assert(kQueueChunkLimit + kQueueChunksInFlight < 1ull << kQueueChunkBits, "chunks");

SWR_QUEUE_FN unsigned long long queue_claim(uint32_t slots, uint32_t chunks) {
    return ((unsigned long long)slots << kQueueChunkBits) | chunks;
}
SWR_QUEUE_FN uint32_t queue_slots(unsigned long long tail) { return (uint32_t)(tail >> kQueueChunkBits); }
SWR_QUEUE_FN unsigned long long queue_chunks(unsigned long long tail) { return tail & ((1ull << kQueueChunkBits) - 1); }
// Whether a triangle of `slots` slots whose claim starts at slot and chunk `base` has room. The claims without room
// are the last ones: what follows one of them starts past its slots and chunks.
SWR_QUEUE_FN bool queue_fits(uint32_t slot, unsigned long long base, uint32_t slots, uint32_t capacity) {
    return slot + slots <= capacity && base < kQueueChunkLimit;
}

}  // namespace swr
