// slot_ranges.cuh -- how the CTAs that update the LRU's slots (k_slots and
// k_query_front, pipeline.cu) share them out, and which of them have a status
// word.  Free of the CUDA runtime, so that a host build of it can be checked.
#pragma once

#include <stdint.h>

namespace bcmc {

constexpr uint32_t kSlotChunk = 1024;  // four slots to each of a CTA's 256 threads

// A contiguous range of slots.  A CTA without any publishes no count and adds up
// none: its rank may lie past the status words (a cluster has more CTAs than a
// small cache has chunks).
struct SlotRange {
    uint32_t first, end;

    __host__ __device__ __forceinline__ bool any() const { return first < end; }
};

// The range of CTA `rank` of `ctas`: whole chunks, as even as these allow.
__host__ __device__ __forceinline__ SlotRange slot_range(uint32_t slots, uint32_t ctas, uint32_t rank)
{
    const uint64_t share = ((uint64_t)slots + ctas - 1u) / ctas;
    const uint64_t range = (share + kSlotChunk - 1u) / kSlotChunk * kSlotChunk;
    const uint64_t first = (uint64_t)rank * range, end = first + range;
    return SlotRange{(uint32_t)(first < slots ? first : slots), (uint32_t)(end < slots ? end : slots)};
}

// Status words that CTAs with slots use: ranges are whole chunks, so no more CTAs
// have one than there are chunks.
__host__ __device__ __forceinline__ uint32_t slot_tiles(uint32_t slots)
{
    return (uint32_t)(((uint64_t)slots + kSlotChunk - 1u) / kSlotChunk);
}

}  // namespace bcmc
