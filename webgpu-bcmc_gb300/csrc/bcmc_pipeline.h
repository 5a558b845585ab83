// bcmc_pipeline.h -- argument blocks and launchers of the query pipeline
// kernels (pipeline.cu).  Internal to libbcmc_gb300.
#pragma once

#include "bcmc_impl.h"

namespace bcmc {

// k_query_flags: every block's range tested against the isovalue, in words of
// 32 consecutive blocks
struct FlagArgs {
    const float2* ranges;
    BlockGrid grid;  // id -> (x, y, z) without integer division
    uint32_t total;  // blocks
    uint32_t wpw;    // words a warp takes at a time
    uint4* near;     // per word: A, B and A & B ORed with the x neighbours', and A
    uint4* up;       // per word: A and B ORed with the next block's along x, and B
};

// Of which blocks the range, and the ranges of the neighbours on the + sides, hold
// all voxels: those below these coordinates and this id.
struct SoundRanges {
    uint32_t x, y, z, id;
};
// dims in voxels; `ranged`: how many blocks have their range (zfp_ranged_blocks)
SoundRanges sound_ranges(const uint32_t dims[3], const BlockGrid& grid, uint64_t ranged);

struct ActiveArgs {
    BlockGrid grid;
    const uint32_t* item_needed;  // standalone LRU update: the items needed (k_active)
    uint32_t* active_out;     // per-block active flags (MC path)
    const int32_t* item_slots;  // cachedItemSlots
    uint32_t total;           // blocks / items
    uint32_t* active_ids;     // compacted active ids (nullable)
    uint32_t* new_ids;        // compacted ids that need caching
    uint64_t* status_a;
    uint64_t* status_n;
    // MC path: k_query_flags' words, and room for each word's active and needed bits
    const uint4* near = nullptr;
    const uint4* up = nullptr;
    uint2* words = nullptr;
    // MC path: the active blocks that can have vertices, their ids and their places
    // among the active ids, and the blocks for which the ranges can tell
    uint32_t* live_ids = nullptr;
    uint32_t* live_at = nullptr;
    uint64_t* status_l = nullptr;
    uint32_t* live_words = nullptr;
    SoundRanges sound{};
};

struct SlotArgs {
    const uint32_t* needed;   // per item: 1 if needed this update
    uint32_t* slot_age;
    uint32_t* slot_avail;
    int32_t* slot_item;
    uint32_t* avail_ids;      // compacted available slots (ascending)
    uint32_t* avail_keys;     // their ages
    uint64_t* status;
    // computeSurface skips the cache update when no block is active
    // (compressed_marching_cubes.js:630-641); LRUCache.update itself always ages
    uint32_t skip_when_inactive;
    // 1: also accumulate the digit histograms of ~age (the descending sort's
    // keys) and make the sort's pass plan in the last CTA, so the sort that
    // follows runs without its histogram kernel
    uint32_t plan;
    // the joint histogram of the 16-bit age keys whose age is below 256 in
    // its class (kAgeBins bins: class, low byte), zero between updates, and
    // the dense rank of each bin, for a one-pass sort when every key is such
    // and at most 256 bins are used
    uint32_t* age_hist;
    uint8_t* age_rank;
};

struct AssignArgs {
    const uint32_t* new_ids;
    const uint32_t* sorted_b;  // sorted slot ids in sort buffer b or c
    const uint32_t* sorted_c;
    uint32_t* slot_age;
    uint32_t* slot_avail;
    int32_t* slot_item;
    int32_t* item_slots;
    const uint64_t* words;    // set: decode each new block into its slot
    uint32_t max_bits;
    float* cache;
    // set: new blocks [0, stage_blocks) were decoded into stage (one element
    // per new-block index) by k_decode_new and are copied into their slots
    const float* stage;
    uint32_t stage_blocks;
};

// k_decode_new: the new blocks' ZFP decode, run beside the LRU's slot
// selection (it needs only the new ids) into a staging buffer.
struct DecodeArgs {
    const uint32_t* new_ids;
    const uint64_t* words;
    uint32_t max_bits;
    float* stage;           // stage_blocks * 64 floats
    uint32_t stage_blocks;
};

struct McArgs {
    const uint32_t* active;
    const uint32_t* active_ids;
    const uint32_t* live_ids;  // the blocks to look at (ActiveArgs)
    const uint32_t* live_at;
    const int32_t* item_slots;
    const float* cache;
    BlockGrid grid;
    uint32_t* with_verts;
    uint32_t* vert_offsets;
    uint32_t* block_counts;  // vertices of each block looked at (count pass -> list entries)
    uint2* verts;
    uint64_t* status_v;
    uint64_t* status_b;
    // 1: verts is page-locked host memory; each warp's vertex stores then
    // cover one 256 B-aligned window, which such stores need for full speed
    uint32_t host_verts;
};

void query_begin_launch(QueryState* q, float iso, int mc_only, uint32_t capacity, uint32_t vert_capacity,
                        cudaStream_t s);
// Bytes of the word buffers of a volume of `total` blocks.
size_t flag_bytes(uint64_t total);
// Starts a query and makes its words; `in` set: the inputs come from there.
void query_flags_launch(bcmc_ctx* ctx, QueryState* q, float iso, uint32_t capacity, uint32_t vert_capacity,
                        const float* ranges, const BlockGrid& grid, uint32_t total, void* words, cudaStream_t s,
                        const QueryInputs* in = nullptr);
// The active test on the words.
void active_words_launch(bcmc_ctx* ctx, QueryState* q, ActiveArgs a, void* words, cudaStream_t s);
void query_end_launch(const QueryState* q, QueryState* host, cudaStream_t s);
// The flags, the active test and the slots of a volume that is small enough, in one launch.
bool query_front_takes(uint32_t total);
void query_front_launch(QueryState* q, const QueryInputs* in, const float* ranges, ActiveArgs a, void* words, const SlotArgs& sa,
                        cudaStream_t s);
void active_launch(bcmc_ctx* ctx, QueryState* q, const ActiveArgs& a, cudaStream_t s);
void slots_launch(bcmc_ctx* ctx, QueryState* q, const SlotArgs& a, uint32_t max_slots, cudaStream_t s);
void assign_launch(bcmc_ctx* ctx, QueryState* q, const AssignArgs& a, uint32_t max_new, cudaStream_t s);
void decode_new_launch(bcmc_ctx* ctx, const QueryState* q, const DecodeArgs& a, cudaStream_t s);
void mc_launch(bcmc_ctx* ctx, QueryState* q, const McArgs& a, uint32_t max_active, cudaStream_t s);
uint32_t active_tiles(uint32_t total);
uint32_t mc_grid(bcmc_ctx* ctx, uint32_t max_active);

}  // namespace bcmc
