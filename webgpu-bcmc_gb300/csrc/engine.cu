// engine.cu -- batched isosurface queries over several resident volumes with
// one shared pool of decoded-block slots (bcmc_engine_* in include/bcmc.h).
//
// A launch sequence answers up to max_batch (volume, isovalue) queries:
//   k_bbegin   new epoch of the status words, counters cleared
//   k_bactive  every query's active test over its volume's blocks, as one
//              stream of 1024-block tiles (query-major), in words of 32 blocks.
//              A tile whose extended value range (its blocks and their 26
//              neighbours, from volume load) excludes the isovalue is skipped
//              whole.  Active bits go to a per-query bitmap, counts to the tiles
//   k_bentries (not for a batch of up to eight tiles, whose entries k_bactive makes)
//              (query, block) entries of the active blocks that can have vertices
//              in query-major, block-ascending order from the tiles' counts;
//              active blocks no slot holds are claimed
//              (one claim per block across the batch) and given a slot from
//              the pool's free list
//   k_bdecode  ZFP decode of every claimed block into its slot
//   k_bmc      marching cubes over all entries: the per-query kernel's
//              range-per-CTA count pass, one round trip for the counts of the
//              CTAs before, the list of entries with vertices, a grid barrier
//              (cooperative launch) and the emit shared out over the grid;
//              per-block isovalue, volume and neighbour flags come from the
//              entry's query; every query's vertices come out contiguous and
//              in the plain path's order
//   k_bfinish  per-query vertex offsets and counts
// replayed as one CUDA graph per batch-size bucket.  The host reads the batch
// state once at the end and re-runs only when a capacity was exceeded (entry
// list, slot pool -> eviction of slots the batch does not use, vertex buffer).
#include <algorithm>
#include <map>
#include <memory>
#include <new>
#include <stdexcept>
#include <string>
#include <vector>

#include "active_test.cuh"
#include "bcmc_impl.h"
#include "engine_tuning.h"
#include "mc_common.cuh"
#include "zfp_device.cuh"

namespace bcmc {
namespace {

constexpr int kEngThreads = 256;
constexpr uint32_t kEngTile = 1024;  // blocks per active tile (4 per thread)
// k_bmc CTAs of 8, 16 or 32 "tile blocks", 16 threads to each; 1024 threads per
// SM resident whatever the tile (4 CTAs of 16)
constexpr int kBmcThreadsPerSm = 1024;
constexpr int kBmcMaxPerSm = 2 * kBmcPerSm;  // CTAs per SM asked for at 8 blocks: sizes the MC status words
constexpr uint32_t kMaxVolumes = 4096;

struct EngVolDev {
    const uint64_t* words;
    const float2* ranges;
    const float2* tile_ext;  // extended range of each 1024-block tile
    int32_t* item_slots;     // slot of each block, -1 none, -2 claimed by this batch
    BlockGrid grid;
    uint32_t total;
    uint32_t max_bits;
    SoundRanges sound;
};

struct EngQuery {
    uint32_t vol;
    float iso;
    uint32_t tile0;  // first tile of this query in the batch's tile stream
    uint32_t bit0;   // first word of its active bitmap
};

struct EngResult {
    unsigned long long vstart;
    uint32_t nverts;
    uint32_t nactive;
};

// Batch state: written by the host before a sequence (inputs) and by the
// kernels (counters, outputs), read back once at the end.
struct EngState {
    // inputs
    uint32_t nq, ntiles, entry_capacity, use_epoch;
    unsigned long long vert_capacity, vert_base;
    // device-side
    uint32_t epoch, num_entries, with_verts;  // with_verts: entries with vertices
    uint32_t num_decode, pool_exhausted, entry_overflow, vert_overflow;
    uint32_t error, mc_arrived;  // mc_arrived: k_bmc's grid barrier
    unsigned long long num_verts;  // this sequence's vertices (64-bit, from the per-query totals)
};

// Free list of pool slots: slots free_list[head % cap .. tail % cap) are free.
struct EngPool {
    uint32_t capacity;
    uint32_t head;  // advanced by allocations (may overshoot tail; the host clamps)
    uint32_t tail;  // advanced by evictions
    uint32_t pad;
};

struct BatchArgs {
    const EngVolDev* vols;
    const EngQuery* queries;
    EngResult* results;
    EngState* st;
    EngPool* pool;
    uint32_t* free_list;
    uint32_t* last_use;
    uint32_t* owner_vol;
    uint32_t* owner_block;
    float* cache;
    uint32_t* bitmap;  // a bit per block of every query: active
    uint32_t* live;    // the same: and can have vertices (k_active_words, pipeline.cu)
    uint32_t* ent_id;
    uint32_t* ent_q;
    uint32_t* block_counts;
    uint32_t* wv_list;  // entries with vertices, in entry order (k_bmc)
    uint32_t* wv_off;   // their vertex offsets (32-bit, from vert_base)
    uint32_t* q_nactive;
    uint32_t* q_nverts;
    uint32_t* dec_vol;
    uint32_t* dec_block;
    uint32_t* dec_slot;
    uint2* verts;
    uint32_t* tile_counts;  // live and (from bit 16) active blocks of each tile, then live of each group of tiles
    uint64_t* status_v;  // counts of the MC CTAs (vertices)
    uint64_t* status_b;  // counts of the MC CTAs (entries with vertices)
};

// ---------------------------------------------------------------------------
// volume set-up: extended range of every 1024-block tile
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kEngThreads) k_tile_ext(const float2* __restrict__ ranges, BlockGrid g,
                                                         uint32_t total, float2* __restrict__ ext)
{
    __shared__ float s_lo[kEngThreads / 32], s_hi[kEngThreads / 32];
    const uint32_t tile = blockIdx.x;
    float lo = INFINITY, hi = -INFINITY;
    for (uint32_t i = threadIdx.x; i < kEngTile; i += kEngThreads) {
        const uint32_t b = tile * kEngTile + i;
        if (b >= total) break;
        const uint3 c = block_coords(b, g);
        for (int dz = -1; dz < 2; ++dz)
            for (int dy = -1; dy < 2; ++dy)
                for (int dx = -1; dx < 2; ++dx) {
                    const int x = (int)c.x + dx, y = (int)c.y + dy, z = (int)c.z + dz;
                    if (x < 0 || y < 0 || z < 0 || x >= (int)g.nb.x || y >= (int)g.nb.y || z >= (int)g.nb.z)
                        continue;
                    const float2 r = __ldg(ranges + ((uint32_t)x + g.nb.x * ((uint32_t)y + g.nb.y * (uint32_t)z)));
                    lo = fminf(lo, r.x);  // NaN ranges never make a block active: ignored
                    hi = fmaxf(hi, r.y);
                }
    }
    for (int o = 16; o; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31u) == 0) {
        s_lo[threadIdx.x >> 5] = lo;
        s_hi[threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kEngThreads / 32; ++w) {
            lo = fminf(lo, s_lo[w]);
            hi = fmaxf(hi, s_hi[w]);
        }
        ext[tile] = make_float2(lo, hi);
    }
}

// ---------------------------------------------------------------------------
// k_bbegin
// ---------------------------------------------------------------------------
__global__ void k_bbegin(EngState* st, uint32_t* q_nverts, uint32_t* q_nactive, uint32_t nq)
{
    if (threadIdx.x == 0) {
        st->epoch += 1;
        st->mc_arrived = st->with_verts = 0;
        st->num_entries = st->num_decode = 0;
        st->pool_exhausted = st->entry_overflow = st->vert_overflow = 0;
        st->error = 0;
        st->num_verts = 0;
    }
    for (uint32_t i = threadIdx.x; i < nq; i += blockDim.x) q_nverts[i] = q_nactive[i] = 0;
}

// ---------------------------------------------------------------------------
// k_bactive: the active test of every query over its volume's blocks, a bit per
// block, which of those can have vertices, another, and the counts of the tiles and of groups of eight tiles.
//
// The tests of a batch read each block's range over and over: what bounds the
// kernel is the instructions and loads per block.  A warp takes a tile of 1024
// blocks.  The neighbours of its blocks lie in three runs of ids, one per z:
// the tile moved by a plane, a row and a block longer at either end.  A lane
// reads a block's range once for a run and two ballots make it two bits of a
// word; the words are ORed along x, and a lane ORs the nine (y, z) rows of its
// word of the tile, each two words and a funnel shift (the test in bit words is
// k_active_words', pipeline.cu).  That is 3.4 ranges read per block at 64 blocks
// a row.  Rows longer than kRunRow blocks would make the runs mostly ends: each
// of the nine rows is then a run of its own, 9.1 ranges per block.
// 32 queries over 64^3-block volumes (8.4 M block tests): 23 us, and
// 15 us in k_bentries; 105 us as one kernel that read six ranges of each of the
// nine rows for four blocks and ordered the entries by a look-back over tiles.
// ---------------------------------------------------------------------------
constexpr uint32_t kGroup = kEngThreads / 32;  // tiles of a CTA's turn, a warp each
constexpr uint32_t kRunRow = 256;
constexpr uint32_t kRunWords = (kEngTile + 2 * kRunRow + 2) / 32 + 2;  // 1538 bits that start anywhere in a word
constexpr uint32_t kRunBatch = 10;  // ranges in flight per lane

// The query that tile `tile` of the batch's stream belongs to: the last with
// tile0 <= tile.  A warp's lanes look at 32 queries spread over those that are
// left, which leaves a 32nd of them: three rounds for 32,768 queries.
__device__ __forceinline__ uint32_t find_query(const EngQuery* __restrict__ qs, uint32_t nq, uint32_t tile)
{
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t q0 = 0, left = nq;  // the query is in q0 .. q0 + left - 1
    for (;;) {
        const uint32_t step = div_up(left, 32u), q = lane * step;
        const uint32_t at = __popc(__ballot_sync(0xffffffffu, q < left && __ldg(&qs[q0 + min(q, left - 1u)].tile0) <= tile)) - 1u;
        q0 += at * step;
        if (step == 1u) return q0;
        left = min(step, left - at * step);
    }
}

// Counts of the batch's tiles, then of its groups of tiles.
__device__ __forceinline__ uint32_t* group_counts(const BatchArgs& a, uint32_t ntiles) { return a.tile_counts + ntiles; }

struct RunWords {
    uint2 bits[kRunWords];  // iso >= lo, iso <= hi of the run's blocks
    uint32_t near[3][kRunWords + 1];  // those and their AND, of a block or a neighbour along x
    uint2 up[kRunWords + 1];          // those, of a block or the next along x
};

// Active and live bits of the 32 blocks of the lane's word of the tile that starts at b0.
__device__ __forceinline__ uint2 tile_active(const EngVolDev& V, uint32_t b0, float iso, RunWords& run)
{
    const uint32_t lane = threadIdx.x & 31u, total = V.total, nwords = div_up(total, 32u);
    const uint3 nb = V.grid.nb;
    const int64_t nx = nb.x, nxy = (int64_t)nb.x * nb.y;
    const float2* ranges = V.ranges;
    const uint32_t mine = b0 + 32u * lane;
    const WordRows in_volume = word_rows(min(mine, total - 1u), V.grid, V.sound);
    const int rows = nb.x <= kRunRow ? 3 : 1;  // rows in a run
    uint32_t any_a = 0, any_b = 0, any_c = 0, self_a = 0, self_b = 0, up_a = 0, up_b = 0;
    for (int dz = -1; dz < 2; ++dz)
        for (int dy0 = -1; dy0 < 2; dy0 += rows) {
            // its words: the run's blocks and one more at either end
            const int64_t lo = (int64_t)b0 + dz * nxy + dy0 * nx - 1,
                          hi = (int64_t)b0 + dz * nxy + (dy0 + rows - 1) * nx + kEngTile;
            const int64_t k0 = lo >> 5;
            // of them those that the volume has (the masks let no bit of the others through)
            const int64_t first = max(k0, (int64_t)0), end = min((hi >> 5) + 1, (int64_t)nwords);
            if (first >= end) continue;
            const uint32_t w0 = (uint32_t)(first - k0), n = (uint32_t)(end - k0);
            const int64_t r0 = k0 * 32 + lane;
            for (uint32_t w = w0; w < n; w += kRunBatch) {
                float2 r[kRunBatch];
#pragma unroll
                for (uint32_t u = 0; u < kRunBatch; ++u) {
                    const int64_t b = r0 + 32 * (w + u);
                    r[u] = w + u < n && b < (int64_t)total ? __ldg(ranges + b) : make_float2(NAN, NAN);  // NaN: no bits
                }
                uint2 ab = make_uint2(0u, 0u);
#pragma unroll
                for (uint32_t u = 0; u < kRunBatch; ++u) {
                    const uint32_t wa = __ballot_sync(0xffffffffu, iso >= r[u].x),
                                   wb = __ballot_sync(0xffffffffu, iso <= r[u].y);
                    if (lane == u) ab = make_uint2(wa, wb);
                }
                if (lane < kRunBatch && w + lane < n) run.bits[w + lane] = ab;
            }
            __syncwarp();
            for (uint32_t i = w0 + lane; i < n; i += 32u) {
                const uint2 v = run.bits[i];
                const uint2 p = i > w0 ? run.bits[i - 1u] : make_uint2(0u, 0u),
                            q = i + 1u < n ? run.bits[i + 1u] : make_uint2(0u, 0u);
                const WordEnds ends = word_ends((uint32_t)(k0 + i) * 32u, V.grid);
                run.near[0][i] = ends.spread(v.x, p.x, q.x);
                run.near[1][i] = ends.spread(v.y, p.y, q.y);
                run.near[2][i] = ends.spread(v.x & v.y, p.x & p.y, q.x & q.y);
                run.up[i] = make_uint2(ends.up(v.x, q.x), ends.up(v.y, q.y));
            }
            __syncwarp();
            for (int dy = dy0; dy < dy0 + rows; ++dy) {
                const uint32_t m = in_volume.mask(dy, dz);
                const int64_t s = (int64_t)mine + dz * nxy + dy * nx;
                const uint32_t k = (uint32_t)((s >> 5) - k0), sh = (uint32_t)s & 31u;
                any_a |= __funnelshift_r(run.near[0][k], run.near[0][k + 1u], sh) & m;
                any_b |= __funnelshift_r(run.near[1][k], run.near[1][k + 1u], sh) & m;
                any_c |= __funnelshift_r(run.near[2][k], run.near[2][k + 1u], sh) & m;
                if (dz >= 0 && dy >= 0) {
                    const uint2 l = run.up[k], h = run.up[k + 1u];
                    up_a |= __funnelshift_r(l.x, h.x, sh) & m;
                    up_b |= __funnelshift_r(l.y, h.y, sh) & m;
                }
                if (dz == 0 && dy == 0) {
                    self_a = run.bits[k].x;
                    self_b = run.bits[k].y;
                }
            }
            __syncwarp();
        }
    uint32_t act = mine >= total ? 0u : (self_a & any_b) | (self_b & any_a) | any_c;
    if (total - mine < 32u) act &= (1u << (total - mine)) - 1u;
    uint32_t sound = mine < V.sound.id ? in_volume.sound : 0u;
    if (V.sound.id - mine < 32u) sound &= (1u << (V.sound.id - mine)) - 1u;
    return make_uint2(act, act & ((up_a & up_b) | ~sound));
}

// Claims for this batch those of a warp's blocks b[0 .. kN) that no slot held
// (`open`, bit j for b[j]), and gives them slots from the free list; when the
// pool has no free slot the claims are released and the batch flagged (the host
// evicts and re-runs).  A claim is a chain of four round trips, so a warp takes
// the slots and the decode list's places of all its claims at once
// (k_bentries of a
// first batch, all of whose blocks are new: 130 -> 57 us; of one with a few: 48 -> 29 us).
template <int kN>
__device__ __forceinline__ void claim_blocks(const BatchArgs& a, uint32_t v, int32_t* item_slots, const uint32_t b[kN],
                                             uint32_t open, uint32_t use_epoch)
{
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    uint32_t won = 0, n = 0, at[kN];
#pragma unroll
    for (int j = 0; j < kN; ++j)  // not: cached meanwhile, or claimed by another query
        if (open >> j & 1u) won |= (atomicCAS(item_slots + b[j], -1, -2) == -1 ? 1u : 0u) << j;
#pragma unroll
    for (int j = 0; j < kN; ++j) {
        const uint32_t m = __ballot_sync(0xffffffffu, won >> j & 1u);
        at[j] = n + __popc(m & below);
        n += __popc(m);
    }
    if (!n) return;
    EngPool* pool = a.pool;
    uint32_t head = 0, tail = 0, d = 0;
    if (lane == 0) {
        tail = *(volatile uint32_t*)&pool->tail;
        head = atomicAdd(&pool->head, n);
    }
    head = __shfl_sync(0xffffffffu, head, 0);
    tail = __shfl_sync(0xffffffffu, tail, 0);
    const int32_t free_slots = (int32_t)(tail - head);
    const uint32_t got = free_slots <= 0 ? 0u : min(n, (uint32_t)free_slots);
    uint32_t slot[kN];
#pragma unroll
    for (int j = 0; j < kN; ++j)
        slot[j] = (won >> j & 1u) && at[j] < got ? __ldg(a.free_list + (head + at[j]) % pool->capacity) : 0u;
    if (lane == 0) {
        if (got) d = atomicAdd(&a.st->num_decode, got);
        if (got < n) atomicOr(&a.st->pool_exhausted, 1u);
    }
    d = __shfl_sync(0xffffffffu, d, 0);
#pragma unroll
    for (int j = 0; j < kN; ++j) {
        if (!(won >> j & 1u)) continue;
        if (at[j] < got) {
            a.last_use[slot[j]] = use_epoch;
            a.dec_vol[d + at[j]] = v;
            a.dec_block[d + at[j]] = b[j];
            a.dec_slot[d + at[j]] = slot[j];
        } else {
            atomicExch(item_slots + b[j], -1);  // no free slot: release the claim
        }
    }
}

// The entries of a tile of query qi, the first at `at`, and the claims of its blocks:
// `word` and `live` are the lane's words of the tile.  Words without an active block
// are passed over, four of the others are taken at a time, their blocks' slots read
// together.
__device__ __forceinline__ void tile_entries(const BatchArgs& a, uint32_t qi, const EngQuery& Q, uint32_t tile, uint32_t word,
                                             uint32_t live, uint32_t at, uint32_t cap, uint32_t use_epoch)
{
    constexpr int kN = 4;
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    const uint32_t b0 = (tile - Q.tile0) * kEngTile + lane;
    int32_t* item_slots = a.vols[Q.vol].item_slots;
    const uint32_t n = __popc(live), first = at + warp_inclusive_scan(n) - n;  // of the lane's word
    for (uint32_t some = __ballot_sync(0xffffffffu, word != 0u); some;) {
        uint32_t i[kN], w[kN], b[kN], open = 0;
        int32_t s[kN];
#pragma unroll
        for (int j = 0; j < kN; ++j) {
            i[j] = some ? (uint32_t)__ffs(some) - 1u : 32u;
            some &= some - 1u;
            w[j] = __shfl_sync(0xffffffffu, word, i[j]);
            if (i[j] == 32u) w[j] = 0u;
            b[j] = b0 + 32u * i[j];
            s[j] = w[j] >> lane & 1u ? *(volatile int32_t*)(item_slots + b[j]) : -2;
        }
#pragma unroll
        for (int j = 0; j < kN; ++j) {
            const uint32_t l = __shfl_sync(0xffffffffu, live, i[j]), f = __shfl_sync(0xffffffffu, first, i[j]);
            if (w[j] >> lane & 1u) {
                const uint32_t pos = f + __popc(l & below);
                if ((l >> lane & 1u) && pos < cap) {
                    a.ent_id[pos] = b[j];
                    a.ent_q[pos] = qi;
                }
                if (s[j] >= 0) a.last_use[s[j]] = use_epoch;
                open |= (s[j] == -1 ? 1u : 0u) << j;
            }
        }
        if (__any_sync(0xffffffffu, open)) claim_blocks<kN>(a, Q.vol, item_slots, b, open, use_epoch);
    }
}

// A batch of one group of tiles is one CTA's: its warps have the words and the counts
// at hand and go on to the entries themselves, and k_bentries is not launched.  With
// the runs' missing words left out and the words without active blocks passed over,
// single queries on 8^3 volumes 40.7 -> 31.9 us on the device, on 48^3 44.0 -> 39.8,
// four on 32^3 42.7 -> 38.3.
__global__ void __launch_bounds__(kEngThreads, 3) k_bactive(BatchArgs a)
{
    __shared__ RunWords s_run[kGroup];
    __shared__ uint32_t s_count[2][kGroup];
    EngState* st = a.st;
    const uint32_t ntiles = st->ntiles, nq = st->nq, ngroups = div_up(ntiles, kGroup);
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t turn = 0;
    for (uint32_t g = blockIdx.x; g < ngroups; g += gridDim.x, turn ^= 1u) {
        const uint32_t tile = g * kGroup + warp;
        uint32_t count = 0, qi = 0;
        EngQuery Q{};
        uint2 w = make_uint2(0u, 0u);
        if (tile < ntiles) {
            qi = find_query(a.queries, nq, tile);
            Q = a.queries[qi];
            const EngVolDev& V = a.vols[Q.vol];
            const uint32_t lt = tile - Q.tile0;
            const float2 ext = __ldg(V.tile_ext + lt);
            if (Q.iso >= ext.x && Q.iso <= ext.y) w = tile_active(V, lt * kEngTile, Q.iso, s_run[warp]);
            a.bitmap[Q.bit0 + lt * (kEngTile / 32) + lane] = w.x;
            a.live[Q.bit0 + lt * (kEngTile / 32) + lane] = w.y;
            count = __reduce_add_sync(0xffffffffu, __popc(w.y) + ((uint32_t)__popc(w.x) << 16));
            if (lane == 0) a.tile_counts[tile] = count;
        }
        if (lane == 0) s_count[turn][warp] = count & 0xffffu;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t sum = 0;
            for (uint32_t w = 0; w < kGroup; ++w) sum += s_count[turn][w];
            group_counts(a, ntiles)[g] = sum;
        }
        if (ngroups > 1u) continue;
        const uint32_t cap = st->entry_capacity, n = lane < kGroup ? s_count[turn][lane] : 0u;
        const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? n : 0u), all = __reduce_add_sync(0xffffffffu, n);
        if (count >> 16) {
            if (lane == 0) atomicAdd(a.q_nactive + qi, count >> 16);
            tile_entries(a, qi, Q, tile, w.x, w.y, before, cap, st->use_epoch);
        }
        if (threadIdx.x == 0) {
            st->num_entries = all;
            if (all > cap) st->entry_overflow = 1;
        }
    }
}

// ---------------------------------------------------------------------------
// k_bentries: the live (block, query) entries in the order of the tile stream,
// and the claims of the active blocks that no slot holds
//
// A CTA owns a contiguous range of groups of tiles.  Every count is known, so
// it adds up those of the groups before its range and waits for nobody; a warp
// takes a tile of a group, whose words' bits say where each entry goes.  (Not
// launched for a batch of one group, whose entries k_bactive makes.)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kEngThreads) k_bentries(BatchArgs a)
{
    __shared__ uint32_t s_sum;
    EngState* st = a.st;
    const uint32_t ntiles = st->ntiles, nq = st->nq, cap = st->entry_capacity, use_epoch = st->use_epoch;
    const uint32_t ngroups = div_up(ntiles, kGroup), per = div_up(ngroups, gridDim.x);
    const uint32_t first = blockIdx.x * per, end = min(ngroups, first + per);
    if (first >= ngroups) return;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t* groups = group_counts(a, ntiles);
    if (threadIdx.x == 0) s_sum = 0;
    __syncthreads();
    uint32_t sum = 0;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < first; i += kEngThreads) sum += __ldg(groups + i);
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0 && sum) atomicAdd(&s_sum, sum);
    __syncthreads();
    uint32_t base = s_sum;
    for (uint32_t g = first; g < end; ++g) {
        const uint32_t t0 = g * kGroup, tile = t0 + warp;
        const uint32_t n2 = lane < kGroup && t0 + lane < ntiles ? __ldg(a.tile_counts + t0 + lane) : 0u, n = n2 & 0xffffu;
        const uint32_t before = __reduce_add_sync(0xffffffffu, lane < warp ? n : 0u);
        const uint32_t count = __shfl_sync(0xffffffffu, n2, warp) >> 16;  // active
        const uint32_t at = base + before;
        base += __reduce_add_sync(0xffffffffu, n);
        if (!count) continue;
        const uint32_t qi = find_query(a.queries, nq, tile);
        const EngQuery Q = a.queries[qi];
        const uint32_t at32 = Q.bit0 + (tile - Q.tile0) * (kEngTile / 32) + lane;
        const uint32_t word = __ldg(a.bitmap + at32), live = __ldg(a.live + at32);
        if (lane == 0) atomicAdd(a.q_nactive + qi, count);
        tile_entries(a, qi, Q, tile, word, live, at, cap, use_epoch);
    }
    if (end == ngroups && threadIdx.x == 0) {
        st->num_entries = base;
        if (base > cap) st->entry_overflow = 1;
    }
}

// ---------------------------------------------------------------------------
// k_bdecode: claimed blocks into their slots, then publish the slot
// ---------------------------------------------------------------------------
// Volumes of a batch differ in rate: the staged words of one CTA are laid out
// at the largest rate of the resident volumes (`max_rate` u64 words per block).

template <int kThreads>
__global__ void __launch_bounds__(kThreads, 640 / kThreads) k_bdecode(BatchArgs a, uint32_t max_rate)
{
    extern __shared__ __align__(16) uint32_t s_words[];
    uint32_t* pl = zfp_stage_planes(s_words, kThreads, max_rate);
    if (threadIdx.x < 4) s_words[kThreads * 2u * max_rate + threadIdx.x] = 0u;
    const uint32_t n = a.st->num_decode;
    for (uint32_t i0 = blockIdx.x * kThreads; i0 < n; i0 += gridDim.x * kThreads) {
        const uint32_t i = i0 + threadIdx.x;
        uint32_t v = 0, b = 0, slot = 0;
        __syncthreads();
        if (i < n) {
            v = a.dec_vol[i];
            b = a.dec_block[i];
            slot = a.dec_slot[i];
            const EngVolDev& V = a.vols[v];
            // this thread's slot of the staged words, at the CTA's stride
            uint2* dst = reinterpret_cast<uint2*>(s_words + threadIdx.x * 2u * max_rate);
            const uint32_t rate = V.max_bits / 64u;
            for (uint32_t k = 0; k < rate; ++k) {
                const uint64_t x = __ldg(V.words + (uint64_t)b * rate + k);
                dst[k] = make_uint2((uint32_t)x, (uint32_t)(x >> 32));
            }
        }
        __syncthreads();
        if (i >= n) continue;
        const EngVolDev& V = a.vols[v];
        float out[64];
        zfp_decode_staged(s_words + threadIdx.x * 2u * max_rate, V.max_bits, pl, out);
        float4* d4 = reinterpret_cast<float4*>(a.cache + (uint64_t)slot * 64u);
#pragma unroll
        for (int k = 0; k < 16; ++k) d4[k] = make_float4(out[4 * k], out[4 * k + 1], out[4 * k + 2], out[4 * k + 3]);
        a.owner_vol[slot] = v;
        a.owner_block[slot] = b;
        V.item_slots[b] = (int32_t)slot;
    }
}

// The autotuner's decode probe: k_bdecode's inner loop into a scratch buffer.
template <int kThreads>
__global__ void __launch_bounds__(kThreads, 640 / kThreads) k_decode_probe(const uint64_t* __restrict__ words, uint32_t rate,
                                                           uint32_t n, float* __restrict__ scratch)
{
    extern __shared__ __align__(16) uint32_t s_words[];
    uint32_t* pl = zfp_stage_planes(s_words, kThreads, rate);
    const uint32_t wb = threadIdx.x & ~31u;
    for (uint32_t i0 = blockIdx.x * kThreads; i0 < n; i0 += gridDim.x * kThreads) {
        const uint32_t nb = n - i0 < (uint32_t)kThreads ? n - i0 : (uint32_t)kThreads;
        __syncthreads();
        zfp_stage_run(words, i0, nb, rate, s_words);
        __syncthreads();
        if (wb >= nb) continue;
        const bool mine = threadIdx.x < nb;
        float out[64];
        if (mine) zfp_decode_staged(s_words + threadIdx.x * 2u * rate, 64u * rate, pl, out);
        zfp_store_warp(pl, out, mine, scratch + (uint64_t)(i0 + wb) * 64u, nb - wb);
    }
}

// ---------------------------------------------------------------------------
// k_bmc: the per-query MC kernel (pipeline.cu, k_mc) over a batch's entries:
// the same warp work (mc_common.cuh), the isovalue, volume and neighbour flags
// taken from each entry's query, and the emit always shared out over the grid
// ---------------------------------------------------------------------------
template <int kTileBlocks>
__global__ void __launch_bounds__(16 * kTileBlocks, kBmcThreadsPerSm / (16 * kTileBlocks)) k_bmc(BatchArgs a)
{
    constexpr int kThreads = 16 * kTileBlocks, kWarps = kThreads / 32;
    extern __shared__ __align__(16) unsigned char s_dyn[];
    McShared<kThreads, false>& sm = *reinterpret_cast<McShared<kThreads, false>*>(s_dyn);
    __shared__ uint32_t s_warp[kWarps + 1];
    __shared__ uint32_t s_pv, s_pb, s_cta_v, s_cta_b;

    EngState* st = a.st;
    const uint32_t A = min(st->num_entries, st->entry_capacity);
    if (A == 0 || st->entry_overflow || st->pool_exhausted) return;
    const uint32_t epoch = st->epoch;
    const uint64_t cap = st->vert_capacity, vbase = st->vert_base;
    const uint32_t slots = a.pool->capacity;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5, jb = lane >> 3;
    const uint32_t G = gridDim.x, rank = blockIdx.x;
    // whole batches for every warp: up to kMcBlocks blocks each, or a multiple of a batch
    const uint32_t share = div_up(A, G);
    const uint32_t range = align_up(share, share <= kWarps * kMcBlocks ? (uint32_t)kWarps : kMcBlocks);
    const uint32_t start = min(A, rank * range), end = min(A, start + range);
    // ranks 0 .. worked - 1 own entries; the others only help with the emit
    const uint32_t worked = div_up(A, range);
    mc_shared_begin(sm);
    if (t == 0) s_cta_v = s_cta_b = s_pv = s_pb = 0;
    const McLane geo = mc_lane(a.cache, sm.warp[warp].slot);
    McWarpMem<false>& mem = sm.warp[warp];

    // an entry: its block, its query, and the query's isovalue
    struct Entry {
        uint32_t id, qi;
    };
    struct Look {
        McLook l;
        uint32_t qi;
        float iso;
    };
    const auto load = [&](bool valid, uint32_t e) {
        return valid ? Entry{__ldg(a.ent_id + e), __ldg(a.ent_q + e)} : Entry{0u, 0u};
    };
    const auto look = [&](bool valid, const Entry& e) {
        const EngQuery* Q = a.queries + e.qi;
        const EngVolDev& V = a.vols[__ldg(&Q->vol)];
        const uint32_t* bits = a.bitmap + __ldg(&Q->bit0);
        return Look{mc_look(valid, e.id, V.grid, V.item_slots,
                            [&](uint32_t nid) { return __ldg(bits + (nid >> 5)) >> (nid & 31u) & 1u; }),
                    e.qi, __ldg(&Q->iso)};
    };
    const auto look_end = [&](const Look& l) {
        uint32_t has;
        mc_look_end(l.l, sm.tab, slots, &st->error, 62u, mem.slot, has);
        return has;
    };

    // ---- count pass: entries two rounds ahead, lookups one round ahead
    {
        const uint32_t batch = min(kMcBlocks, max(range / kWarps, 1u)), step = kWarps * batch;
        uint32_t base = start + warp * batch;
        const auto mine = [&](uint32_t at) { return jb < batch && at + jb < end; };
        Look next = look(mine(base), load(mine(base), base + jb));
        Entry e2 = load(mine(base + step), base + step + jb);
        uint32_t wv = 0, wb = 0;
        uint32_t cur = 0xffffffffu, cur_v = 0;  // the query being added up (one atomic per warp and run of a query)
        async_wait<1>();
        __syncthreads();
        for (; base < end; base += step) {
            const uint32_t n = min(batch, end - base), qi = next.qi;
            const float iso = next.iso;
            const uint32_t has = look_end(next);
            uint32_t total = 0;
            float f[kMcBlocks][4];
            mc_voxels(geo, n, f);
            next = look(mine(base + step), e2);
            e2 = load(mine(base + 2u * step), base + 2u * step + jb);
#pragma unroll
            for (uint32_t j = 0; j < kMcBlocks; ++j)
                if (j < n) {
                    uint32_t c0, c1;
                    if (!mc_cases<true>(geo, f[j], __shfl_sync(kFull, iso, 8u * j), __shfl_sync(kFull, has, 8u * j), c0, c1))
                        continue;
                    const uint32_t v = 3u * __reduce_add_sync(kFull, (uint32_t)sm.tab.count.n[c0] + sm.tab.count.n[c1]);
                    if (lane == j) total = v;
                    wv += v;
                    wb += v != 0u ? 1u : 0u;
                    const uint32_t qj = __shfl_sync(kFull, qi, 8u * j);
                    if (qj != cur) {
                        if (cur_v && lane == 0) atomicAdd(a.q_nverts + cur, cur_v);
                        cur = qj;
                        cur_v = 0;
                    }
                    cur_v += v;
                }
            if (lane < n) a.block_counts[base + lane] = total;
        }
        if (lane == 0 && wb) {
            if (cur_v) atomicAdd(a.q_nverts + cur, cur_v);
            atomicAdd(&s_cta_v, wv);
            atomicAdd(&s_cta_b, wb);
        }
    }
    __syncthreads();
    if (rank < worked)
        cta_prefix_sums<kThreads>({{a.status_v, s_cta_v, 61u, &s_pv}, {a.status_b, s_cta_b, 64u, &s_pb}}, rank, epoch,
                                  &st->error);
    async_wait<0>();
    __syncthreads();
    // 32-bit prefix: a sequence over 2^32 vertices wraps here; k_bfinish
    // detects it from the 64-bit per-query totals and the host splits
    uint32_t pv = s_pv, pb = s_pb;
    if (rank == worked - 1 && t == 0) st->with_verts = pb + s_cta_b;
    const bool fits = vbase + pv + s_cta_v <= cap;
    if (!fits && t == 0) atomicOr(&st->vert_overflow, 1u);
    // the range's entries with vertices: list positions and vertex offsets
    if (fits)
        for (uint32_t b0 = start; b0 < end; b0 += kThreads) {
            const uint32_t i = b0 + t;
            const uint32_t c = i < end ? a.block_counts[i] : 0u;  // <= 64 cells x 15 vertices
            uint32_t v, w;
            const uint32_t ex_v = cta_exclusive_scan<kThreads>(c, s_warp, &v);
            const uint32_t ex_w = cta_exclusive_scan<kThreads>(c ? 1u : 0u, s_warp, &w);
            if (c) {
                a.wv_list[pb + ex_w] = i;
                a.wv_off[pb + ex_w] = pv + ex_v;
            }
            pv += v;
            pb += w;
        }
    grid_barrier(&st->mc_arrived, G, &st->error, 65u);
    if (__ldcg(&st->error) | __ldcg(&st->vert_overflow)) return;
    // emit: runs of `per` list entries, warp by warp over the whole grid; a
    // run's list entries are read two runs ahead, its neighbours one run ahead
    const uint32_t W = __ldcg(&st->with_verts);
    const uint32_t per = min(kMcBlocks, div_up(W, G * kWarps)), step = G * kWarps * per;
    const auto mine = [&](uint32_t at) { return jb < per && at + jb < W; };
    const auto load_entry = [&](uint32_t at) { return mine(at) ? __ldcg(a.wv_list + at + jb) : 0u; };
    uint32_t at = (rank * kWarps + warp) * per;
    if (at >= W) return;
    Look next = look(mine(at), load(mine(at), load_entry(at)));
    uint32_t entry = load_entry(at + step), off = __ldcg(a.wv_off + at);
    for (; at < W; at += step) {
        const uint32_t n = min(per, W - at), id = next.l.id, at1 = at + step;
        const float iso = next.iso;
        const uint32_t has = look_end(next);
        mc_grids(geo, mem, n);
        McSink<false> sink{a.verts + vbase + off};
        const Entry e1 = load(mine(at1), entry);
        entry = load_entry(at1 + step);
        off = at1 < W ? __ldcg(a.wv_off + at1) : 0u;
        mc_emit<false, false>(geo, sm.tab, mem, n, id, has, iso, sink, [&] { next = look(mine(at1), e1); });
    }
}

// ---------------------------------------------------------------------------
// k_bfinish: per-query results (one CTA; queries in order)
// ---------------------------------------------------------------------------
constexpr int kFinThreads = 1024;
__global__ void __launch_bounds__(kFinThreads) k_bfinish(BatchArgs a)
{
    __shared__ unsigned long long s_sum[kFinThreads / 32 + 1];
    EngState* st = a.st;
    const uint32_t nq = st->nq;
    const uint64_t vbase = st->vert_base;
    unsigned long long carry = 0;
    for (uint32_t b0 = 0; b0 < nq; b0 += kFinThreads) {
        const uint32_t i = b0 + threadIdx.x;
        const unsigned long long v = i < nq ? a.q_nverts[i] : 0ull;
        // inclusive scan in 64 bits: warp shuffles, then the warp totals
        unsigned long long x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
            if ((threadIdx.x & 31u) >= (uint32_t)o) x += y;
        }
        if ((threadIdx.x & 31u) == 31u) s_sum[threadIdx.x >> 5] = x;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned long long r = 0;
            for (int w = 0; w < kFinThreads / 32; ++w) {
                const unsigned long long tw = s_sum[w];
                s_sum[w] = r;
                r += tw;
            }
            s_sum[kFinThreads / 32] = r;
        }
        __syncthreads();
        const unsigned long long excl = carry + s_sum[threadIdx.x >> 5] + x - v;
        if (i < nq) {
            EngResult r;
            r.vstart = vbase + excl;
            r.nverts = (uint32_t)v;
            r.nactive = a.q_nactive[i];
            a.results[i] = r;
        }
        carry += s_sum[kFinThreads / 32];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        st->num_verts = carry;
        if (vbase + carry > st->vert_capacity || carry >= (1ull << 32)) st->vert_overflow = 1;
    }
}

// ---------------------------------------------------------------------------
// k_bevict: free every slot the current batch does not use
// ---------------------------------------------------------------------------
__global__ void k_bevict(BatchArgs a, uint32_t use_epoch, uint32_t nslots, unsigned long long* evicted)
{
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < nslots; s += gridDim.x * blockDim.x) {
        const uint32_t v = a.owner_vol[s];
        if (v == 0xffffffffu || a.last_use[s] == use_epoch) continue;
        a.vols[v].item_slots[a.owner_block[s]] = -1;
        a.owner_vol[s] = 0xffffffffu;
        const uint32_t pos = atomicAdd(&a.pool->tail, 1u);
        a.free_list[pos % a.pool->capacity] = s;
        atomicAdd(evicted, 1ull);
    }
}

__global__ void k_fill_u32(uint32_t* p, uint64_t n, uint32_t v)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        p[i] = v;
}
__global__ void k_iota(uint32_t* p, uint32_t n)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = i;
}

}  // namespace
}  // namespace bcmc

using namespace bcmc;

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
struct EngVolume {
    uint32_t dims[3];
    uint32_t rate;
    uint64_t* words = nullptr;
    size_t words_bytes = 0;
    float2* ranges = nullptr;
    float2* tile_ext = nullptr;
    int32_t* item_slots = nullptr;
    uint32_t total = 0, tiles = 0;
    BlockGrid grid;
};

// The buffers of one batch in flight.  Two lanes let the server keep two
// batches on the device at once: the next batch's active test, claims and
// decode (phase 1) run while the current batch's marching cubes (phase 2) do.
struct EngLane {
    bool ready = false;  // buffers allocated
    EngQuery* d_queries = nullptr;
    EngQuery* h_queries = nullptr;  // pinned
    EngResult* d_results = nullptr;
    EngResult* h_results = nullptr;  // pinned
    EngState* d_st = nullptr;
    EngState* h_st = nullptr;  // pinned
    uint32_t *q_nactive = nullptr, *q_nverts = nullptr;
    uint32_t* bitmap = nullptr;
    uint64_t bitmap_words = 0;  // of the active bits, and as many of the live ones after them
    uint32_t *ent_id = nullptr, *ent_q = nullptr, *block_counts = nullptr, *wv_list = nullptr, *wv_off = nullptr;
    uint32_t entry_cap = 0;
    uint2* verts = nullptr;
    uint64_t vert_cap = 0, vert_used = 0;
    uint64_t* status = nullptr;
    uint64_t status_words = 0;
    uint64_t status_a_words = 0;
    uint64_t epoch_calls = 0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    // one graph per batch-size bucket and number of tile groups, one or more (graph_key),
    // rebuilt when buffers move
    struct Graph {
        cudaGraphExec_t exec = nullptr;        // the whole sequence on one stream
        cudaGraphExec_t front = nullptr;       // phase 1 (pipelined runs)
        cudaGraphExec_t back = nullptr;        // phase 2 (pipelined runs)
        uint32_t kernels = 0, split_kernels = 0;  // in exec, in front and back
        uint64_t generation = 0, split_generation = 0;
        int cfg_key = -1, split_cfg_key = -1;  // the launch parameters they were captured with
    };
    std::map<uint32_t, Graph> graphs;
    uint64_t generation = 1;
    // pipelined batch in flight on this lane
    cudaEvent_t ev_front = nullptr;  // its phase 1 finished
    cudaEvent_t ev_done = nullptr;   // its phase 2 and the state copies finished
    bool in_flight = false;
    uint32_t batch_epoch = 0;        // use epoch of its sequence (protected from eviction)
    uint32_t n = 0, bucket = 0;
    std::vector<bcmc_query> queries;
};

struct bcmc_engine {
    bcmc_ctx* ctx = nullptr;
    cudaStream_t stream = nullptr;       // every synchronous run; phase 1 of pipelined runs
    cudaStream_t stream_back = nullptr;  // phase 2 of pipelined runs
    cudaStream_t stream_copy = nullptr;  // vertex copies of completed pipelined batches
    bcmc_engine_opts opts{};
    std::vector<EngVolume> vols;
    EngVolDev* d_vols = nullptr;
    uint32_t d_vols_cap = 0;
    // pool
    uint64_t pool_slots = 0;
    float* cache = nullptr;
    uint32_t *free_list = nullptr, *last_use = nullptr, *owner_vol = nullptr, *owner_block = nullptr;
    EngPool* d_pool = nullptr;
    EngPool* h_pool = nullptr;
    unsigned long long* d_evicted = nullptr;
    // the decode list of a sequence's claims: written and read in phase 1 only,
    // which runs one batch at a time, so both lanes share it
    uint32_t *dec_vol = nullptr, *dec_block = nullptr, *dec_slot = nullptr;
    uint32_t dec_cap = 0;
    uint32_t max_batch = 0;
    uint32_t max_rate = 1;  // largest rate of the resident volumes (k_bdecode's staging stride)
    uint32_t use_epoch = 0;
    EngLane lanes[2];
    EngLane* L = &lanes[0];  // the lane the next sequence runs on, and whose vertices the API returns
    std::map<uint32_t, EngConfig> tuned;  // per bucket
    EngConfig cfg;                        // of the sequence being enqueued
    bcmc_engine_stats stats{};
    uint64_t overlapped = 0;  // pipelined batches launched while another was in flight
};

namespace {

int eng_grid_mc_max(bcmc_engine* e) { return e->ctx->num_sms * kBmcMaxPerSm; }  // sizes the status words
// k_bmc<kB> CTAs resident per SM: the bound of its cooperative grid
template <int kB>
int bmc_resident()
{
    static const int n = [] {
        constexpr size_t smem = sizeof(McShared<16 * kB, false>);
        allow_smem(k_bmc<kB>, smem);
        int r = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, k_bmc<kB>, 16 * kB, smem) != cudaSuccess || r < 1) r = 1;
        return r;
    }();
    return n;
}
int bmc_resident(int mc_blocks)
{
    return mc_blocks == 8 ? bmc_resident<8>() : (mc_blocks == 32 ? bmc_resident<32>() : bmc_resident<16>());
}
int eng_grid_mc(bcmc_engine* e) { return e->ctx->num_sms * mc_ctas(e->cfg, bmc_resident(e->cfg.mc_blocks)); }
int eng_grid_act(bcmc_engine* e) { return e->ctx->num_sms * e->cfg.act_per_sm; }
int eng_grid_dec(bcmc_engine* e) { return e->ctx->num_sms * e->cfg.dec_per_sm; }

template <typename T>
void eng_realloc(bcmc_engine* e, T*& p, uint64_t old_n, uint64_t new_n)
{
    dev_free(e->ctx, p, old_n * sizeof(T));
    p = nullptr;
    p = (T*)dev_alloc(e->ctx, new_n * sizeof(T));
}

BatchArgs eng_args(bcmc_engine* e)
{
    BatchArgs a;
    a.vols = e->d_vols;
    a.queries = e->L->d_queries;
    a.results = e->L->d_results;
    a.st = e->L->d_st;
    a.pool = e->d_pool;
    a.free_list = e->free_list;
    a.last_use = e->last_use;
    a.owner_vol = e->owner_vol;
    a.owner_block = e->owner_block;
    a.cache = e->cache;
    a.bitmap = e->L->bitmap;
    a.live = e->L->bitmap + e->L->bitmap_words;
    a.ent_id = e->L->ent_id;
    a.ent_q = e->L->ent_q;
    a.block_counts = e->L->block_counts;
    a.wv_list = e->L->wv_list;
    a.wv_off = e->L->wv_off;
    a.q_nactive = e->L->q_nactive;
    a.q_nverts = e->L->q_nverts;
    a.dec_vol = e->dec_vol;
    a.dec_block = e->dec_block;
    a.dec_slot = e->dec_slot;
    a.verts = e->L->verts;
    a.tile_counts = reinterpret_cast<uint32_t*>(e->L->status);  // two words to a tile: the groups fit as well
    a.status_v = e->L->status + e->L->status_a_words;
    a.status_b = a.status_v + eng_grid_mc_max(e) + 1;
    return a;
}

void eng_ensure_status(bcmc_engine* e, uint64_t active_tiles)
{
    const uint64_t need_a = std::max<uint64_t>(active_tiles + 1, 1024);
    const uint64_t mc_words = 2 * ((uint64_t)eng_grid_mc_max(e) + 1);  // status_v, status_b
    const uint64_t need = need_a + mc_words;
    if (need_a <= e->L->status_a_words && need <= e->L->status_words) return;
    BCMC_CUDA(cudaStreamSynchronize(e->stream));
    const uint64_t words = std::max<uint64_t>(need_a * 2, 4096) + mc_words;
    eng_realloc(e, e->L->status, e->L->status_words, words);
    BCMC_CUDA(cudaMemsetAsync(e->L->status, 0, words * 8, e->stream));
    e->L->status_words = words;
    e->L->status_a_words = words - mc_words;
    ++e->L->generation;
}

// Every 2^26 sequences the look-back epoch restarts over cleared status words.
void eng_epoch_tick(bcmc_engine* e)
{
    if (++e->L->epoch_calls < (1ull << 26)) return;
    BCMC_CUDA(cudaMemsetAsync(e->L->status, 0, e->L->status_words * 8, e->stream));
    BCMC_CUDA(cudaMemsetAsync(&e->L->d_st->epoch, 0, 4, e->stream));
    e->L->epoch_calls = 0;
}

void eng_upload_vols(bcmc_engine* e)
{
    const uint32_t n = (uint32_t)e->vols.size();
    if (n > e->d_vols_cap) {
        eng_realloc(e, e->d_vols, e->d_vols_cap, std::max<uint32_t>(n * 2, 8));
        e->d_vols_cap = std::max<uint32_t>(n * 2, 8);
        for (EngLane& l : e->lanes) ++l.generation;
    }
    std::vector<EngVolDev> h(n);
    for (uint32_t i = 0; i < n; ++i) {
        const EngVolume& v = e->vols[i];
        h[i] = EngVolDev{v.words, v.ranges, v.tile_ext, v.item_slots, v.grid, v.total, 64u * v.rate,
                         sound_ranges(v.dims, v.grid, zfp_ranged_blocks(e->ctx, v.dims))};
    }
    BCMC_CUDA(cudaMemcpyAsync(e->d_vols, h.data(), n * sizeof(EngVolDev), cudaMemcpyHostToDevice, e->stream));
    BCMC_CUDA(cudaStreamSynchronize(e->stream));
}

void eng_alloc_pool(bcmc_engine* e, uint64_t slots)
{
    if (slots == 0 || slots > 0xffffffffull) throw std::invalid_argument("pool_slots out of range");
    e->pool_slots = slots;
    e->cache = (float*)dev_alloc(e->ctx, slots * 256);
    e->free_list = (uint32_t*)dev_alloc(e->ctx, slots * 4);
    e->last_use = (uint32_t*)dev_alloc(e->ctx, slots * 4);
    e->owner_vol = (uint32_t*)dev_alloc(e->ctx, slots * 4);
    e->owner_block = (uint32_t*)dev_alloc(e->ctx, slots * 4);
    // every successful claim of a batch takes a free slot: the decode list
    // never needs more entries than the pool has slots
    e->dec_vol = (uint32_t*)dev_alloc(e->ctx, slots * 4);
    e->dec_block = (uint32_t*)dev_alloc(e->ctx, slots * 4);
    e->dec_slot = (uint32_t*)dev_alloc(e->ctx, slots * 4);
    e->dec_cap = (uint32_t)slots;
    const int grid = e->ctx->num_sms * 8;
    k_iota<<<grid, 256, 0, e->stream>>>(e->free_list, (uint32_t)slots);
    k_fill_u32<<<grid, 256, 0, e->stream>>>(e->owner_vol, slots, 0xffffffffu);
    k_fill_u32<<<grid, 256, 0, e->stream>>>(e->last_use, slots, 0u);
    count_launches(3);
    e->h_pool->capacity = (uint32_t)slots;
    e->h_pool->head = 0;
    e->h_pool->tail = (uint32_t)slots;
    BCMC_CUDA(cudaMemcpyAsync(e->d_pool, e->h_pool, sizeof(EngPool), cudaMemcpyHostToDevice, e->stream));
    BCMC_CUDA(cudaStreamSynchronize(e->stream));
    for (EngLane& l : e->lanes) ++l.generation;
}

void eng_ensure_batch(bcmc_engine* e, uint64_t bitmap_words, uint32_t entries)
{
    if (bitmap_words > e->L->bitmap_words) {
        BCMC_CUDA(cudaStreamSynchronize(e->stream));
        const uint64_t n = std::max<uint64_t>(bitmap_words + bitmap_words / 2, 1u << 16);
        eng_realloc(e, e->L->bitmap, 2 * e->L->bitmap_words, 2 * n);
        e->L->bitmap_words = n;
        ++e->L->generation;
    }
    if (entries > e->L->entry_cap) {
        BCMC_CUDA(cudaStreamSynchronize(e->stream));
        const uint64_t n64 = std::min<uint64_t>((uint64_t)entries + entries / 2, 0xffffffffull);
        const uint32_t n = (uint32_t)std::max<uint64_t>(n64, 1u << 16);
        eng_realloc(e, e->L->ent_id, e->L->entry_cap, n);
        eng_realloc(e, e->L->ent_q, e->L->entry_cap, n);
        eng_realloc(e, e->L->block_counts, e->L->entry_cap, n);
        eng_realloc(e, e->L->wv_list, e->L->entry_cap, n);
        eng_realloc(e, e->L->wv_off, e->L->entry_cap, n);
        e->L->entry_cap = n;
        ++e->L->generation;
    }
}

void eng_ensure_verts(bcmc_engine* e, uint64_t need)
{
    if (need <= e->L->vert_cap) return;
    BCMC_CUDA(cudaStreamSynchronize(e->stream));
    uint64_t n = std::max<uint64_t>(need + need / 2, 1u << 20);
    if (e->opts.vertex_budget) n = std::max<uint64_t>(need, std::min<uint64_t>(n, e->opts.vertex_budget));
    // keep the vertices already written by earlier sequences of this run
    uint2* nv = (uint2*)dev_alloc(e->ctx, n * sizeof(uint2));
    if (e->L->vert_used)
        BCMC_CUDA(cudaMemcpyAsync(nv, e->L->verts, e->L->vert_used * sizeof(uint2), cudaMemcpyDeviceToDevice, e->stream));
    BCMC_CUDA(cudaStreamSynchronize(e->stream));
    dev_free(e->ctx, e->L->verts, e->L->vert_cap * sizeof(uint2));
    e->L->verts = nv;
    e->L->vert_cap = n;
    ++e->L->generation;
}

// Allocates lane k's buffers (lane 0 at creation; lane 1 on the first
// pipelined run) and makes k the current lane.
void eng_lane_init(bcmc_engine* e, int k)
{
    EngLane& l = e->lanes[k];
    e->L = &l;
    if (l.ready) return;
    bcmc_ctx* ctx = e->ctx;
    BCMC_CUDA(cudaEventCreate(&l.ev0));
    BCMC_CUDA(cudaEventCreate(&l.ev1));
    BCMC_CUDA(cudaEventCreateWithFlags(&l.ev_front, cudaEventDisableTiming));
    BCMC_CUDA(cudaEventCreateWithFlags(&l.ev_done, cudaEventDisableTiming));
    BCMC_CUDA(cudaMallocHost(&l.h_queries, e->max_batch * sizeof(EngQuery)));
    BCMC_CUDA(cudaMallocHost(&l.h_results, e->max_batch * sizeof(EngResult)));
    BCMC_CUDA(cudaMallocHost(&l.h_st, sizeof(EngState)));
    memset(l.h_st, 0, sizeof(EngState));
    l.d_queries = (EngQuery*)dev_alloc(ctx, e->max_batch * sizeof(EngQuery));
    l.d_results = (EngResult*)dev_alloc(ctx, e->max_batch * sizeof(EngResult));
    l.d_st = (EngState*)dev_alloc(ctx, sizeof(EngState));
    BCMC_CUDA(cudaMemsetAsync(l.d_st, 0, sizeof(EngState), e->stream));
    l.q_nactive = (uint32_t*)dev_alloc(ctx, e->max_batch * 4);
    l.q_nverts = (uint32_t*)dev_alloc(ctx, e->max_batch * 4);
    l.ready = true;
    // with a vertex budget the buffer is sized for it once, up front
    eng_ensure_verts(e, e->opts.vertex_budget ? e->opts.vertex_budget
                                              : (e->opts.vertex_capacity ? e->opts.vertex_capacity : (1ull << 24)));
    eng_ensure_status(e, 1024);
    eng_ensure_batch(e, 1u << 16, 1u << 16);
    BCMC_CUDA(cudaStreamSynchronize(e->stream));
}

void eng_lane_free(bcmc_engine* e, EngLane& l)
{
    bcmc_ctx* ctx = e->ctx;
    for (auto& kv : l.graphs) {
        if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
        if (kv.second.front) cudaGraphExecDestroy(kv.second.front);
        if (kv.second.back) cudaGraphExecDestroy(kv.second.back);
    }
    l.graphs.clear();
    dev_free(ctx, l.d_queries, e->max_batch * sizeof(EngQuery));
    dev_free(ctx, l.d_results, e->max_batch * sizeof(EngResult));
    dev_free(ctx, l.d_st, sizeof(EngState));
    dev_free(ctx, l.q_nactive, e->max_batch * 4);
    dev_free(ctx, l.q_nverts, e->max_batch * 4);
    dev_free(ctx, l.bitmap, 2 * l.bitmap_words * 4);
    dev_free(ctx, l.ent_id, (size_t)l.entry_cap * 4);
    dev_free(ctx, l.ent_q, (size_t)l.entry_cap * 4);
    dev_free(ctx, l.block_counts, (size_t)l.entry_cap * 4);
    dev_free(ctx, l.wv_list, (size_t)l.entry_cap * 4);
    dev_free(ctx, l.wv_off, (size_t)l.entry_cap * 4);
    dev_free(ctx, l.verts, l.vert_cap * sizeof(uint2));
    dev_free(ctx, l.status, l.status_words * 8);
    if (l.h_queries) cudaFreeHost(l.h_queries);
    if (l.h_results) cudaFreeHost(l.h_results);
    if (l.h_st) cudaFreeHost(l.h_st);
    if (l.ev0) cudaEventDestroy(l.ev0);
    if (l.ev1) cudaEventDestroy(l.ev1);
    if (l.ev_front) cudaEventDestroy(l.ev_front);
    if (l.ev_done) cudaEventDestroy(l.ev_done);
    l = EngLane{};
}

// The launch sequence of one batch (also what a graph captures).
// Phase 1 of a batch: inputs in, active test, claims, decode of the claimed
// blocks into their slots.  Returns the kernels it launches, as the others do.
uint32_t eng_enqueue_front(bcmc_engine* e, uint32_t bucket, bool one_group, cudaStream_t s)
{
    const BatchArgs a = eng_args(e);
    BCMC_CUDA(cudaMemcpyAsync(e->L->d_queries, e->L->h_queries, bucket * sizeof(EngQuery), cudaMemcpyHostToDevice, s));
    BCMC_CUDA(cudaMemcpyAsync(e->L->d_st, e->L->h_st, offsetof(EngState, epoch), cudaMemcpyHostToDevice, s));
    BCMC_CUDA(cudaEventRecordWithFlags(e->L->ev0, s, cudaEventRecordExternal));
    k_bbegin<<<1, 1024, 0, s>>>(e->L->d_st, e->L->q_nverts, e->L->q_nactive, bucket);
    // one group: one CTA's work, entries included
    k_bactive<<<one_group ? 1 : eng_grid_act(e), kEngThreads, 0, s>>>(a);
    if (!one_group) k_bentries<<<eng_grid_act(e), kEngThreads, 0, s>>>(a);
    const uint32_t r = e->max_rate;
    if (e->cfg.dec_threads == 64) {
        const size_t smem = zfp_stage_smem(64, r);
        allow_smem(k_bdecode<64>, smem);
        k_bdecode<64><<<eng_grid_dec(e), 64, smem, s>>>(a, r);
    } else if (e->cfg.dec_threads == 256) {
        const size_t smem = zfp_stage_smem(256, r);
        allow_smem(k_bdecode<256>, smem);
        k_bdecode<256><<<eng_grid_dec(e), 256, smem, s>>>(a, r);
    } else {
        const size_t smem = zfp_stage_smem(128, r);
        allow_smem(k_bdecode<128>, smem);
        k_bdecode<128><<<eng_grid_dec(e), 128, smem, s>>>(a, r);
    }
    BCMC_CUDA(cudaGetLastError());
    return one_group ? 3 : 4;
}

template <int kB>
void bmc_launch(cudaLaunchConfig_t cfg, const BatchArgs& a)
{
    cfg.dynamicSmemBytes = sizeof(McShared<16 * kB, false>);
    allow_smem(k_bmc<kB>, cfg.dynamicSmemBytes);
    BCMC_CUDA(cudaLaunchKernelEx(&cfg, k_bmc<kB>, a));
}

// Phase 2: marching cubes over the batch's entries, per-query results, state out.
uint32_t eng_enqueue_back(bcmc_engine* e, uint32_t bucket, cudaStream_t s)
{
    const BatchArgs a = eng_args(e);
    // cooperative: k_bmc's grid barrier needs every CTA resident
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(eng_grid_mc(e));
    cfg.blockDim = dim3(16 * e->cfg.mc_blocks);
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (e->cfg.mc_blocks == 8) bmc_launch<8>(cfg, a);
    else if (e->cfg.mc_blocks == 32) bmc_launch<32>(cfg, a);
    else bmc_launch<16>(cfg, a);
    k_bfinish<<<1, kFinThreads, 0, s>>>(a);
    BCMC_CUDA(cudaGetLastError());
    BCMC_CUDA(cudaEventRecordWithFlags(e->L->ev1, s, cudaEventRecordExternal));
    BCMC_CUDA(cudaMemcpyAsync(e->L->h_st, e->L->d_st, sizeof(EngState), cudaMemcpyDeviceToHost, s));
    BCMC_CUDA(cudaMemcpyAsync(e->L->h_results, e->L->d_results, bucket * sizeof(EngResult), cudaMemcpyDeviceToHost, s));
    return 2;
}

// The launch sequence of one batch on one stream (what a graph captures).
uint32_t eng_enqueue(bcmc_engine* e, uint32_t bucket, bool one_group)
{
    return eng_enqueue_front(e, bucket, one_group, e->stream) + eng_enqueue_back(e, bucket, e->stream);
}

int eng_cfg_key(const EngConfig& c)
{
    const int log_blocks = c.mc_blocks == 8 ? 3 : (c.mc_blocks == 32 ? 5 : 4);
    return c.act_per_sm | (c.dec_threads << 8) | (c.dec_per_sm << 18) | (c.mc_per_sm << 24) | (log_blocks << 27);
}

// Captures what `enqueue` issues on stream s into a graph; adds its kernels to *kernels.
template <typename F>
cudaGraphExec_t eng_capture(cudaStream_t s, uint32_t* kernels, F&& enqueue)
{
    cudaGraph_t graph = nullptr;
    BCMC_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    try {
        *kernels += enqueue();
    } catch (...) {
        cudaStreamEndCapture(s, &graph);
        if (graph) cudaGraphDestroy(graph);
        throw;
    }
    BCMC_CUDA(cudaStreamEndCapture(s, &graph));
    cudaGraphExec_t exec = nullptr;
    const cudaError_t err = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    BCMC_CUDA(err);
    return exec;
}

// A batch as it is launched: its batch-size bucket, tiles and bitmap words.
struct SeqShape {
    uint32_t bucket;
    uint64_t tiles, words;

    bool one_group() const { return tiles <= kGroup; }
    uint32_t graph_key() const { return 2u * bucket + (one_group() ? 1u : 0u); }
};

void eng_launch(bcmc_engine* e, const SeqShape& sh)
{
    auto it = e->tuned.find(sh.bucket);
    e->cfg = it != e->tuned.end() ? it->second : EngConfig{};
    auto& g = e->L->graphs[sh.graph_key()];
    const int key = eng_cfg_key(e->cfg);
    if (!g.exec || g.generation != e->L->generation || g.cfg_key != key) {
        if (g.exec) cudaGraphExecDestroy(g.exec);
        g.exec = nullptr;
        g.kernels = 0;
        g.exec = eng_capture(e->stream, &g.kernels, [&] { return eng_enqueue(e, sh.bucket, sh.one_group()); });
        g.generation = e->L->generation;
        g.cfg_key = key;
    }
    BCMC_CUDA(cudaGraphLaunch(g.exec, e->stream));
    count_launches(g.kernels);
}

// Pipelined launch: phase 1 on the front stream, phase 2 on the back stream
// after it.  The next batch's phase 1 (front stream) can then run while this
// batch's phase 2 does.
void eng_launch_split(bcmc_engine* e, const SeqShape& sh)
{
    auto it = e->tuned.find(sh.bucket);
    e->cfg = it != e->tuned.end() ? it->second : EngConfig{};
    auto& g = e->L->graphs[sh.graph_key()];
    const int key = eng_cfg_key(e->cfg);
    if (!g.front || g.split_generation != e->L->generation || g.split_cfg_key != key) {
        if (g.front) cudaGraphExecDestroy(g.front);
        if (g.back) cudaGraphExecDestroy(g.back);
        g.front = g.back = nullptr;
        g.split_kernels = 0;
        g.front = eng_capture(e->stream, &g.split_kernels, [&] { return eng_enqueue_front(e, sh.bucket, sh.one_group(), e->stream); });
        g.back = eng_capture(e->stream_back, &g.split_kernels, [&] { return eng_enqueue_back(e, sh.bucket, e->stream_back); });
        g.split_generation = e->L->generation;
        g.split_cfg_key = key;
    }
    BCMC_CUDA(cudaGraphLaunch(g.front, e->stream));
    BCMC_CUDA(cudaEventRecord(e->L->ev_front, e->stream));
    BCMC_CUDA(cudaStreamWaitEvent(e->stream_back, e->L->ev_front, 0));
    BCMC_CUDA(cudaGraphLaunch(g.back, e->stream_back));
    count_launches(g.split_kernels);
}

uint32_t bucket_of(uint32_t n)
{
    uint32_t b = 1;
    while (b < n) b <<= 1;
    return b;
}

// Refusal of a launch sequence by the vertex budget: only its first `fit`
// queries fit (their counts are known from the count pass).
struct AdmitPrefix : std::length_error {
    uint32_t fit;
    explicit AdmitPrefix(uint32_t f) : std::length_error("batch above the vertex budget"), fit(f) {}
};

// The current lane's query table for queries[0..n), padded to the batch-size
// bucket, and its buffers sized for it.
SeqShape eng_prepare(bcmc_engine* e, const bcmc_query* queries, uint32_t n)
{
    SeqShape sh{std::min(bucket_of(n), e->max_batch), 0, 0};
    for (uint32_t i = 0; i < sh.bucket; ++i) {
        EngQuery q{};
        if (i < n) {
            if (queries[i].volume >= e->vols.size()) throw std::invalid_argument("unknown volume id");
            const EngVolume& v = e->vols[queries[i].volume];
            q.vol = queries[i].volume;
            q.iso = queries[i].isovalue;
            q.tile0 = (uint32_t)sh.tiles;
            q.bit0 = (uint32_t)sh.words;
            sh.tiles += v.tiles;
            sh.words += (uint64_t)v.tiles * (kEngTile / 32);
        } else {  // padding queries of the bucket: no tiles
            q.vol = 0;
            q.iso = 0.0f;
            q.tile0 = (uint32_t)sh.tiles;
            q.bit0 = (uint32_t)sh.words;
        }
        e->L->h_queries[i] = q;
    }
    if (sh.tiles >= 0xffffffffull || sh.words >= 0xffffffffull) throw std::invalid_argument("batch too large");
    eng_ensure_status(e, sh.tiles);
    eng_ensure_batch(e, sh.words, std::max<uint32_t>(e->L->entry_cap, 1u << 16));
    return sh;
}

// The current lane's batch inputs for one launch of the sequence.
void eng_set_inputs(bcmc_engine* e, const SeqShape& sh)
{
    EngState& st = *e->L->h_st;
    st.nq = sh.bucket;
    st.ntiles = (uint32_t)sh.tiles;
    st.entry_capacity = e->L->entry_cap;
    st.use_epoch = e->use_epoch;
    st.vert_capacity = e->L->vert_cap;
    st.vert_base = e->L->vert_used;
}

void eng_take_results(bcmc_engine* e, uint32_t n, bcmc_query_result* out)
{
    for (uint32_t i = 0; i < n; ++i) {
        out[i].vertex_offset = e->L->h_results[i].vstart;
        out[i].num_vertices = e->L->h_results[i].nverts;
        out[i].num_active_blocks = e->L->h_results[i].nactive;
    }
    e->L->vert_used += e->L->h_st->num_verts;
    float ms = 0.0f;
    if (cudaEventElapsedTime(&ms, e->L->ev0, e->L->ev1) == cudaSuccess) e->stats.last_batch_ms = ms;
    e->stats.queries += n;
}

// Runs queries[0..n) (n <= max_batch) as one launch sequence; results go to out.
// Throws std::length_error when the pool cannot hold the sequence's active blocks.
void eng_run_sequence(bcmc_engine* e, const bcmc_query* queries, uint32_t n, bcmc_query_result* out)
{
    const SeqShape sh = eng_prepare(e, queries, n);
    const uint32_t bucket = sh.bucket;
    const uint64_t words = sh.words;
    ++e->use_epoch;
    for (int attempt = 0;; ++attempt) {
        if (attempt > 8) throw std::runtime_error("batch did not converge");
        eng_ensure_verts(e, e->L->vert_used + 1);
        EngState& st = *e->L->h_st;
        eng_set_inputs(e, sh);
        eng_epoch_tick(e);
        eng_launch(e, sh);
        BCMC_CUDA(cudaStreamSynchronize(e->stream));
        ++e->stats.launch_sequences;
        if (st.error) throw std::runtime_error("device wait timed out in the batched engine");
        e->stats.decoded_blocks += st.num_decode;
        if (st.entry_overflow) {
            eng_ensure_batch(e, words, st.num_entries);
            continue;
        }
        if (st.pool_exhausted) {
            // the pool's head overshot its tail: clamp, then free what this batch does not use
            BCMC_CUDA(cudaMemcpyAsync(e->h_pool, e->d_pool, sizeof(EngPool), cudaMemcpyDeviceToHost, e->stream));
            BCMC_CUDA(cudaStreamSynchronize(e->stream));
            e->h_pool->head = e->h_pool->tail;
            BCMC_CUDA(cudaMemcpyAsync(e->d_pool, e->h_pool, sizeof(EngPool), cudaMemcpyHostToDevice, e->stream));
            BCMC_CUDA(cudaMemsetAsync(e->d_evicted, 0, 8, e->stream));
            k_bevict<<<e->ctx->num_sms * 8, 256, 0, e->stream>>>(eng_args(e), e->use_epoch, (uint32_t)e->pool_slots,
                                                                 e->d_evicted);
            count_launches(1);
            unsigned long long ev = 0;
            BCMC_CUDA(cudaMemcpyAsync(&ev, e->d_evicted, 8, cudaMemcpyDeviceToHost, e->stream));
            BCMC_CUDA(cudaStreamSynchronize(e->stream));
            e->stats.evicted_blocks += ev;
            if (ev == 0) throw std::length_error("the slot pool cannot hold one batch's active blocks");
            continue;
        }
        // vertex admission from the count pass: per-query totals are complete
        // even when the emit pass was refused for lack of room
        const uint64_t limit_seq = std::min<uint64_t>(
            (1ull << 32) - 1, e->opts.vertex_budget ? e->opts.vertex_budget - std::min(e->opts.vertex_budget, e->L->vert_used)
                                                    : ~0ull);
        if (st.vert_overflow || st.num_verts > limit_seq) {
            uint64_t cum = 0;
            uint32_t fit = 0;
            for (; fit < n; ++fit) {
                const uint64_t v = e->L->h_results[fit].nverts;
                if (cum + v > limit_seq) break;
                cum += v;
            }
            if (fit < n) throw AdmitPrefix(fit);
            eng_ensure_verts(e, e->L->vert_used + cum);
            continue;  // the re-run finds every block cached: no decode work repeats
        }
        break;
    }
    eng_take_results(e, n, out);
}

// Admission by slot memory: a batch whose active blocks do not fit the pool
// (even after evicting every slot it does not use) runs as two halves.
void eng_run_chunk(bcmc_engine* e, const bcmc_query* queries, uint32_t n, bcmc_query_result* out)
{
    try {
        eng_run_sequence(e, queries, n, out);
    } catch (const std::length_error&) {
        if (n < 2) throw;
        const uint32_t h = n / 2;
        eng_run_chunk(e, queries, h, out);
        eng_run_chunk(e, queries + h, n - h, out + h);
    }
}

void eng_free(bcmc_engine* e)
{
    bcmc_ctx* ctx = e->ctx;
    if (e->stream) cudaStreamSynchronize(e->stream);
    if (e->stream_back) cudaStreamSynchronize(e->stream_back);
    if (e->stream_copy) cudaStreamSynchronize(e->stream_copy);
    for (EngLane& l : e->lanes) eng_lane_free(e, l);
    for (auto& v : e->vols) {
        dev_free(ctx, v.words, v.words_bytes);
        dev_free(ctx, v.ranges, (size_t)v.total * 8);
        dev_free(ctx, v.tile_ext, (size_t)v.tiles * 8);
        dev_free(ctx, v.item_slots, (size_t)v.total * 4);
    }
    dev_free(ctx, e->d_vols, e->d_vols_cap * sizeof(EngVolDev));
    dev_free(ctx, e->cache, e->pool_slots * 256);
    dev_free(ctx, e->free_list, e->pool_slots * 4);
    dev_free(ctx, e->last_use, e->pool_slots * 4);
    dev_free(ctx, e->owner_vol, e->pool_slots * 4);
    dev_free(ctx, e->owner_block, e->pool_slots * 4);
    dev_free(ctx, e->d_pool, sizeof(EngPool));
    dev_free(ctx, e->d_evicted, 8);
    dev_free(ctx, e->dec_vol, (size_t)e->dec_cap * 4);
    dev_free(ctx, e->dec_block, (size_t)e->dec_cap * 4);
    dev_free(ctx, e->dec_slot, (size_t)e->dec_cap * 4);
    if (e->h_pool) cudaFreeHost(e->h_pool);
    if (e->stream) cudaStreamDestroy(e->stream);
    if (e->stream_back) cudaStreamDestroy(e->stream_back);
    if (e->stream_copy) cudaStreamDestroy(e->stream_copy);
    delete e;
    ctx_child_removed(ctx);
}

template <typename F>
bcmc_status eng_guarded(bcmc_engine* e, F&& f)
{
    try {
        return f();
    } catch (const CudaError& x) {
        e->ctx->last_error = std::string(x.what) + ": " + cudaGetErrorString(x.err);
        return x.err == cudaErrorMemoryAllocation ? BCMC_E_OOM : BCMC_E_CUDA;
    } catch (const std::invalid_argument& x) {
        e->ctx->last_error = x.what();
        return BCMC_E_ARG;
    } catch (const std::length_error& x) {
        e->ctx->last_error = x.what();
        return BCMC_E_ADMISSION;
    } catch (const std::bad_alloc&) {
        e->ctx->last_error = "host allocation failed";
        return BCMC_E_OOM;
    } catch (const std::exception& x) {
        e->ctx->last_error = x.what();
        return BCMC_E_CUDA;
    }
}

}  // namespace

extern "C" bcmc_status bcmc_engine_create(bcmc_ctx* ctx, const bcmc_engine_opts* opts, bcmc_engine** out)
{
    if (!ctx || !out) return BCMC_E_ARG;
    *out = nullptr;
    bcmc_engine* e = new (std::nothrow) bcmc_engine();
    if (!e) return BCMC_E_OOM;
    e->ctx = ctx;
    if (opts) e->opts = *opts;
    if (e->opts.flags != 0) {
        delete e;
        return BCMC_E_ARG;
    }
    ctx_child_added(ctx);  // eng_free removes it, also on the error path below
    const bcmc_status st = eng_guarded(e, [&]() -> bcmc_status {
        BCMC_CUDA(cudaSetDevice(ctx->device));
        BCMC_CUDA(cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking));
        BCMC_CUDA(cudaStreamCreateWithFlags(&e->stream_back, cudaStreamNonBlocking));
        BCMC_CUDA(cudaStreamCreateWithFlags(&e->stream_copy, cudaStreamNonBlocking));
        e->max_batch = bucket_of(e->opts.max_batch ? std::min<uint32_t>(e->opts.max_batch, 1u << 16) : 1024u);
        BCMC_CUDA(cudaMallocHost(&e->h_pool, sizeof(EngPool)));
        e->d_pool = (EngPool*)dev_alloc(ctx, sizeof(EngPool));
        e->d_evicted = (unsigned long long*)dev_alloc(ctx, 8);
        eng_lane_init(e, 0);
        BCMC_CUDA(cudaStreamSynchronize(e->stream));
        return BCMC_OK;
    });
    if (st != BCMC_OK) {
        eng_free(e);
        return st;
    }
    *out = e;
    return BCMC_OK;
}

extern "C" void bcmc_engine_destroy(bcmc_engine* e)
{
    if (e) eng_free(e);
}

extern "C" bcmc_status bcmc_engine_add_volume(bcmc_engine* e, const uint8_t* zfp, size_t len, uint32_t rate,
                                              const uint32_t dims[3], uint32_t* volume)
{
    if (!e || !zfp || !dims || !volume || rate == 0 || rate > 32 || !dims[0] || !dims[1] || !dims[2])
        return BCMC_E_ARG;
    if (e->vols.size() >= kMaxVolumes) return BCMC_E_ARG;
    if (e->pool_slots) return BCMC_E_STATE;  // volumes are added before the first run sizes the pool
    return eng_guarded(e, [&]() -> bcmc_status {
        EngVolume v;
        for (int i = 0; i < 3; ++i) v.dims[i] = dims[i];
        v.rate = rate;
        const uint3 nb = make_uint3(div_up(dims[0], 4u), div_up(dims[1], 4u), div_up(dims[2], 4u));
        const uint64_t total = (uint64_t)nb.x * nb.y * nb.z;
        if (total >= (1ull << 31)) throw std::invalid_argument("volume too large");
        const uint64_t need = (total * 64u * rate + 7) / 8;
        if (len < need) throw std::invalid_argument("compressed stream shorter than the volume needs");
        v.total = (uint32_t)total;
        v.tiles = div_up(v.total, kEngTile);
        v.grid = make_block_grid(nb);
        const uint64_t words = (need + 7) / 8 + 2;
        v.words_bytes = words * 8;
        v.words = (uint64_t*)dev_alloc(e->ctx, v.words_bytes);
        BCMC_CUDA(cudaMemsetAsync(v.words, 0, v.words_bytes, e->stream));
        BCMC_CUDA(cudaMemcpyAsync(v.words, zfp, need, cudaMemcpyHostToDevice, e->stream));
        v.ranges = (float2*)dev_alloc(e->ctx, (size_t)v.total * 8);
        v.tile_ext = (float2*)dev_alloc(e->ctx, (size_t)v.tiles * 8);
        v.item_slots = (int32_t*)dev_alloc(e->ctx, (size_t)v.total * 4);
        BCMC_CUDA(cudaMemsetAsync(v.item_slots, 0xff, (size_t)v.total * 4, e->stream));  // -1
        zfp_ranges_launch(e->ctx, v.words, dims, 64u * rate, reinterpret_cast<float*>(v.ranges), e->stream);
        k_tile_ext<<<v.tiles, kEngThreads, 0, e->stream>>>(v.ranges, v.grid, v.total, v.tile_ext);
        count_launches(1);
        BCMC_CUDA(cudaGetLastError());
        BCMC_CUDA(cudaStreamSynchronize(e->stream));
        *volume = (uint32_t)e->vols.size();
        e->vols.push_back(v);
        if (rate > e->max_rate) {
            e->max_rate = rate;
            for (EngLane& l : e->lanes) ++l.generation;  // graphs captured k_bdecode's staging size
        }
        eng_upload_vols(e);
        return BCMC_OK;
    });
}

extern "C" bcmc_status bcmc_engine_run(bcmc_engine* e, const bcmc_query* queries, uint32_t n,
                                       bcmc_query_result* results)
{
    if (!e || (n && (!queries || !results))) return BCMC_E_ARG;
    if (e->vols.empty()) return BCMC_E_STATE;
    return eng_guarded(e, [&]() -> bcmc_status {
        if (!e->pool_slots) {
            uint64_t all = 0;
            for (auto& v : e->vols) all += v.total;
            eng_alloc_pool(e, e->opts.pool_slots ? e->opts.pool_slots : all);
        }
        e->L->vert_used = 0;
        for (uint32_t i = 0; i < n; i += e->max_batch) {
            const uint32_t m = std::min(e->max_batch, n - i);
            eng_run_chunk(e, queries + i, m, results + i);
        }
        ++e->stats.batches;
        return BCMC_OK;
    });
}

namespace {
// Runs the longest prefix of queries[0..n) that the slot pool and the vertex
// budget admit (halving on refusal); returns its length.  Throws
// std::length_error when not even queries[0] alone fits.
uint32_t eng_run_prefix(bcmc_engine* e, const bcmc_query* queries, uint32_t n, bcmc_query_result* out)
{
    try {
        eng_run_sequence(e, queries, n, out);
        return n;
    } catch (const AdmitPrefix& x) {  // the count pass says how many fit
        if (x.fit == 0) throw;
        return eng_run_prefix(e, queries, x.fit, out);
    } catch (const std::length_error&) {  // the slot pool: halve
        if (n < 2) throw;
        return eng_run_prefix(e, queries, n / 2, out);
    }
}
}  // namespace

namespace {
// device time of one launch sequence under the current tuned config: best of 3
double eng_time_sequence(bcmc_engine* e, const bcmc_query* qs, uint32_t n, bcmc_query_result* out)
{
    double best = 1e30;
    for (int r = 0; r < 3; ++r) {
        e->L->vert_used = 0;
        eng_run_sequence(e, qs, n, out);
        best = std::min(best, e->stats.last_batch_ms);
    }
    return best;
}

double eng_time_decode(bcmc_engine* e, const EngVolume& v, uint32_t nblk, float* scratch, int threads, int per_sm)
{
    float best = 1e30f;
    for (int r = 0; r < 3; ++r) {
        BCMC_CUDA(cudaEventRecord(e->L->ev0, e->stream));
        const int grid = e->ctx->num_sms * per_sm;
        const size_t smem = zfp_stage_smem((uint32_t)threads, v.rate);
        if (threads == 64) {
            allow_smem(k_decode_probe<64>, smem);
            k_decode_probe<64><<<grid, 64, smem, e->stream>>>(v.words, v.rate, nblk, scratch);
        } else if (threads == 256) {
            allow_smem(k_decode_probe<256>, smem);
            k_decode_probe<256><<<grid, 256, smem, e->stream>>>(v.words, v.rate, nblk, scratch);
        } else {
            allow_smem(k_decode_probe<128>, smem);
            k_decode_probe<128><<<grid, 128, smem, e->stream>>>(v.words, v.rate, nblk, scratch);
        }
        count_launches(1);
        BCMC_CUDA(cudaGetLastError());
        BCMC_CUDA(cudaEventRecord(e->L->ev1, e->stream));
        BCMC_CUDA(cudaEventSynchronize(e->L->ev1));
        float ms = 0.0f;
        BCMC_CUDA(cudaEventElapsedTime(&ms, e->L->ev0, e->L->ev1));
        best = std::min(best, ms);
    }
    return best;
}
}  // namespace

extern "C" bcmc_status bcmc_engine_autotune(bcmc_engine* e, const bcmc_query* queries, uint32_t n,
                                            bcmc_tune_report* out)
{
    if (!e || !queries || !n || !out) return BCMC_E_ARG;
    if (e->vols.empty()) return BCMC_E_STATE;
    return eng_guarded(e, [&]() -> bcmc_status {
        if (!e->pool_slots) {
            uint64_t all = 0;
            for (auto& v : e->vols) all += v.total;
            eng_alloc_pool(e, e->opts.pool_slots ? e->opts.pool_slots : all);
        }
        const uint32_t m = std::min(n, e->max_batch);
        const uint32_t bucket = std::min(bucket_of(m), e->max_batch);
        std::vector<bcmc_query_result> res(m);
        e->tuned.erase(bucket);
        e->L->vert_used = 0;
        eng_run_sequence(e, queries, m, res.data());  // warm-up: decodes, buffer growth, graph
        EngConfig best{};
        e->tuned[bucket] = best;
        double t_best = eng_time_sequence(e, queries, m, res.data());
        out->batch_ms_default = t_best;
        // coordinate descent over the sequence's launch parameters
        const auto take_faster = [&](const std::vector<EngConfig>& others) {
            for (const EngConfig& c : others) {
                e->tuned[bucket] = c;
                const double t = eng_time_sequence(e, queries, m, res.data());
                if (t < t_best) best = c, t_best = t;
            }
        };
        take_faster(other_mc_sizes(best));
        take_faster(other_mc_ctas(best, bmc_resident(best.mc_blocks)));
        std::vector<EngConfig> acts;
        for (int act : {4, 16}) {
            acts.push_back(best);
            acts.back().act_per_sm = act;
        }
        take_faster(acts);
        out->batch_ms_tuned = t_best;
        // decode: a probe over (up to 2^18) blocks of the largest volume
        const EngVolume* big = &e->vols[0];
        for (auto& v : e->vols)
            if (v.total > big->total) big = &v;
        const uint32_t nblk = std::min<uint32_t>(big->total, 1u << 18);
        float* scratch = (float*)dev_alloc(e->ctx, (size_t)nblk * 256);
        double d_best = 1e30, d_default = 0.0;
        try {
            for (int thr : {64, 128, 256})
                for (int per_sm : {8, 16, 32}) {
                    const double t = eng_time_decode(e, *big, nblk, scratch, thr, per_sm);
                    if (thr == 128 && per_sm == 16) d_default = t;
                    if (t < d_best) {
                        d_best = t;
                        best.dec_threads = thr;
                        best.dec_per_sm = per_sm;
                    }
                }
        } catch (...) {
            dev_free(e->ctx, scratch, (size_t)nblk * 256);
            throw;
        }
        dev_free(e->ctx, scratch, (size_t)nblk * 256);
        e->tuned[bucket] = best;
        out->decode_ms_default = d_default;
        out->decode_ms_tuned = d_best;
        out->act_ctas_per_sm = best.act_per_sm;
        out->decode_threads = best.dec_threads;
        out->decode_ctas_per_sm = best.dec_per_sm;
        out->mc_ctas_per_sm = best.mc_per_sm;
        out->mc_blocks_per_tile = best.mc_blocks;
        out->bucket = bucket;
        return BCMC_OK;
    });
}

extern "C" bcmc_status bcmc_engine_set_tuning(bcmc_engine* e, const bcmc_tune_report* c)
{
    if (!e || !c) return BCMC_E_ARG;
    const uint32_t b = c->bucket;
    const auto in = [](int v, std::initializer_list<int> ok) { return std::find(ok.begin(), ok.end(), v) != ok.end(); };
    if (b == 0 || (b & (b - 1)) != 0 || b > e->max_batch || !in(c->act_ctas_per_sm, {4, 8, 16}) ||
        !in(c->decode_threads, {64, 128, 256}) || !in(c->decode_ctas_per_sm, {8, 16, 32}) ||
        !in(c->mc_ctas_per_sm, {4, 5, 6}) || !in(c->mc_blocks_per_tile, {8, 16, 32}))
        return BCMC_E_ARG;
    EngConfig cfg;
    cfg.act_per_sm = c->act_ctas_per_sm;
    cfg.dec_threads = c->decode_threads;
    cfg.dec_per_sm = c->decode_ctas_per_sm;
    cfg.mc_per_sm = c->mc_ctas_per_sm;
    cfg.mc_blocks = c->mc_blocks_per_tile;
    e->tuned[b] = cfg;
    return BCMC_OK;
}

extern "C" bcmc_status bcmc_engine_run_admit(bcmc_engine* e, const bcmc_query* queries, uint32_t n,
                                             bcmc_query_result* results, uint32_t* admitted)
{
    if (!e || !admitted || (n && (!queries || !results))) return BCMC_E_ARG;
    if (e->vols.empty()) return BCMC_E_STATE;
    *admitted = 0;
    return eng_guarded(e, [&]() -> bcmc_status {
        if (!e->pool_slots) {
            uint64_t all = 0;
            for (auto& v : e->vols) all += v.total;
            eng_alloc_pool(e, e->opts.pool_slots ? e->opts.pool_slots : all);
        }
        e->L->vert_used = 0;
        uint32_t done = 0;
        while (done < n) {
            const uint32_t m = std::min(e->max_batch, n - done);
            uint32_t got;
            try {
                got = eng_run_prefix(e, queries + done, m, results + done);
            } catch (const std::length_error&) {
                if (done) break;  // the rest waits for the next run
                throw;
            }
            done += got;
            if (got < m) break;
        }
        *admitted = done;
        ++e->stats.batches;
        return BCMC_OK;
    });
}

extern "C" bcmc_status bcmc_engine_vertices(bcmc_engine* e, const void** d_vertices, uint64_t* count)
{
    if (!e || !d_vertices || !count) return BCMC_E_ARG;
    *d_vertices = e->L->verts;
    *count = e->L->vert_used;
    return BCMC_OK;
}

extern "C" bcmc_status bcmc_engine_copy_vertices(bcmc_engine* e, uint64_t first, uint64_t count, void* host)
{
    if (!e || (count && !host) || first > e->L->vert_used || count > e->L->vert_used - first) return BCMC_E_ARG;
    return eng_guarded(e, [&]() -> bcmc_status {
        if (count)
            BCMC_CUDA(cudaMemcpyAsync(host, e->L->verts + first, count * sizeof(uint2), cudaMemcpyDeviceToHost, e->stream));
        BCMC_CUDA(cudaStreamSynchronize(e->stream));
        return BCMC_OK;
    });
}

extern "C" bcmc_status bcmc_engine_stats_get(bcmc_engine* e, bcmc_engine_stats* out)
{
    if (!e || !out) return BCMC_E_ARG;
    return eng_guarded(e, [&]() -> bcmc_status {
        bcmc_engine_stats s = e->stats;
        s.pool_slots = e->pool_slots;
        if (e->pool_slots) {
            BCMC_CUDA(cudaMemcpyAsync(e->h_pool, e->d_pool, sizeof(EngPool), cudaMemcpyDeviceToHost, e->stream));
            BCMC_CUDA(cudaStreamSynchronize(e->stream));
            const uint32_t head = std::min(e->h_pool->head, e->h_pool->tail);
            s.pool_used = e->pool_slots - (e->h_pool->tail - head);
        }
        s.vertex_capacity = e->L->vert_cap;
        s.overlapped_batches = e->overlapped;
        s.device_bytes = e->ctx->device_bytes;
        *out = s;
        return BCMC_OK;
    });
}

namespace bcmc {
namespace {
void eng_ensure_pool(bcmc_engine* e)
{
    if (e->pool_slots) return;
    uint64_t all = 0;
    for (auto& v : e->vols) all += v.total;
    eng_alloc_pool(e, e->opts.pool_slots ? e->opts.pool_slots : all);
}
}  // namespace

bcmc_status engine_submit(bcmc_engine* e, int k, const bcmc_query* queries, uint32_t n, void (*on_done)(void*),
                          void* arg)
{
    if (!e || k < 0 || k > 1 || !n || !queries || n > e->max_batch) return BCMC_E_ARG;
    if (e->vols.empty() || e->lanes[k].in_flight) return BCMC_E_STATE;
    return eng_guarded(e, [&]() -> bcmc_status {
        eng_ensure_pool(e);
        eng_lane_init(e, k);
        EngLane& me = *e->L;
        me.vert_used = 0;
        const SeqShape sh = eng_prepare(e, queries, n);
        ++e->use_epoch;
        eng_ensure_verts(e, 1);
        eng_set_inputs(e, sh);
        eng_epoch_tick(e);
        eng_launch_split(e, sh);
        BCMC_CUDA(cudaEventRecord(me.ev_done, e->stream_back));
        if (on_done) BCMC_CUDA(cudaLaunchHostFunc(e->stream_back, on_done, arg));
        me.in_flight = true;
        me.n = n;
        me.bucket = sh.bucket;
        me.batch_epoch = e->use_epoch;
        me.queries.assign(queries, queries + n);
        if (e->lanes[1 - k].in_flight) ++e->overlapped;
        ++e->stats.launch_sequences;
        ++e->stats.batches;
        return BCMC_OK;
    });
}

bcmc_status engine_complete(bcmc_engine* e, int k, bcmc_query_result* out, uint32_t* admitted)
{
    if (!e || k < 0 || k > 1 || !out || !admitted) return BCMC_E_ARG;
    EngLane& me = e->lanes[k];
    if (!me.in_flight) return BCMC_E_STATE;
    *admitted = 0;
    me.in_flight = false;
    return eng_guarded(e, [&]() -> bcmc_status {
        e->L = &me;
        BCMC_CUDA(cudaEventSynchronize(me.ev_done));
        const EngState& st = *me.h_st;
        e->stats.decoded_blocks += st.num_decode;
        if (st.error) throw std::runtime_error("device wait timed out in the batched engine");
        const uint64_t limit = std::min<uint64_t>((1ull << 32) - 1, e->opts.vertex_budget ? e->opts.vertex_budget : ~0ull);
        if (st.entry_overflow || st.pool_exhausted || st.vert_overflow || st.num_verts > limit) {
            // buffer growth, eviction or admission: run this batch again on its
            // own, after both streams have drained (an eviction must not free a
            // slot the other lane's batch still reads)
            BCMC_CUDA(cudaStreamSynchronize(e->stream));
            BCMC_CUDA(cudaStreamSynchronize(e->stream_back));
            me.vert_used = 0;
            *admitted = eng_run_prefix(e, me.queries.data(), me.n, out);
            return BCMC_OK;
        }
        eng_take_results(e, me.n, out);
        *admitted = me.n;
        return BCMC_OK;
    });
}

bcmc_status engine_copy_lane_vertices(bcmc_engine* e, int k, uint64_t first, uint64_t count, void* host)
{
    if (!e || k < 0 || k > 1 || (count && !host)) return BCMC_E_ARG;
    EngLane& l = e->lanes[k];
    if (first > l.vert_used || count > l.vert_used - first) return BCMC_E_ARG;
    return eng_guarded(e, [&]() -> bcmc_status {
        if (count) {
            BCMC_CUDA(cudaMemcpyAsync(host, l.verts + first, count * sizeof(uint2), cudaMemcpyDeviceToHost,
                                      e->stream_copy));
            BCMC_CUDA(cudaStreamSynchronize(e->stream_copy));
        }
        return BCMC_OK;
    });
}

void engine_drain(bcmc_engine* e)
{
    cudaStreamSynchronize(e->stream);
    cudaStreamSynchronize(e->stream_back);  // also waits for its host callbacks
    cudaStreamSynchronize(e->stream_copy);
}

uint32_t engine_max_batch(bcmc_engine* e) { return e->max_batch; }
uint32_t engine_num_volumes(bcmc_engine* e) { return (uint32_t)e->vols.size(); }

int engine_device(bcmc_engine* e) { return e->ctx->device; }
uint64_t engine_vertex_budget(bcmc_engine* e) { return e->opts.vertex_budget; }
bcmc_ctx* engine_ctx(bcmc_engine* e) { return e->ctx; }
}  // namespace bcmc
