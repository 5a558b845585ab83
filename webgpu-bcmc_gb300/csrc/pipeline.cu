// pipeline.cu -- device side of one isosurface query (computeSurface,
// js/compressed_marching_cubes.js:580-809) and of LRUCache.update
// (js/lru_cache.js:312-843).
//
// The reference runs ~20 dispatches with six host readbacks per query.  Here a
// query is a fixed sequence of launches that read every count from the
// QueryState on the device:
//   k_query_flags  new epoch of the status words, counters cleared; every block's
//                  range against the isovalue, in words of 32 blocks
//   k_active_words active test (compute_block_active.comp) on those words,
//                  fused with the compaction of active ids, the cache lookup
//                  (lru_cache_mark_new_items.comp's "needs caching"), the
//                  compaction of new item ids and that of the blocks that can
//                  have vertices; its last CTA decides the cache growth
//                  (js/lru_cache.js:510-522).  The standalone LRU update has
//                  k_query_begin and k_active in their place
//   (k_query_front those two and the next in one launch, for a small volume)
//   k_slots        age/mark/grow of every slot (lru_cache_age_slots.comp,
//                  lru_cache_mark_new_items.comp, lru_cache_init.comp) fused
//                  with the compaction of available slots and their ages, the
//                  sort keys' digit histograms and (last CTA) the sort's plan
//   sort           available slots by age, oldest first (sort.cu)
//   k_decode_new   beside k_slots and the sort (a branch of the query graph):
//                  the ZFP decode of the new blocks (zfp_decompress_block.comp)
//                  into a staging buffer
//   k_assign       lru_cache_update.comp, and the staged blocks copied into
//                  their slots
//   k_mc           marching cubes count + scan + emit in one cooperative launch
//                  (compute_block_has_vertices.comp,
//                  compute_block_voxel_num_verts.comp,
//                  compute_block_vertices.comp)
//   k_query_end    the query state the host reads, into its pinned copy
#include <algorithm>

#include "active_test.cuh"
#include "bcmc_pipeline.h"
#include "mc_common.cuh"
#include "slot_ranges.cuh"
#include "zfp_device.cuh"

namespace bcmc {

// Starts a query's state: counters cleared, a new epoch.  All threads
// of one CTA call it.
__device__ __forceinline__ void query_begin(QueryState* q, float iso, bool mc_only, uint32_t capacity,
                                            uint32_t vert_capacity, uint32_t drop_tile)
{
    const int t = threadIdx.x;
    if (t == 0) {
        q->epoch += 1;
        q->capacity = capacity;
        q->vert_capacity = vert_capacity;
        q->mc_arrived = 0;
        q->error = 0;
        q->vert_overflow = 0;
        q->num_with_verts = 0;
        q->num_verts = 0;
        if (!mc_only) {
            q->debug_drop_tile = drop_tile;
            q->isovalue = iso;
            q->tiles_active = q->tiles_slots = q->tiles_sort_hist = 0;
            for (int i = 0; i < 4; ++i) q->tiles_sort[i] = 0;
            q->sort_arrived = 0;
            q->num_active = q->num_live = q->num_new = q->num_avail = 0;
            q->grow_needed = 0;
            // the sort plan of zero keys (k_slots replaces it when it sorts)
            for (int i = 0; i < 4; ++i) q->sort_run[i] = q->sort_src[i] = 0;
            q->sort_first = 4;
            q->sort_final = 1;
            q->sort_key16 = q->sort_wide = 0;
        }
    }
    if (!mc_only)
        for (int i = t; i < 1536; i += blockDim.x) (&q->sort_hist[0][0])[i] = 0;  // and sort_hist16
}

__global__ void k_query_begin(QueryState* q, float iso, int mc_only, uint32_t capacity, uint32_t vert_capacity)
{
    query_begin(q, iso, mc_only != 0, capacity, vert_capacity, 0u);
}

// ---------------------------------------------------------------------------
// k_query_flags: starts a query, and tests every block's range against the
// isovalue: bit A of a block is iso >= lo, bit B iso <= hi.  The bits go out in
// words of 32 consecutive blocks, together with A, B and A & B ORed with those
// of the x neighbours (first step of the active test's 3x3x3 neighbourhood).
//
// Every range is read once, 8 bytes to a lane, and a ballot makes the words; a
// warp takes `wpw` of them, and its lanes then do the x neighbours of a word
// each.  k_active_words, which follows, works on these words: a byte a block
// where the ranges are 8.  Before, its tiles read the ranges of all three
// z-layers around them and tested 27 flag bytes a block, a tile at a time per
// CTA with a look-back between tiles: 565 us of the 1024 x 1024 x 1080 volume's
// query, for ranges that take 21 us to read.
// The inputs come from the arguments, or, when `in` is set, from the host's
// pinned copy, read directly (a query graph needs no copy node for them).
// ---------------------------------------------------------------------------
constexpr int kFlagThreads = 256;
constexpr uint32_t kFlagBatch = 8;  // ranges in flight per lane

__device__ __forceinline__ void query_flags(QueryState* q, float iso, uint32_t capacity, uint32_t vert_capacity,
                                            const QueryInputs* in, const FlagArgs& a)
{
    const uint32_t lane = threadIdx.x & 31u, total = a.total, wpw = a.wpw;
    const uint32_t nwords = div_up(total, 32u);
    const uint32_t step = gridDim.x * (kFlagThreads / 32) * wpw;
    uint32_t w0 = (blockIdx.x * (kFlagThreads / 32) + (threadIdx.x >> 5)) * wpw;
    const auto load = [&](int64_t b) {
        return b >= 0 && b < (int64_t)total ? __ldg(a.ranges + b) : make_float2(NAN, NAN);  // NaN: no flags
    };
    // ranges of a batch of words (none past the warp's last)
    const auto load_batch = [&](uint32_t w, uint32_t i, float2 r[kFlagBatch]) {
#pragma unroll
        for (uint32_t u = 0; u < kFlagBatch; ++u)
            r[u] = i + u < wpw ? load((int64_t)w * 32 + 32 * (i + u) + lane) : make_float2(NAN, NAN);
    };
    // of the blocks before the warp's first word and after its last
    const auto load_ends = [&](uint32_t w) {
        const int64_t b0 = (int64_t)w * 32;
        return lane == 0 ? load(b0 - 1) : lane == wpw - 1u ? load(b0 + 32 * wpw) : make_float2(NAN, NAN);
    };
    float2 r[kFlagBatch], e;
    load_batch(w0, 0, r);  // on their way while the isovalue is
    e = load_ends(w0);
    if (in) {  // one read of host memory per CTA
        __shared__ float s_iso;
        if (threadIdx.x == 0) s_iso = __ldcv(&in->isovalue);
        __syncthreads();
        iso = s_iso;
    }
    if (blockIdx.x == 0) {
        uint32_t drop = 0;
        if (in) {
            capacity = __ldcv(&in->capacity);
            vert_capacity = __ldcv(&in->vert_capacity);
            drop = __ldcv(&in->debug_drop_tile);
        }
        query_begin(q, iso, false, capacity, vert_capacity, drop);
    }
    for (; w0 < nwords; w0 += step) {
        uint32_t A = 0, B = 0;
        for (uint32_t i = 0; i < wpw; i += kFlagBatch) {
            if (i) load_batch(w0, i, r);
#pragma unroll
            for (uint32_t u = 0; u < kFlagBatch; ++u) {
                const uint32_t wa = __ballot_sync(0xffffffffu, iso >= r[u].x),
                               wb = __ballot_sync(0xffffffffu, iso <= r[u].y);
                if (lane == i + u) {
                    A = wa;
                    B = wb;
                }
            }
        }
        const WordEnds ends = word_ends((w0 + lane) * 32u, a.grid);
        uint32_t pa = __shfl_up_sync(0xffffffffu, A, 1), pb = __shfl_up_sync(0xffffffffu, B, 1);
        uint32_t na = __shfl_down_sync(0xffffffffu, A, 1), nb = __shfl_down_sync(0xffffffffu, B, 1);
        if (lane == 0) {
            pa = iso >= e.x ? 1u << 31 : 0u;
            pb = iso <= e.y ? 1u << 31 : 0u;
        }
        if (lane == wpw - 1u) {
            na = iso >= e.x;
            nb = iso <= e.y;
        }
        if (lane < wpw && w0 + lane < nwords) {
            a.near[w0 + lane] = make_uint4(ends.spread(A, pa, na), ends.spread(B, pb, nb),
                                           ends.spread(A & B, pa & pb, na & nb), A);
            a.up[w0 + lane] = make_uint4(ends.up(A, na), ends.up(B, nb), B, 0u);
        }
        if (w0 + step < nwords) {
            load_batch(w0 + step, 0, r);
            e = load_ends(w0 + step);
        }
    }
}

__global__ void __launch_bounds__(kFlagThreads) k_query_flags(QueryState* q, float iso, uint32_t capacity,
                                                             uint32_t vert_capacity, const QueryInputs* in, FlagArgs a)
{
    query_flags(q, iso, capacity, vert_capacity, in, a);
}

// Ends a query graph: the query state the host reads (the fields before the
// sort histograms) into the host's pinned copy, stored to mapped host memory
// by one warp instead of a copy node.
constexpr uint32_t kHostStateWords = offsetof(QueryState, sort_hist) / 4;

__global__ void k_query_end(const QueryState* q, QueryState* host)
{
    const uint32_t* src = reinterpret_cast<const uint32_t*>(q);
    uint32_t* dst = reinterpret_cast<uint32_t*>(host);
    for (uint32_t i = threadIdx.x; i < kHostStateWords; i += blockDim.x) dst[i] = __ldcg(src + i);
}

void query_end_launch(const QueryState* q, QueryState* host, cudaStream_t s)
{
    k_query_end<<<1, 64, 0, s>>>(q, host);
    count_launches(1);
    BCMC_CUDA(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// k_active
// ---------------------------------------------------------------------------
constexpr int kActThreads = 256;
constexpr int kActiveItems = 4;
constexpr int kActiveTile = kActThreads * kActiveItems;  // blocks per k_active tile

// The last tile of the active test: totals, and the cache growth decision.
__device__ __forceinline__ void active_finish(QueryState* q, uint32_t A, uint32_t N, uint32_t total)
{
    q->num_active = A;
    q->num_new = N;
    const uint32_t old = q->cache_size;
    uint32_t new_size = old;
    if (A > 0 && N > 0) {
        const uint32_t kept = A - N;
        const uint32_t avail = old - kept;
        if (avail < N) {  // js/lru_cache.js:519-522
            uint64_t grown = (uint64_t)old + (3ull * (N - avail) + 1ull) / 2ull;
            if (grown > total) grown = total;
            new_size = align_up((uint32_t)grown, 32u);
        }
        q->display_slots_available = new_size - A;
    }
    q->old_cache_size = old;
    q->new_cache_size = new_size;
    if (new_size > q->capacity) {  // host grows the buffers and re-runs the query
        q->grow_needed = new_size;
        q->num_avail = 0;
    } else {
        q->cache_size = new_size;
        q->num_avail = (A > 0 && N > 0) ? new_size - (A - N) : 0u;
    }
}

// k_active_words: the active test of the MC path (compute_block_active.comp:24-61)
// on k_query_flags' words, with the compaction of the active ids and of the ids
// that no slot holds.  With A = iso >= lo and B = iso <= hi of a block, the
// reference's test over a block's 26 neighbours is (see active_test.cuh)
//   active = (A && anyB) || (B && anyA) || any(A_n && B_n),
// any over the 3x3x3 neighbourhood.  The words hold the ORs along x, so a lane
// ORs the nine (y, z) neighbour rows of its word, each two words and a funnel
// shift, with masks for the blocks that have no such row.
// A block is active for neighbours on all sides, but its cells reach into those
// on the + sides only: where the isovalue lies outside the ranges of the block and
// of these seven (up_a, up_b), all its voxels and ghost voxels are on one side of
// it, and it cannot have vertices.  k_mc looks at the others, the live ones, alone:
// an and of two words here saves it 125 voxel loads and their tests a block (1024 x
// 1024 x 1080, a quarter of whose active blocks have vertices: MC 586 -> 529 us
// for 10 us more here; 512^3 789 -> 771 us for 2).  Blocks whose ranges do not hold
// all their voxels (SoundRanges) are live when they are active.
// A CTA owns one contiguous range of words: it tests them, keeping the results
// in shared memory, publishes its totals, adds up those of the CTAs before
// it in one round trip (cooperative launch: all are resident), and writes its
// ids.  The last CTA with words decides the cache growth.
constexpr int kWordThreads = 256;
constexpr int kWordPerSm = 5;
constexpr uint32_t kWordRange = 2048;  // words whose results fit in shared memory; longer ranges keep them in global memory

// kSameLaunch: other CTAs of this launch wrote the words, which are read from L2.
template <bool kSameLaunch>
__device__ __forceinline__ void active_words(QueryState* q, const ActiveArgs& a, uint32_t wpw, uint32_t range)
{
    __shared__ uint2 s_words[kWordRange];
    __shared__ uint32_t s_live[kWordRange];
    __shared__ uint32_t s_warp[kWordThreads / 32 + 1];
    __shared__ uint2 s_at[kWordThreads];
    __shared__ uint32_t s_sum_a, s_sum_n, s_sum_l, s_pa, s_pn, s_pl;
    constexpr uint32_t kWarps = kWordThreads / 32;
    const uint32_t total = a.total, nwords = div_up(total, 32u), rank = blockIdx.x;
    const uint32_t first = rank * range, end = min(nwords, first + range);
    if (first >= nwords) return;
    const auto word = [](const uint4* p) { return kSameLaunch ? __ldcg(p) : __ldg(p); };
    const uint32_t epoch = status_tag(q);
    const uint3 nb = a.grid.nb;
    const int32_t nx = (int32_t)nb.x;
    const int64_t nxy = (int64_t)nb.x * nb.y;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5, below = (1u << lane) - 1u;
    uint2* words = range <= kWordRange ? s_words : a.words + first;  // active and needed bits
    uint32_t* live_words = range <= kWordRange ? s_live : a.live_words + first;
    if (t == 0) s_sum_a = s_sum_n = s_sum_l = s_pa = s_pn = s_pl = 0;
    __syncthreads();
    uint32_t na = 0, nn = 0, nl = 0;  // the lane's words' counts
    for (uint32_t w0 = first + warp * wpw; w0 < end; w0 += kWarps * wpw) {
        const uint32_t w = w0 + lane, b0 = 32u * w;
        uint32_t act = 0, live = 0;
        if (lane < wpw && w < end) {
            const WordRows in_volume = word_rows(b0, a.grid, a.sound);
            uint32_t any_a = 0, any_b = 0, any_c = 0, up_a = 0, up_b = 0, self_a = 0, self_b = 0;
#pragma unroll
            for (int dz = -1; dz < 2; ++dz)
#pragma unroll
                for (int dy = -1; dy < 2; ++dy) {
                    const uint32_t m = in_volume.mask(dy, dz);
                    // the row's first block; a word out of the volume holds no block that the masks leave
                    const int64_t s = (int64_t)b0 + dz * nxy + dy * nx;
                    const int64_t k = s >> 5;
                    const uint32_t sh = (uint32_t)s & 31u;
                    const int64_t k0 = min(max(k, (int64_t)0), (int64_t)nwords - 1),
                                  k1 = min(max(k + 1, (int64_t)0), (int64_t)nwords - 1);
                    const uint4 lo = word(a.near + k0), hi = word(a.near + k1);
                    any_a |= __funnelshift_r(lo.x, hi.x, sh) & m;
                    any_b |= __funnelshift_r(lo.y, hi.y, sh) & m;
                    any_c |= __funnelshift_r(lo.z, hi.z, sh) & m;
                    if (dz >= 0 && dy >= 0) {
                        const uint4 l = word(a.up + k0), h = word(a.up + k1);
                        up_a |= __funnelshift_r(l.x, h.x, sh) & m;
                        up_b |= __funnelshift_r(l.y, h.y, sh) & m;
                        if (dz == 0 && dy == 0) self_b = l.z;
                    }
                    if (dz == 0 && dy == 0) self_a = lo.w;
                }
            act = (self_a & any_b) | (self_b & any_a) | any_c;
            if (total - b0 < 32u) act &= (1u << (total - b0)) - 1u;
            uint32_t sound = b0 < a.sound.id ? in_volume.sound : 0u;
            if (a.sound.id - b0 < 32u) sound &= (1u << (a.sound.id - b0)) - 1u;
            live = act & ((up_a & up_b) | ~sound);
        }
        // the flags out, and which active blocks no slot holds: four words at a
        // time, four blocks to a lane
        uint32_t need = 0;
        const uint32_t n = min(wpw, end - w0);
#pragma unroll 2
        for (uint32_t i = 0; i < n; i += 4u) {
            const uint32_t on = __shfl_sync(0xffffffffu, act, i + (lane >> 3)) >> (4u * (lane & 7u)) & 15u;
            const uint32_t b = 32u * (w0 + i) + 4u * lane;
            uint32_t no_slot = 0;
            if (i + (lane >> 3) < n) {
                if (b + 4u <= total) {
                    *reinterpret_cast<uint4*>(a.active_out + b) =
                        make_uint4(on & 1u, on >> 1 & 1u, on >> 2 & 1u, on >> 3);
                    if (on && a.item_slots) {
                        const int4 s4 = __ldg(reinterpret_cast<const int4*>(a.item_slots + b));
                        no_slot = on & ((s4.x < 0 ? 1u : 0u) | (s4.y < 0 ? 2u : 0u) | (s4.z < 0 ? 4u : 0u) |
                                        (s4.w < 0 ? 8u : 0u));
                    }
                } else {
                    for (uint32_t k = 0; b + k < total; ++k) {
                        a.active_out[b + k] = on >> k & 1u;
                        if ((on >> k & 1u) && a.item_slots && a.item_slots[b + k] < 0) no_slot |= 1u << k;
                    }
                }
            }
            uint32_t word = no_slot << (4u * (lane & 7u));
            word |= __shfl_xor_sync(0xffffffffu, word, 1);
            word |= __shfl_xor_sync(0xffffffffu, word, 2);
            word |= __shfl_xor_sync(0xffffffffu, word, 4);
            word = __shfl_sync(0xffffffffu, word, 8u * (lane - i));  // lanes i .. i + 3: their word
            if (lane - i < 4u) need = word;
        }
        if (lane < n) {
            words[w - first] = make_uint2(act, need);
            live_words[w - first] = live;
            nl += __popc(live);
            na += __popc(act);
            nn += __popc(need);
        }
    }
    na = __reduce_add_sync(0xffffffffu, na);
    nn = __reduce_add_sync(0xffffffffu, nn);
    nl = __reduce_add_sync(0xffffffffu, nl);
    if (lane == 0 && na) {
        atomicAdd(&s_sum_a, na);
        if (nn) atomicAdd(&s_sum_n, nn);
        if (nl) atomicAdd(&s_sum_l, nl);
    }
    __syncthreads();
    if (a.active_ids)
        cta_prefix_sums<kWordThreads>({{a.status_a, s_sum_a, 30u, &s_pa}, {a.status_n, s_sum_n, 31u, &s_pn}, {a.status_l, s_sum_l, 33u, &s_pl}},
                                      rank, epoch, &q->error, lb_dropped(q, rank));
    else
        cta_prefix_sums<kWordThreads>({{a.status_a, s_sum_a, 30u, &s_pa}, {a.status_n, s_sum_n, 31u, &s_pn}}, rank, epoch,
                                      &q->error, lb_dropped(q, rank));
    __syncthreads();
    uint32_t pa = s_pa, pn = s_pn, pl = s_pl;
    if (end == nwords && t == 0) {
        active_finish(q, pa + s_sum_a, pn + s_sum_n, total);
        q->num_live = pl + s_sum_l;
    }
    if (!a.active_ids) return;
    for (uint32_t c0 = 0; c0 < end - first; c0 += kWordThreads) {
        const uint32_t i = c0 + t;
        const uint2 mine = i < end - first ? words[i] : make_uint2(0u, 0u);
        const uint32_t mine_live = i < end - first ? live_words[i] : 0u;
        uint32_t tot, tot_n = 0, ex_n = 0;
        const uint32_t ex = cta_exclusive_scan<kWordThreads>((uint32_t)__popc(mine.x) | ((uint32_t)__popc(mine_live) << 16),
                                                             s_warp, &tot);
        if (s_sum_n) ex_n = cta_exclusive_scan<kWordThreads>((uint32_t)__popc(mine.y), s_warp, &tot_n);
        s_at[t] = make_uint2(ex, ex_n);
        __syncthreads();
        // a word at a time, so that the ids go out together
        const uint32_t n = min((uint32_t)kWordThreads, end - first - c0);
        for (uint32_t k = warp; k < n; k += kWarps) {
            const uint2 wd = words[c0 + k];
            if (!wd.x) continue;
            const uint32_t wl = live_words[c0 + k];
            const uint2 at = s_at[k];
            const uint32_t b = 32u * (first + c0 + k) + lane;
            const uint32_t place = pa + (at.x & 0xffffu) + __popc(wd.x & below);
            if (wd.x >> lane & 1u) a.active_ids[place] = b;
            if (wd.y >> lane & 1u) a.new_ids[pn + at.y + __popc(wd.y & below)] = b;
            if (wl >> lane & 1u) {
                const uint32_t l = pl + (at.x >> 16) + __popc(wl & below);
                a.live_ids[l] = b;
                a.live_at[l] = place;
            }
        }
        __syncthreads();
        pa += tot & 0xffffu;
        pl += tot >> 16;
        pn += tot_n;
    }
}

__global__ void __launch_bounds__(kWordThreads, kWordPerSm) k_active_words(QueryState* q, ActiveArgs a, uint32_t wpw,
                                                                          uint32_t range)
{
    active_words<false>(q, a, wpw, range);
}

// k_active: the standalone LRU update's side of the same: the items that are
// needed, and of those the ones no slot holds, compacted.
__global__ void __launch_bounds__(kActThreads) k_active(QueryState* q, ActiveArgs a)
{
    __shared__ uint32_t s_warp[kActThreads / 32 + 1];
    __shared__ uint32_t s_tile, s_pa, s_pn;
    const uint32_t total = a.total;
    const uint32_t ntiles = div_up(total, kActiveTile);
    const uint32_t epoch = status_tag(q);
    for (;;) {
        if (threadIdx.x == 0) s_tile = atomicAdd(&q->tiles_active, 1u);
        __syncthreads();
        const uint32_t tile = s_tile;
        if (tile >= ntiles) break;
        // thread -> 4 consecutive items (thread-blocked order = item order)
        const uint32_t b0 = tile * kActiveTile + kActiveItems * threadIdx.x;
        uint32_t act = 0, need = 0;  // bit i = item b0 + i
        if (b0 < total) {
            const uint32_t n = min(4u, total - b0);
            for (uint32_t i = 0; i < n; ++i) act |= (a.item_needed[b0 + i] != 0u ? 1u : 0u) << i;
            if (act) {
                if (n == 4) {
                    const int4 s4 = __ldg(reinterpret_cast<const int4*>(a.item_slots + b0));
                    need = (s4.x < 0 ? 1u : 0u) | (s4.y < 0 ? 2u : 0u) | (s4.z < 0 ? 4u : 0u) | (s4.w < 0 ? 8u : 0u);
                } else {
                    for (uint32_t i = 0; i < n; ++i) need |= (a.item_slots[b0 + i] < 0 ? 1u : 0u) << i;
                }
                need &= act;
            }
        }
        const uint32_t cnt = (uint32_t)__popc(act) | ((uint32_t)__popc(need) << 16);
        uint32_t tot;
        const uint32_t excl = cta_exclusive_scan<kActThreads>(cnt, s_warp, &tot);
        if (threadIdx.x < 32) {
            const uint32_t p =
                lb_dropped(q, tile) ? 0u : warp_lookback(a.status_a, tile, tot & 0xffffu, epoch, &q->error, 30u);
            if (threadIdx.x == 0) s_pa = p;
        } else if (threadIdx.x < 64) {
            const uint32_t p =
                lb_dropped(q, tile) ? 0u : warp_lookback(a.status_n, tile, tot >> 16, epoch, &q->error, 31u);
            if (threadIdx.x == 32) s_pn = p;
        }
        __syncthreads();
        uint32_t pn = s_pn + (excl >> 16);
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i)
            if (need >> i & 1u) a.new_ids[pn++] = b0 + i;
        if (tile == ntiles - 1 && threadIdx.x == 0) active_finish(q, s_pa + (tot & 0xffffu), s_pn + (tot >> 16), total);
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// k_slots: age + mark + init of new slots, fused with the compaction of the
// available slots (ascending slot id) and their ages.
//
// A CTA owns one contiguous range of slots, four to a thread at a time: ages and
// marks them, then, when new items need slots and it has any, joins its count of
// available ones to those of the CTAs before it (ranks are claimed in order, so
// all of them run) and writes their ids and ages.  512-slot tiles claimed one by
// one, each waiting for its claim, its items and their flags in turn, took 80 us
// on the 1024 x 1024 x 1080 volume's 2.6 M slots.
// ---------------------------------------------------------------------------
static_assert(kSlotChunk == 4u * kActThreads, "four slots to a thread");

__device__ __forceinline__ void update_slots(QueryState* q, const SlotArgs& a)
{
    __shared__ uint32_t s_warp[kActThreads / 32 + 1];
    __shared__ uint32_t s_rank, s_sum, s_prefix;
    __shared__ uint32_t s_hist[6][256];  // ~age digits 0-3, then the 16-bit keys' digits 0-1
    __shared__ uint32_t s_bins[kAgeBins];  // age bins (age_bin)
    __shared__ bool s_last;
    if ((a.skip_when_inactive && q->num_active == 0) || q->grow_needed) return;
    const uint32_t old = q->old_cache_size, nsz = q->new_cache_size;  // multiples of 32
    const bool compact = q->num_new > 0;
    const bool hist = compact && a.plan != 0u;
    // the six digit histograms of the sort keys are needed unless the plan is
    // the one-pass one on the age bins; expect that when the last update's was
    // (a misprediction is repaired by the last CTA below)
    const bool digits = hist && q->sort_prev_dense == 0u;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t wide = 0;     // an age without a 16-bit key
    uint32_t binless = 0;  // an age outside the age bins
    if (hist) {
        if (digits)
            for (int i = threadIdx.x; i < 1536; i += kActThreads) (&s_hist[0][0])[i] = 0;
        for (int i = threadIdx.x; i < (int)kAgeBins; i += kActThreads) s_bins[i] = 0;
    }
    if (threadIdx.x == 0) {
        s_rank = atomicAdd(&q->tiles_slots, 1u);
        s_sum = s_prefix = 0;
    }
    __syncthreads();
    const SlotRange mine = slot_range(nsz, gridDim.x, s_rank);
    const uint32_t first = mine.first, end = mine.end;
    uint32_t count = 0;
    for (uint32_t base = first; base < end; base += kSlotChunk) {
        const uint32_t s = base + 4u * threadIdx.x;
        uint32_t age[4] = {100000u, 100000u, 100000u, 100000u}, av[4] = {1u, 1u, 1u, 1u};
        if (s < old) {
            const int4 i4 = *reinterpret_cast<const int4*>(a.slot_item + s);
            const uint4 a4 = *reinterpret_cast<const uint4*>(a.slot_age + s);
            const int32_t it[4] = {i4.x, i4.y, i4.z, i4.w};
            const uint32_t was[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) av[j] = it[j] >= 0 && a.needed[it[j]] != 0u ? 0u : 1u;
#pragma unroll
            for (int j = 0; j < 4; ++j) age[j] = av[j] ? was[j] + 1u : 0u;
        } else if (s < end) {  // lru_cache_init.comp:27-29
            *reinterpret_cast<int4*>(a.slot_item + s) = make_int4(-1, -1, -1, -1);
        }
        if (s >= end) continue;
        *reinterpret_cast<uint4*>(a.slot_age + s) = make_uint4(age[0], age[1], age[2], age[3]);
        *reinterpret_cast<uint4*>(a.slot_avail + s) = make_uint4(av[0], av[1], av[2], av[3]);
        count += av[0] + av[1] + av[2] + av[3];
        if (!hist) continue;
        // plain increments: shared memory adds up a warp's increments of one
        // counter by itself, and ages take few distinct values
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (av[j]) {
                const uint32_t k = ~age[j], k16 = ~age_key16(age[j]), bin = age_bin(age[j]);
                if (!age_has_key16(age[j])) wide = 1;
                if (bin == kAgeBins) binless = 1;
                else atomicAdd(&s_bins[bin], 1u);
                if (digits) {
#pragma unroll
                    for (int d = 0; d < 6; ++d) atomicAdd(&s_hist[d][((d < 4 ? k : k16) >> (8 * (d & 3))) & 255u], 1u);
                }
            }
    }
    if (compact && mine.any()) {
        count = __reduce_add_sync(0xffffffffu, count);
        if (lane == 0 && count) atomicAdd(&s_sum, count);
        __syncthreads();
        cta_prefix_sums<kActThreads>({{a.status, s_sum, 32u, &s_prefix}}, s_rank, q->epoch, &q->error);
        __syncthreads();
        uint32_t run = s_prefix;
        for (uint32_t base = first; base < end; base += kSlotChunk) {
            const uint32_t s = base + 4u * threadIdx.x;
            uint4 av = make_uint4(0u, 0u, 0u, 0u), age = av;
            if (s < end) {
                av = *reinterpret_cast<const uint4*>(a.slot_avail + s);
                age = *reinterpret_cast<const uint4*>(a.slot_age + s);
            }
            uint32_t tot;
            uint32_t p = run + cta_exclusive_scan<kActThreads>(av.x + av.y + av.z + av.w, s_warp, &tot);
            const uint32_t on[4] = {av.x, av.y, av.z, av.w}, ages[4] = {age.x, age.y, age.z, age.w};
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
                if (on[j]) {
                    a.avail_ids[p] = s + j;
                    a.avail_keys[p] = ages[j];
                    ++p;
                }
            run += tot;
        }
    }
    __syncthreads();
    if (!hist) return;
    // this CTA's histograms into q->sort_hist; the last CTA to finish makes
    // the sort's pass plan (what k_sort_hist's last CTA does)
    uint32_t* gh = &q->sort_hist[0][0];  // sort_hist16 follows it
    if (digits)
        for (int i = threadIdx.x; i < 1536; i += kActThreads) {
            const uint32_t c = (&s_hist[0][0])[i];
            if (c) atomicAdd(gh + i, c);
        }
    for (int i = threadIdx.x; i < (int)kAgeBins; i += kActThreads)
        if (s_bins[i]) atomicAdd(a.age_hist + i, s_bins[i]);
    if (__syncthreads_or(wide) && threadIdx.x == 0) atomicOr(&q->sort_wide, 1u);
    if (__syncthreads_or(binless) && threadIdx.x == 0) atomicOr(&q->sort_wide, 2u);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&q->tiles_sort_hist, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const uint32_t flags = *reinterpret_cast<volatile uint32_t*>(&q->sort_wide);
    const bool key16 = (flags & 1u) == 0u;
    // the age bins in use (two per thread, in age order) and how many
    uint32_t cnt[2], used = 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        cnt[k] = __ldcg(a.age_hist + 2u * threadIdx.x + k);
        used += cnt[k] ? 1u : 0u;
    }
    uint32_t distinct;
    const uint32_t below = cta_exclusive_scan<kActThreads>(used, s_warp, &distinct);
    // every age in a bin and at most 256 bins used: one sort pass on the bins'
    // dense ranks, older ages (higher bins) ranked first
    const bool dense = flags == 0u && distinct <= 256u;
    uint32_t* rank_hist = &q->sort_hist16[0][0];  // reused for the ranks' histogram
    if (dense) {
        rank_hist[threadIdx.x] = 0u;
        __syncthreads();
        uint32_t p = below;
#pragma unroll
        for (int k = 0; k < 2; ++k)
            if (cnt[k]) {
                const uint32_t rank = distinct - 1u - p++;
                a.age_rank[2u * threadIdx.x + k] = (uint8_t)rank;
                rank_hist[rank] = cnt[k];
            }
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) a.age_hist[2u * threadIdx.x + k] = 0u;  // zero again for the next update
    if (!dense && !digits) {
        // the one-pass plan was expected and does not apply: the digit
        // histograms from the compacted keys, by this CTA alone (the CTAs
        // accumulated none, so q->sort_hist is still zero)
        const uint32_t n = q->num_avail;
        for (int i = threadIdx.x; i < 1536; i += kActThreads) (&s_hist[0][0])[i] = 0;
        __syncthreads();
        for (uint32_t i0 = 0; i0 < n; i0 += kActThreads) {
            const uint32_t i = i0 + threadIdx.x;
            const bool v = i < n;
            const uint32_t age = v ? __ldcg(a.avail_keys + i) : 0u;
            const uint32_t k = ~age, k16 = ~age_key16(age);
#pragma unroll
            for (int d = 0; d < 6; ++d) {
                const uint32_t digit = v ? ((d < 4 ? k : k16) >> (8 * (d & 3))) & 255u : 256u;
                const uint32_t peers = __match_any_sync(0xffffffffu, digit);
                if (v && lane == (uint32_t)__ffs(peers) - 1u) atomicAdd(&s_hist[d][digit], (uint32_t)__popc(peers));
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < 1536; i += kActThreads) gh[i] = (&s_hist[0][0])[i];
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        q->sort_key16 = dense ? 2u : (key16 ? 1u : 0u);
        q->sort_prev_dense = dense ? 1u : 0u;
    }
    if (dense) sort_plan<kActThreads>(q, q->num_avail, s_warp, rank_hist, 1);
    else if (key16) sort_plan<kActThreads>(q, q->num_avail, s_warp, &q->sort_hist16[0][0], 2);
    else sort_plan<kActThreads>(q, q->num_avail, s_warp, &q->sort_hist[0][0], 4);
}

__global__ void __launch_bounds__(kActThreads) k_slots(QueryState* q, SlotArgs a) { update_slots(q, a); }

// ---------------------------------------------------------------------------
// k_query_front: k_query_flags, k_active_words and k_slots of a small volume in one
// launch, one cluster of CTAs, with the cluster's barrier where the kernels end.
// A query of a small volume is a chain of launches that each take longer to start
// and to drain than to run; beyond kFrontBlocks the sixteen SMs' throughput costs
// more than two launches.  Whole queries, all cached and with 5 % of the blocks
// cached: 4096 blocks 37.0 -> 35.5 and 35.4 -> 33.2 us, 13,824 41.0 -> 39.9 and 41.4 ->
// 40.3, 21,952 41.6 -> 39.7 and 50.6 -> 49.1, 32,768 42.0 -> 43.0 and 44.5 -> 44.4
// (clusters of eight: as good at 4096, 0.5 us slower than the kernels at 13,824).
// With a perf tracker the three run as kernels, whose times it reports.
// ---------------------------------------------------------------------------
constexpr int kFrontCtas = 16;  // the largest cluster, which a kernel has to ask for
constexpr uint32_t kFrontBlocks = 24576;
static_assert(kFlagThreads == kWordThreads && kFlagThreads == kActThreads, "one CTA does the work of all three");

__device__ __forceinline__ void cluster_barrier()
{
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __cluster_dims__(kFrontCtas, 1, 1) __launch_bounds__(kActThreads)
    k_query_front(QueryState* q, const QueryInputs* in, FlagArgs f, ActiveArgs a, uint32_t wpw, uint32_t range, SlotArgs sa)
{
    query_flags(q, 0.0f, 0u, 0u, in, f);
    cluster_barrier();
    active_words<true>(q, a, wpw, range);
    cluster_barrier();
    update_slots(q, sa);
}

// ---------------------------------------------------------------------------
// k_assign: lru_cache_update.comp:19-37 (+ the new block's data into its slot
// when `words` is set: copied from the staging buffer k_decode_new filled,
// decoded here for new-block indices past it).
// ---------------------------------------------------------------------------
constexpr int kAssignThreads = 128;

__global__ void __launch_bounds__(kAssignThreads) k_assign(QueryState* q, AssignArgs a)
{
    if (q->num_active == 0 || q->grow_needed) return;
    const uint32_t n = q->num_new;
    const uint32_t size = q->new_cache_size;
    const uint32_t* __restrict__ sorted = q->sort_final == 1 ? a.sorted_b : a.sorted_c;
    const uint32_t first_decode = a.stage ? a.stage_blocks : 0u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t item = a.new_ids[i];
        const uint32_t slot = sorted[i];
        if (slot >= size) {  // cannot happen with a consistent sort; never write out of bounds
            atomicCAS(&q->error, 0u, 50u);
            continue;
        }
        const int32_t prev = a.slot_item[slot];
        if (prev != -1) a.item_slots[prev] = -1;
        a.slot_age[slot] = 0;
        a.slot_item[slot] = (int32_t)item;
        a.slot_avail[slot] = 0;
        a.item_slots[item] = (int32_t)slot;
        if (a.words && i >= first_decode) {
            // decoded here: every new block of the standalone LRU update, the ones
            // past the staging buffer on the query path.  Rare enough on the query
            // path that the words are read in place and the plane scratch is
            // thread-local, which keeps this kernel free of shared memory for its
            // assignment and copy work.
            __align__(16) uint32_t pl[64];
            float v[64];
            zfp_decode_staged(reinterpret_cast<const uint32_t*>(a.words + (uint64_t)item * (a.max_bits / 64u)),
                              a.max_bits, pl, v);
            float4* d4 = reinterpret_cast<float4*>(a.cache + (uint64_t)slot * 64u);
#pragma unroll
            for (int k = 0; k < 16; ++k) d4[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
        }
    }
    if (!a.stage) return;
    // staged blocks into their slots: 16 threads per block, 16 B each
    const uint32_t ns = n < a.stage_blocks ? n : a.stage_blocks;
    const float4* __restrict__ src = reinterpret_cast<const float4*>(a.stage);
    float4* dst = reinterpret_cast<float4*>(a.cache);
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < ns * 16u; e += gridDim.x * blockDim.x) {
        const uint32_t i = e >> 4, k = e & 15u;
        const uint32_t slot = sorted[i];
        if (slot < size) dst[(uint64_t)slot * 16u + k] = __ldcs(src + (uint64_t)i * 16u + k);
    }
}

// ---------------------------------------------------------------------------
// k_decode_new: zfp_decompress_block.comp's decode of the query's new blocks,
// by new-block index into the staging buffer.  It depends on the active test
// only, so it runs beside k_slots and the sort; k_assign then copies the
// staged blocks into the slots the sort chose.
// ---------------------------------------------------------------------------
constexpr int kDecodeNewThreads = 128;

__global__ void __launch_bounds__(kDecodeNewThreads, 5) k_decode_new(const QueryState* q, DecodeArgs a)
{
    if (q->num_active == 0 || q->grow_needed) return;
    const uint32_t n = q->num_new < a.stage_blocks ? q->num_new : a.stage_blocks;
    extern __shared__ __align__(16) uint32_t s_words[];
    const uint32_t rate = a.max_bits / 64u;
    uint32_t* pl = zfp_stage_planes(s_words, kDecodeNewThreads, rate);
    if (threadIdx.x < 4) s_words[kDecodeNewThreads * 2u * rate + threadIdx.x] = 0u;
    const uint32_t wb = threadIdx.x & ~31u;
    for (uint32_t i0 = blockIdx.x * kDecodeNewThreads; i0 < n; i0 += gridDim.x * kDecodeNewThreads) {
        const uint32_t i = i0 + threadIdx.x;
        __syncthreads();
        if (i < n) zfp_stage_block(a.words, a.new_ids[i], rate, s_words);
        __syncthreads();
        if (i0 + wb >= n) continue;  // the whole warp
        const bool mine = i < n;
        float v[64];
        if (mine) zfp_decode_staged(s_words + threadIdx.x * 2u * rate, a.max_bits, pl, v);
        zfp_store_warp(pl, v, mine, a.stage + (uint64_t)(i0 + wb) * 64u, n - (i0 + wb));
    }
}

// ---------------------------------------------------------------------------
// k_mc: marching cubes over the active blocks.
// ---------------------------------------------------------------------------
constexpr int kMcThreads = 512;
constexpr int kMcWarps = kMcThreads / 32;
constexpr int kMcPerSm = 2;  // resident CTAs per SM (the grid: one launch, all resident)
// Ranges of at most this many blocks per CTA (small queries) are emitted by
// their own CTA; longer ones go through a grid barrier and an even share-out.
constexpr uint32_t kMcOwnRange = kMcWarps * kMcBlocks;
// Ranges longer than this are counted by all CTAs together, which costs a barrier.
// The same queries both ways, 76 isovalues of 224^3 to 1024 x 1024 x 1080 voxels: up
// to 2,000 active blocks to a CTA the barrier costs 2 to 4 us (512^3 82 -> 84, 256^3 47
// -> 49), to 5,000 neither way is faster by more than 1 %, above that sharing gains 0.2
// to 1.2 % (800^3 653 -> 649 us, 640^3 1,026 -> 1,018, 1024 x 1024 x 1080 1,753 -> 1,733).
constexpr uint32_t kMcSharedRange = 4096;

// Marching cubes over the active blocks, one cooperative launch (every CTA
// resident), all of its block work done by single warps (mc_common.cuh):
//   count pass: the live blocks in batches of four to a warp: look the neighbours up,
//     load the grids and count the triangles of the cells from the corner masks;
//     block totals are kept.  Each CTA counts its own range of the blocks, or,
//     when the ranges are long, its share of batches from the whole grid, with a
//     barrier after it: a batch's cost depends on whether the surface passes
//     through it (kMcSharedRange);
//   each CTA publishes its range's totals and adds up those of the CTAs before
//     it: its vertex offset and its place in the blocks-with-vertices list;
//   it writes its entries of that list and their vertex offsets, then a grid
//     barrier;
//   emit: the list in runs of up to four consecutive entries, warp by warp over
//     the whole grid.  Entries that follow each other in the list have their
//     vertices one after the other, so a run needs only its first entry's offset.
// Few blocks (at most kMcOwnRange a CTA): a warp keeps the grids of the up to
// four blocks it counted and emits them itself, once its place is known; the
// barrier and the second load would take longer than the balance saves (64^3:
// 16.6 -> 13.9 us against own entries shared out in the CTA and loaded again).
// Output order = the reference's: active-block order, cell order, table order.
// kHost: the vertices go to page-locked host memory (a.host_verts).
template <bool kHost>
__global__ void __launch_bounds__(kMcThreads, kMcPerSm) k_mc(QueryState* q, McArgs a)
{
    extern __shared__ __align__(16) unsigned char s_dyn[];
    McShared<kMcThreads, kHost>& sm = *reinterpret_cast<McShared<kMcThreads, kHost>*>(s_dyn);
    __shared__ uint32_t s_warp[kMcWarps + 1];
    __shared__ uint32_t s_cnt[kMcOwnRange];  // few blocks: the counts of the CTA's
    __shared__ uint32_t s_pv, s_pb, s_cta_v, s_cta_b;

    const uint32_t A = q->num_live;
    if (A == 0 || q->grow_needed) return;
    const uint32_t epoch = q->epoch;
    const float iso = q->isovalue;
    const uint32_t cap = q->vert_capacity;
    const uint32_t slots = q->cache_size;
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5, jb = lane >> 3;
    const uint32_t G = gridDim.x, rank = blockIdx.x;
    const uint32_t share = div_up(A, G);
    const bool own = share <= kMcOwnRange, together = share > kMcSharedRange;
    const uint32_t range = own ? align_up(share, (uint32_t)kMcWarps) : share;
    const uint32_t start = min(A, rank * range), end = min(A, start + range);
    // ranks 0 .. worked - 1 have blocks in their range
    const uint32_t worked = div_up(A, range);
    mc_shared_begin(sm);
    if (t == 0) s_cta_v = s_cta_b = s_pv = s_pb = 0;
    const McLane geo = mc_lane(a.cache, sm.warp[warp].slot);
    McWarpMem<kHost>& mem = sm.warp[warp];
    const auto look = [&](bool valid, uint32_t id) {
        return mc_look(valid, id, a.grid, a.item_slots, [&](uint32_t nid) { return __ldg(a.active + nid); });
    };
    const auto look_end = [&](const McLook& l) {
        uint32_t has;
        mc_look_end(l, sm.tab, slots, &q->error, 51u, mem.slot, has);
        return has;
    };

    // ---- count pass: ids two rounds ahead, lookups one round ahead
    uint32_t own_n = 0, own_id = 0, own_has = 0, own_at = 0;  // few blocks: the warp's batch
    const uint32_t batch = own ? range / kMcWarps : kMcBlocks;
    {
        const uint32_t stop = together ? A : end, step = (together ? G : 1u) * kMcWarps * batch;
        uint32_t base = together ? (rank * kMcWarps + warp) * batch : start + warp * batch;
        const auto mine = [&](uint32_t at) { return jb < batch && at + jb < stop; };
        const auto load_id = [&](uint32_t at) { return mine(at) ? __ldg(a.live_ids + at + jb) : 0u; };
        McLook next = look(mine(base), load_id(base));
        uint32_t id2 = load_id(base + step);
        uint32_t wv = 0, wb = 0;
        async_wait<1>();
        __syncthreads();
        for (; base < stop; base += step) {
            const uint32_t n = min(batch, stop - base), id = next.id;
            const uint32_t has = look_end(next);
            uint32_t total = 0;
            float f[kMcBlocks][4];
            mc_voxels(geo, n, f);
            next = look(mine(base + step), id2);
            id2 = load_id(base + 2u * step);
            if (own) {
                own_n = n;
                own_id = id;
                own_has = has;
                if (lane < n) own_at = __ldg(a.live_at + base + lane);
#pragma unroll
                for (uint32_t j = 0; j < kMcBlocks; ++j)
                    if (j < n) {
#pragma unroll
                        for (uint32_t r = 0; r < 4; ++r) mem.vol[j][lane + 32u * r] = f[j][r];
                    }
            }
#pragma unroll
            for (uint32_t j = 0; j < kMcBlocks; ++j)
                if (j < n) {
                    uint32_t c0, c1;
                    if (!mc_cases<true>(geo, f[j], iso, __shfl_sync(kFull, has, 8u * j), c0, c1)) continue;
                    const uint32_t v = 3u * __reduce_add_sync(kFull, (uint32_t)sm.tab.count.n[c0] + sm.tab.count.n[c1]);
                    if (lane == j) total = v;
                    wv += v;
                    wb += v != 0u ? 1u : 0u;
                }
            if (lane < n) {
                a.block_counts[base + lane] = total;
                if (own) s_cnt[base - start + lane] = total;
            }
        }
        if (!together && lane == 0 && wb) {
            atomicAdd(&s_cta_v, wv);
            atomicAdd(&s_cta_b, wb);
        }
    }
    if (together) {
        grid_barrier(&q->mc_arrived, G, &q->error, 42u);
        uint32_t v = 0, b = 0;
        for (uint32_t i = start + t; i < end; i += kMcThreads) {
            const uint32_t c = __ldcg(a.block_counts + i);
            v += c;
            b += c ? 1u : 0u;
        }
        v = __reduce_add_sync(kFull, v);
        b = __reduce_add_sync(kFull, b);
        if (lane == 0 && b) {
            atomicAdd(&s_cta_v, v);
            atomicAdd(&s_cta_b, b);
        }
    }
    __syncthreads();
    if (rank < worked)
        cta_prefix_sums<kMcThreads>({{a.status_v, s_cta_v, 40u, &s_pv}, {a.status_b, s_cta_b, 41u, &s_pb}}, rank, epoch,
                                    &q->error);
    async_wait<0>();
    __syncthreads();
    uint32_t pv = s_pv, pb = s_pb;
    if (rank == worked - 1 && t == 0) {
        q->num_verts = pv + s_cta_v;
        q->num_with_verts = pb + s_cta_b;
    }
    const bool fits = (uint64_t)pv + s_cta_v <= cap;
    if (!fits && t == 0) atomicOr(&q->vert_overflow, 1u);

    if (own) {
        if (!fits || own_n == 0) return;
        // the CTA's blocks before the warp's: their vertices, and those that have any
        const uint32_t first = warp * batch, done = first < 32u ? first : 32u;
        static_assert(kMcOwnRange <= 64, "two counts to a lane");
        const uint32_t c0 = lane < done ? s_cnt[lane] : 0u, c1 = 32u + lane < first ? s_cnt[32u + lane] : 0u;
        pv += __reduce_add_sync(kFull, c0 + c1);
        pb += __popc(__ballot_sync(kFull, c0 != 0u)) + __popc(__ballot_sync(kFull, c1 != 0u));
        // the warp's own
        const uint32_t c = lane < own_n ? s_cnt[first + lane] : 0u;
        const uint32_t off = pv + mc_scan(c) - c;
        const uint32_t some = __ballot_sync(kFull, c != 0u);
        if (c) {
            const uint32_t r = pb + __popc(some & ((1u << lane) - 1u));
            a.with_verts[r] = own_at;
            a.vert_offsets[r] = off;
        }
        if (!some) return;
        McSink<kHost> sink{a.verts + pv};
        mc_emit<kHost, true>(geo, sm.tab, mem, own_n, own_id, own_has, iso, sink, [] {});
        sink.finish(mem.out);
        return;
    }
    // the range's blocks with vertices: their list entries and vertex offsets
    if (fits)
        for (uint32_t b0 = start; b0 < end; b0 += kMcThreads) {
            const uint32_t i = b0 + t;
            const uint32_t c = i < end ? __ldcg(a.block_counts + i) : 0u, at = i < end ? __ldg(a.live_at + i) : 0u;
            // <= 512 blocks x 64 cells x 15 vertices < 2^20, and the blocks above them
            static_assert(kMcThreads * 64 * 15 < 1 << 20 && kMcThreads < 1 << 12, "fields of the scan");
            uint32_t tot;
            const uint32_t ex = cta_exclusive_scan<kMcThreads>(c | (c ? 1u << 20 : 0u), s_warp, &tot);
            if (c) {
                const uint32_t r = pb + (ex >> 20);
                a.with_verts[r] = at;
                a.vert_offsets[r] = pv + (ex & 0xfffffu);
            }
            pv += tot & 0xfffffu;
            pb += tot >> 20;
        }
    grid_barrier(&q->mc_arrived, together ? 2u * G : G, &q->error, 42u);
    if (__ldcg(&q->error) | __ldcg(&q->vert_overflow)) return;
    // emit: runs of `per` entries, one from each warp's turn over the grid; into
    // host memory a turn is four runs that follow each other, which leaves fewer
    // windows of 32 vertices partly filled.  A run's list entries are read two
    // runs ahead, its block ids and neighbours one run ahead.
    const uint32_t W = __ldcg(&q->num_with_verts);
    const uint32_t per = min(kMcBlocks, div_up(W, G * kMcWarps));
    constexpr uint32_t kRuns = kHost ? 4u : 1u;
    const uint32_t turn = per * kRuns, skip = (G * kMcWarps - 1u) * turn;
    const auto after = [&](uint32_t at, uint32_t run) { return at + per + (run == kRuns - 1u ? skip : 0u); };
    const auto mine = [&](uint32_t at) { return jb < per && at + jb < W; };
    const auto load_entry = [&](uint32_t at) { return mine(at) ? __ldcg(a.with_verts + at + jb) : 0u; };
    const auto load_id = [&](uint32_t at, uint32_t entry) { return mine(at) ? __ldg(a.active_ids + entry) : 0u; };
    uint32_t at = (rank * kMcWarps + warp) * turn, run = 0;
    if (at >= W) return;
    McLook next = look(mine(at), load_id(at, load_entry(at)));
    uint32_t entry = load_entry(after(at, 0u));
    McSink<kHost> sink{a.verts + __ldcg(a.vert_offsets + at)};
    for (;;) {
        const uint32_t n = min(per, W - at), id = next.id;
        const uint32_t has = look_end(next);
        mc_grids(geo, mem, n);
        const uint32_t at1 = after(at, run), run1 = run == kRuns - 1u ? 0u : run + 1u;
        const uint32_t id1 = load_id(at1, entry);
        entry = load_entry(after(at1, run1));
        const uint32_t off1 = run1 == 0u && at1 < W ? __ldcg(a.vert_offsets + at1) : 0u;
        mc_emit<kHost, true>(geo, sm.tab, mem, n, id, has, iso, sink, [&] { next = look(mine(at1), id1); });
        at = at1;
        run = run1;
        if (at >= W) break;
        if (run == 0u) {
            sink.finish(mem.out);
            sink.start(a.verts + off1);
        }
    }
    sink.finish(mem.out);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static int pgrid(bcmc_ctx* ctx, uint32_t tiles, uint32_t per_sm)
{
    const uint32_t r = (uint32_t)ctx->num_sms * per_sm;
    return (int)(tiles < r ? (tiles ? tiles : 1) : r);
}

void query_begin_launch(QueryState* q, float iso, int mc_only, uint32_t capacity, uint32_t vert_capacity,
                        cudaStream_t s)
{
    k_query_begin<<<1, 256, 0, s>>>(q, iso, mc_only, capacity, vert_capacity);
    count_launches(1);
    BCMC_CUDA(cudaGetLastError());
}

size_t flag_bytes(uint64_t total) { return (size_t)((total + 31u) / 32u) * (2u * sizeof(uint4) + sizeof(uint2) + 4u); }

SoundRanges sound_ranges(const uint32_t dims[3], const BlockGrid& grid, uint64_t ranged)
{
    // the last block on an axis that is not a multiple of 4 has voxels past the
    // volume, which its range leaves out and its grid does not
    const auto axis = [](uint32_t n, uint32_t blocks) { return n % 4u == 0u ? blocks : blocks > 2u ? blocks - 2u : 0u; };
    const uint64_t total = (uint64_t)grid.nb.x * grid.nb.y * grid.nb.z, reach = (uint64_t)grid.nb.x * grid.nb.y + grid.nb.x + 1u;
    return {axis(dims[0], grid.nb.x), axis(dims[1], grid.nb.y), axis(dims[2], grid.nb.z),
            (uint32_t)(ranged >= total ? total : ranged > reach ? ranged - reach : 0u)};
}

// CTAs of k_active_words resident per SM: the bound of its cooperative grid
static uint32_t word_per_sm()
{
    static const uint32_t n = [] {
        int r = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, k_active_words, kWordThreads, 0) != cudaSuccess || r < 1) r = 1;
        return (uint32_t)std::min(r, kWordPerSm);
    }();
    return n;
}

// Words a warp takes, a multiple of 4 up to a word to a lane: enough for
// `warps_per_sm` warps on every SM first, then longer runs (4 words each keep
// the 64^3 volume's 128 words on 32 warps).
static uint32_t words_per_warp(const bcmc_ctx* ctx, uint32_t nwords, uint32_t warps_per_sm)
{
    const uint32_t w = align_up(div_up(nwords, (uint32_t)ctx->num_sms * warps_per_sm), 4u);
    return w >= 32u ? 32u : w;
}

void query_flags_launch(bcmc_ctx* ctx, QueryState* q, float iso, uint32_t capacity, uint32_t vert_capacity,
                        const float* ranges, const BlockGrid& grid, uint32_t total, void* words, cudaStream_t s,
                        const QueryInputs* in)
{
    const uint32_t nwords = div_up(total, 32u), wpw = words_per_warp(ctx, nwords, 32u);
    uint4* near = static_cast<uint4*>(words);
    const FlagArgs f{reinterpret_cast<const float2*>(ranges), grid, total, wpw, near,
                     near + nwords};
    k_query_flags<<<pgrid(ctx, div_up(nwords, wpw * (kFlagThreads / 32)), 8), kFlagThreads, 0, s>>>(
        q, iso, capacity, vert_capacity, in, f);
    count_launches(1);
    BCMC_CUDA(cudaGetLastError());
}

// Where the words of a query lie in their buffer (flag_bytes).
static void word_buffers(ActiveArgs& a, void* words, uint32_t nwords)
{
    a.near = static_cast<const uint4*>(words);
    a.up = a.near + nwords;
    a.words = reinterpret_cast<uint2*>(static_cast<uint4*>(words) + 2u * (size_t)nwords);
    a.live_words = reinterpret_cast<uint32_t*>(a.words + nwords);
}

void active_words_launch(bcmc_ctx* ctx, QueryState* q, ActiveArgs a, void* words, cudaStream_t s)
{
    const uint32_t nwords = div_up(a.total, 32u), wpw = words_per_warp(ctx, nwords, kWordThreads / 32);
    word_buffers(a, words, nwords);
    // a CTA an SM first: the CTAs wait for each other's counts (256^3: 128 of them
    // 1.3 us faster than 256); then a range of whole rounds per resident CTA
    const uint32_t round = wpw * (kWordThreads / 32);
    const uint32_t range = div_up(div_up(nwords, round), (uint32_t)ctx->num_sms * word_per_sm()) * round;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(div_up(nwords, range));
    cfg.blockDim = dim3(kWordThreads);
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    BCMC_CUDA(cudaLaunchKernelEx(&cfg, k_active_words, q, a, wpw, range));
    count_launches(1);
}

// Whether the device has room for the cluster (a slice of one may not).
static bool front_fits()
{
    static const bool fits = [] {
        cudaLaunchAttribute attr{};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = kFrontCtas;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kFrontCtas);
        cfg.blockDim = dim3(kActThreads);
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int n = 0;
        const bool ok = cudaFuncSetAttribute(k_query_front, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&n, k_query_front, &cfg) == cudaSuccess && n > 0;
        if (!ok) cudaGetLastError();
        return ok;
    }();
    return fits;
}

bool query_front_takes(uint32_t total) { return total <= kFrontBlocks && front_fits(); }

void query_front_launch(QueryState* q, const QueryInputs* in, const float* ranges, ActiveArgs a, void* words, const SlotArgs& sa,
                        cudaStream_t s)
{
    constexpr uint32_t kWarps = kWordThreads / 32;
    const uint32_t nwords = div_up(a.total, 32u), wpw = std::min(align_up(div_up(nwords, kFrontCtas * kWarps), 4u), 32u);
    const uint32_t range = div_up(div_up(nwords, wpw * kWarps), kFrontCtas) * wpw * kWarps;
    uint4* near = static_cast<uint4*>(words);
    const FlagArgs f{reinterpret_cast<const float2*>(ranges), a.grid, a.total, wpw, near, near + nwords};
    word_buffers(a, words, nwords);
    BCMC_CUDA(cudaFuncSetAttribute(k_query_front, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    k_query_front<<<kFrontCtas, kActThreads, 0, s>>>(q, in, f, a, wpw, range, sa);
    count_launches(1);
    BCMC_CUDA(cudaGetLastError());
}

void active_launch(bcmc_ctx* ctx, QueryState* q, const ActiveArgs& a, cudaStream_t s)
{
    k_active<<<pgrid(ctx, div_up(a.total, kActiveTile), 8), kActThreads, 0, s>>>(q, a);
    count_launches(1);
    BCMC_CUDA(cudaGetLastError());
}

void slots_launch(bcmc_ctx* ctx, QueryState* q, const SlotArgs& a, uint32_t max_slots, cudaStream_t s)
{
    k_slots<<<pgrid(ctx, div_up(max_slots, kSlotChunk), 4), kActThreads, 0, s>>>(q, a);
    count_launches(1);
    BCMC_CUDA(cudaGetLastError());
}

void assign_launch(bcmc_ctx* ctx, QueryState* q, const AssignArgs& a, uint32_t max_new, cudaStream_t s)
{
    k_assign<<<pgrid(ctx, div_up(max_new, (uint32_t)kAssignThreads), 16), kAssignThreads, 0, s>>>(q, a);
    count_launches(1);
    BCMC_CUDA(cudaGetLastError());
}

void decode_new_launch(bcmc_ctx* ctx, const QueryState* q, const DecodeArgs& a, cudaStream_t s)
{
    // two CTAs per SM: the branch it runs on must leave room for the slot
    // selection's CTAs, the critical path beside it
    const size_t smem = zfp_stage_smem(kDecodeNewThreads, a.max_bits / 64u);
    allow_smem(k_decode_new, smem);
    k_decode_new<<<pgrid(ctx, div_up(a.stage_blocks ? a.stage_blocks : 1u, (uint32_t)kDecodeNewThreads), 2),
                   kDecodeNewThreads, smem, s>>>(q, a);
    count_launches(1);
    BCMC_CUDA(cudaGetLastError());
}

static void mc_allow_smem()
{
    allow_smem(k_mc<false>, sizeof(McShared<kMcThreads, false>));
    allow_smem(k_mc<true>, sizeof(McShared<kMcThreads, true>));
}

// CTAs of k_mc resident per SM: the bound of its cooperative grid
static uint32_t mc_per_sm()
{
    static const uint32_t n = [] {
        constexpr size_t sa = sizeof(McShared<kMcThreads, false>), sb = sizeof(McShared<kMcThreads, true>);
        int a = 0, b = 0;
        mc_allow_smem();
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_mc<false>, kMcThreads, sa) != cudaSuccess) a = 1;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_mc<true>, kMcThreads, sb) != cudaSuccess) b = 1;
        const int m = std::min(std::min(a, b), kMcPerSm);
        return (uint32_t)(m > 0 ? m : 1);
    }();
    return n;
}

void mc_launch(bcmc_ctx* ctx, QueryState* q, const McArgs& a, uint32_t max_active, cudaStream_t s)
{
    mc_allow_smem();  // a setting of the current device
    // cooperative: the kernel's grid barrier needs every CTA resident
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(mc_grid(ctx, max_active));
    cfg.blockDim = dim3(kMcThreads);
    cfg.dynamicSmemBytes = a.host_verts ? sizeof(McShared<kMcThreads, true>) : sizeof(McShared<kMcThreads, false>);
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (a.host_verts) BCMC_CUDA(cudaLaunchKernelEx(&cfg, k_mc<true>, q, a));
    else BCMC_CUDA(cudaLaunchKernelEx(&cfg, k_mc<false>, q, a));
    count_launches(1);
}

uint32_t active_tiles(uint32_t total) { return div_up(total, kActiveTile); }
// one CTA per range of active blocks, every CTA resident; at least a block to a warp
uint32_t mc_grid(bcmc_ctx* ctx, uint32_t max_active)
{
    const uint32_t r = (uint32_t)ctx->num_sms * mc_per_sm(), most = div_up(max_active ? max_active : 1, (uint32_t)kMcWarps);
    return most < r ? most : r;
}

}  // namespace bcmc
