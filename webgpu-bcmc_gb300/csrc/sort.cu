// sort.cu -- onesweep LSD radix sort of (uint32 key, uint32 value) pairs.
//
// Replaces RadixSorter.sort (js/radix_sort_by_key.js:161-400): the reference
// sorts 64-element chunks with 32 one-bit splits (radix_sort_chunk.comp), merges
// them pairwise log2(chunks) times (merge_sorted_chunks.comp, where elements of
// the right half come first among equal keys, :82-86) and, for a descending
// sort, reverses the result (reverse_buffer.comp).  That fixes the order among
// equal keys:
//   ascending : key asc,  then chunk (index/64) desc, then index asc
//   descending: key desc, then chunk asc,             then index desc
// Here one stable LSD radix sort reproduces it: the first pass reads the input
// through a permutation that lists the elements in that tie order, and sorts
// ~key for a descending sort.
//
// Kernels: one cooperative kernel that runs the pass of each 8-bit digit in which
// keys differ, grid barriers between them: tiles of 4096
// keys are ranked with warp match/popc, each tile finds its 256 digits' places
// from the tiles' counts before it, and keys are scattered via shared memory
// so that global writes come out in runs.  Up to 304 tiles it finds the digits'
// places by itself; for more, a histogram/plan kernel goes before (all four digit
// histograms in one read, exclusive bucket offsets, and which passes can be skipped
// because every key shares the digit).
//
// The LRU's age sort skips the histogram kernel: k_slots, which compacts the
// ages, accumulates the histograms and makes the plan (sort_plan).  When every
// age has a 16-bit key (age_key16) the plan sorts on that key (sort_key16 1),
// so the first pass maps each age through it and two digit passes suffice;
// when every age lies in an age bin (age_bin) and at most 256 bins are used,
// on the bins' dense ranks (sort_key16 2, older ages ranked first, from a
// table k_slots builds): one pass.
#include <algorithm>

#include "bcmc_impl.h"

namespace bcmc {

// Sequence position q -> input index p giving the reference's tie order.
__device__ __forceinline__ uint32_t tie_perm(uint32_t q, uint32_t n, int reverse)
{
    const uint32_t chunks = (n + 63u) >> 6;
    const uint32_t last_len = n - 64u * (chunks - 1u);
    if (reverse) {
        const uint32_t c = q >> 6, r = q & 63u;
        const uint32_t len = (c == chunks - 1u) ? last_len : 64u;
        return 64u * c + (len - 1u - r);
    }
    if (q < last_len) return 64u * (chunks - 1u) + q;
    const uint32_t qq = q - last_len;
    return 64u * (chunks - 2u - (qq >> 6)) + (qq & 63u);
}

constexpr int kHistThreads = 512;

__global__ void __launch_bounds__(kHistThreads) k_sort_hist(QueryState* q, const uint32_t* d_n, uint32_t n_host,
                                                   const uint32_t* __restrict__ keys, int reverse)
{
    __shared__ uint32_t h[4 * 256];
    __shared__ uint32_t warp_sums[kHistThreads / 32 + 1];
    __shared__ bool is_last;
    const uint32_t n = d_n ? *d_n : n_host;
    for (int i = threadIdx.x; i < 1024; i += kHistThreads) h[i] = 0;
    __syncthreads();
    // plain increments: shared memory adds up a warp's increments of one counter
    // by itself, whether the keys are spread (a match per digit and warp took
    // 39 us on 2^20 random keys) or take few distinct values, as ages do; few
    // CTAs, since each ends with an atomic per counter
    const uint32_t flip = reverse ? 0xffffffffu : 0u;
    const uint32_t step = gridDim.x * kHistThreads;
    for (uint32_t i0 = blockIdx.x * kHistThreads + threadIdx.x; i0 < n; i0 += 8u * step) {
        uint32_t k[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) k[u] = i0 + u * step < n ? __ldg(keys + i0 + u * step) : 0u;
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (i0 + u * step < n) {
#pragma unroll
                for (int d = 0; d < 4; ++d) atomicAdd(&h[256 * d + (((k[u] ^ flip) >> (8 * d)) & 255u)], 1u);
            }
    }
    __syncthreads();
    uint32_t* gh = &q->sort_hist[0][0];
    for (int i = threadIdx.x; i < 1024; i += kHistThreads)
        if (h[i]) atomicAdd(gh + i, h[i]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(&q->tiles_sort_hist, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    sort_plan<kHistThreads>(q, n, warp_sums, &q->sort_hist[0][0], 4);
}

// All the digit passes of the plan in one cooperative launch: the passes
// that run are separated by grid barriers (each reads what the one before it
// scattered, so its key and value loads bypass L1), the others cost nothing.
//
// A tile's place for each digit is the sum of the tiles' counts before it.  Where
// every tile has a CTA of its own (up to 304 tiles), all have their counts at the
// same time and a look-back walks over nearly all of them, eight to a round trip;
// there the tiles store their counts, pass a barrier, and each adds up the rows
// before its own, 256 counts to a warp's load, in one round (kSortWave: from so
// many tiles on the barrier and the sum are the faster; below, the walk is short).
// More tiles are claimed in order and look back, which then mostly finds sums.
// 2^20 random pairs: 88 us by look-back, four passes.
//
// b.out_keys set: the last pass scatters to there, with the key transform undone,
// unless it is the only one (its input lies there): then the CTAs copy at the end.
//
// kSelf: no histogram kernel went before; every tile has a CTA of its own.  The
// first pass tells which bits differ between keys, so that every CTA knows after
// its barrier which digits to sort on, and a pass adds up all tiles' counts, not
// only those before its own, which gives it the digits' totals and so their
// places.  That doubles the counts read (128 KB a CTA at most, from L2) and saves
// a read of the keys and a launch: 2^20 random pairs 83 -> 81 us, 300,000 70 -> 60
// us, 64 44 -> 37 us; of 16 bits 55 -> 49, 47 -> 38, 33 -> 27 us.
constexpr uint32_t kSortWave = 8;

template <bool kSelf>
__global__ void __launch_bounds__(kSortThreads, 2) k_sort(QueryState* q, const uint32_t* d_n, uint32_t n_host,
                                                       SortBuffers b, int reverse)
{
    __shared__ __align__(16) uint32_t s_keys[kSortTile];
    __shared__ __align__(16) uint32_t s_vals[kSortTile];
    __shared__ __align__(16) uint16_t s_whist[kSortThreads / 32][256];  // per warp and digit: < 2^16
    __shared__ uint32_t s_start[256];
    __shared__ uint32_t s_gbase[256];
    __shared__ uint32_t s_warp_sums[kSortThreads / 32 + 1];
    __shared__ uint32_t s_tile, s_set, s_clear;

    const uint32_t n = d_n ? *d_n : n_host;
    const uint32_t ntiles = div_up(n, kSortTile);
    const bool wave = kSelf || (b.counts && ntiles >= kSortWave && ntiles <= gridDim.x);
    const uint32_t ctas = wave ? ntiles : gridDim.x;
    if (blockIdx.x >= ctas) return;
    uint32_t barriers = 0;
    uint32_t run_passes = 1u, ran = 0, cur = 0;  // kSelf: until the first pass's barrier
    if (!kSelf) {
        run_passes = 0;
        for (uint32_t pass = 0; pass < 4u; ++pass) run_passes |= (q->sort_run[pass] ? 1u : 0u) << pass;
    } else if (threadIdx.x == 0) {
        s_set = s_clear = 0;
    }
    for (uint32_t pass = 0; pass < 4u; ++pass) {
        if (!(run_passes >> pass & 1u)) continue;
        if (ran) grid_barrier(&q->sort_arrived, ++barriers * ctas, &q->error, 28u);
        const uint32_t src = kSelf ? cur : q->sort_src[pass];
        const uint32_t* __restrict__ ks = src == 0 ? b.in_keys : (src == 1 ? b.b_keys : b.c_keys);
        const uint32_t* __restrict__ vs = src == 0 ? b.in_vals : (src == 1 ? b.b_vals : b.c_vals);
        const bool gather = src == 0;
        const uint32_t kmode = kSelf ? 0u : q->sort_key16;  // 0: the keys, 1: 16-bit age keys, 2: their dense ranks
        const uint32_t shift = 8u * pass;
        const uint32_t epoch = status_tag(q, pass);
        const uint32_t* bucket = q->sort_hist[pass];
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const uint32_t lt_mask = (1u << lane) - 1u;

        for (;;) {
            if (!wave && threadIdx.x == 0) s_tile = atomicAdd(&q->tiles_sort[pass], 1u);
            reinterpret_cast<uint4*>(&s_whist[0][0])[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
            for (int i = 0; i < 2; ++i)
                reinterpret_cast<uint4*>(s_vals)[threadIdx.x + i * kSortThreads] = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
            uint32_t* mask = s_vals + warp * 256;  // lanes by digit; s_vals is used for values only later
            const uint32_t tile = wave ? blockIdx.x : s_tile;
            if (tile >= ntiles) break;

            uint32_t key[kSortItems], val[kSortItems], rank[kSortItems];
            const uint32_t base = tile * kSortTile + (uint32_t)warp * (32u * kSortItems);
#pragma unroll
            for (int j = 0; j < kSortItems; ++j) {
                const uint32_t qi = base + 32u * j + lane;
                key[j] = 0;
                val[j] = 0;
                if (qi < n) {
                    const uint32_t p = gather ? tie_perm(qi, n, reverse) : qi;
                    uint32_t k = __ldcg(ks + p);
                    if (gather && kmode == 1u) k = age_key16(k);
                    if (gather && kmode == 2u) {
                        k = b.age_rank[age_bin(k)];  // ascending rank = descending age: no complement
                    } else if (gather && reverse) {
                        k = ~k;
                    }
                    key[j] = k;
                    val[j] = __ldcg(vs + p);
                }
            }
            if (kSelf && pass == 0u) {
                uint32_t set = 0, clear = 0;
#pragma unroll
                for (int j = 0; j < kSortItems; ++j)
                    if (base + 32u * j + lane < n) {
                        set |= key[j];
                        clear |= ~key[j];
                    }
                set = __reduce_or_sync(0xffffffffu, set);
                clear = __reduce_or_sync(0xffffffffu, clear);
                if (lane == 0) {
                    atomicOr(&s_set, set);
                    atomicOr(&s_clear, clear);
                }
            }
#pragma unroll
            for (int j = 0; j < kSortItems; ++j) {
                const uint32_t qi = base + 32u * j + lane;
                const uint32_t digit = (key[j] >> shift) & 255u;
                // the lanes with the same digit.  Spread digits: each lane sets its
                // bit in the digit's mask, and the first of them clears it again
                // (a match took 82 us on 2^20 random pairs, a ballot per bit 68,
                // this 61).  Ages have few values, which a match finds at once and
                // whose masks the lanes would queue for
                uint32_t peers;
                if (kmode == 0u) {
                    if (qi < n) atomicOr(&mask[digit], 1u << lane);
                    __syncwarp();
                    peers = qi < n ? mask[digit] : 0u;
                } else {
                    peers = __match_any_sync(0xffffffffu, qi < n ? digit : 256u);
                }
                const uint32_t cnt = qi < n ? s_whist[warp][digit] : 0u;
                __syncwarp();
                if (qi < n && lane == __ffs(peers) - 1) {
                    s_whist[warp][digit] = (uint16_t)(cnt + __popc(peers));
                    mask[digit] = 0u;
                }
                __syncwarp();
                rank[j] = cnt + __popc(peers & lt_mask);
            }
            __syncthreads();
            // thread t owns digit t: warp-exclusive offsets and the tile count
            const uint32_t t = threadIdx.x;
            uint32_t run = 0;
            if (t < 256) {
#pragma unroll
                for (int w = 0; w < kSortThreads / 32; ++w) {
                    const uint32_t c = s_whist[w][t];
                    s_whist[w][t] = (uint16_t)run;
                    run += c;
                }
                if (wave) b.counts[tile * 256u + t] = (uint16_t)run;
            }
            uint32_t tile_total;
            const uint32_t start = cta_exclusive_scan<kSortThreads>(run, s_warp_sums, &tile_total);
            if (wave) {
                if (kSelf && pass == 0u && t == 0) {
                    atomicOr(&q->sort_set, s_set);
                    atomicOr(&q->sort_clear, s_clear);
                }
                grid_barrier(&q->sort_arrived, ++barriers * ctas, &q->error, 28u);
                if (kSelf && pass == 0u) {
                    const uint32_t differ = __ldcg(&q->sort_set) & __ldcg(&q->sort_clear);
                    run_passes = 0;
#pragma unroll
                    for (uint32_t d = 0; d < 4u; ++d) run_passes |= ((differ >> (8u * d)) & 255u ? 1u : 0u) << d;
                    if (!run_passes) run_passes = 1u;  // the tie order still applies
                    if (!(run_passes & 1u)) break;
                }
                // rows of counts before this tile's, every sixteenth to a warp (kSelf: and all rows)
                static_assert(kSortThreads == 512 && kSortTile == 4096, "16 warps: 8 KB of counts, 16 KB of masks or sums");
                uint32_t sum[8] = {}, all[8] = {};
                const uint32_t rows = kSelf ? ntiles : tile;
#pragma unroll 4
                for (uint32_t k = (uint32_t)warp; k < rows; k += kSortThreads / 32) {
                    const uint4 v = __ldcg(reinterpret_cast<const uint4*>(b.counts + k * 256u) + lane);
                    const uint32_t c[4] = {v.x, v.y, v.z, v.w};
                    const bool mine = !kSelf || k < tile;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        sum[2 * i] += mine ? c[i] & 0xffffu : 0u;
                        sum[2 * i + 1] += mine ? c[i] >> 16 : 0u;
                        if (kSelf) {
                            all[2 * i] += c[i] & 0xffffu;
                            all[2 * i + 1] += c[i] >> 16;
                        }
                    }
                }
                uint4* part = reinterpret_cast<uint4*>(s_keys + warp * 256 + lane * 8);
                part[0] = make_uint4(sum[0], sum[1], sum[2], sum[3]);
                part[1] = make_uint4(sum[4], sum[5], sum[6], sum[7]);
                if (kSelf) {
                    uint4* part_all = reinterpret_cast<uint4*>(s_vals + warp * 256 + lane * 8);
                    part_all[0] = make_uint4(all[0], all[1], all[2], all[3]);
                    part_all[1] = make_uint4(all[4], all[5], all[6], all[7]);
                }
                __syncthreads();
                uint32_t excl = 0, total = 0;
                if (t < 256) {
#pragma unroll
                    for (int w = 0; w < kSortThreads / 32; ++w) {
                        excl += s_keys[w * 256 + t];
                        if (kSelf) total += s_vals[w * 256 + t];
                    }
                }
                uint32_t place = t < 256 && !kSelf ? bucket[t] : 0u;
                if (kSelf) {
                    uint32_t sum_all;
                    place = cta_exclusive_scan<kSortThreads>(total, s_warp_sums, &sum_all);
                }
                if (t < 256) {
                    s_start[t] = start;
                    s_gbase[t] = place + excl - start;
                }
            } else if (t < 256) {
                s_start[t] = start;
                const uint32_t excl = lookback_exclusive_w8(b.status + t, tile, run, epoch, &q->error, 20u + pass, 256u);
                s_gbase[t] = bucket[t] + excl - start;
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kSortItems; ++j) {
                const uint32_t qi = base + 32u * j + lane;
                if (qi < n) {
                    const uint32_t d = (key[j] >> shift) & 255u;
                    const uint32_t pos = s_start[d] + s_whist[warp][d] + rank[j];
                    s_keys[pos] = key[j];
                    s_vals[pos] = val[j];
                }
            }
            __syncthreads();
            const bool to_out = b.out_keys && (run_passes >> pass) == 1u && src != 0;  // the last pass
            uint32_t* __restrict__ kd = to_out ? b.out_keys : (src == 1 ? b.c_keys : b.b_keys);
            uint32_t* __restrict__ vd = to_out ? b.out_vals : (src == 1 ? b.c_vals : b.b_vals);
            const uint32_t undo = to_out && reverse ? 0xffffffffu : 0u;
            const uint32_t count = min((uint32_t)kSortTile, n - tile * kSortTile);
            for (uint32_t i = threadIdx.x; i < count; i += kSortThreads) {
                const uint32_t k = s_keys[i];
                const uint32_t pos = s_gbase[(k >> shift) & 255u] + i;
                if (pos < n) {  // always true unless a wait timed out
                    kd[pos] = k ^ undo;
                    vd[pos] = s_vals[i];
                }
            }
            __syncthreads();
            if (wave) break;
        }
        if (run_passes >> pass & 1u) {
            ++ran;
            cur = src == 1u ? 2u : 1u;
        }
    }
    if (b.out_keys && ran == 1u) {  // one pass: in b
        grid_barrier(&q->sort_arrived, ++barriers * ctas, &q->error, 28u);
        for (uint32_t i = blockIdx.x * kSortThreads + threadIdx.x; i < n; i += ctas * kSortThreads) {
            const uint32_t k = __ldcg(b.b_keys + i);
            b.out_keys[i] = reverse ? ~k : k;
            b.out_vals[i] = __ldcg(b.b_vals + i);
        }
    }
}

size_t sort_status_words(uint32_t n_max) { return (size_t)div_up(n_max ? n_max : 1, kSortTile) * 256u; }

// CTAs of k_sort resident per SM: the bound of its cooperative grid
static uint32_t sort_per_sm()
{
    static const uint32_t n = [] {
        int a = 0, b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_sort<false>, kSortThreads, 0) != cudaSuccess || a < 1) a = 1;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_sort<true>, kSortThreads, 0) != cudaSuccess || b < 1) b = 1;
        return (uint32_t)std::min(a, b);
    }();
    return n;
}

size_t sort_count_bytes(bcmc_ctx* ctx) { return (size_t)ctx->num_sms * sort_per_sm() * 256u * 2u; }

int sort_grid(bcmc_ctx* ctx, uint32_t n_max)
{
    const uint32_t tiles = div_up(n_max ? n_max : 1, kSortTile);
    const uint32_t resident = (uint32_t)ctx->num_sms * sort_per_sm();
    return (int)(tiles < resident ? tiles : resident);
}

void sort_launch(bcmc_ctx* ctx, QueryState* q, const uint32_t* d_n, uint32_t n_max,
                 const SortBuffers& bufs, int reverse, cudaStream_t s, int plan_ready)
{
    const uint32_t tiles = div_up(n_max ? n_max : 1, kSortTile);
    const bool self = !plan_ready && !d_n && bufs.counts && tiles <= (uint32_t)ctx->num_sms * sort_per_sm();
    if (!plan_ready && !self) {
        const int hist_grid = (int)min(div_up(n_max ? n_max : 1, (uint32_t)kHistThreads * 8u), (uint32_t)ctx->num_sms);
        k_sort_hist<<<hist_grid, kHistThreads, 0, s>>>(q, d_n, n_max, bufs.in_keys, reverse);
        count_launches(1);
    }
    // cooperative: the grid barriers between digit passes need every CTA resident
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(sort_grid(ctx, n_max));
    cfg.blockDim = dim3(kSortThreads);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeCooperative;
    attr.val.cooperative = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (self) BCMC_CUDA(cudaLaunchKernelEx(&cfg, k_sort<true>, q, d_n, n_max, bufs, reverse));
    else BCMC_CUDA(cudaLaunchKernelEx(&cfg, k_sort<false>, q, d_n, n_max, bufs, reverse));
    count_launches(1);
}

}  // namespace bcmc
