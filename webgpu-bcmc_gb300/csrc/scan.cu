// scan.cu -- single-pass exclusive scan and stream compaction.
//
// Replaces ExclusiveScanner.scan (js/exclusive_scan.js:178-295), which runs a
// three-kernel Blelloch scan (prefix_sum.comp, block_prefix_sum.comp,
// add_block_sums.comp) per 512^2-element chunk with a host-side carry and a
// mapAsync readback of the total, and StreamCompact.compactActiveIDs
// (js/stream_compact.js:56-165, stream_compact.comp:26-32), one thread per
// workgroup.  Here a scan is one launch: a range of 8192-element tiles per CTA,
// scanned with warp shuffles, the ranges joined by their published sums.  uint32 sums wrap mod 2^32 as
// in the reference.
#include "bcmc_impl.h"

namespace bcmc {

__global__ void k_prim_begin(QueryState* q)
{
    // new epoch for the look-back status words; clear counters and the sort plan
    const int t = threadIdx.x;
    if (t == 0) {
        q->epoch += 1;
        q->tiles_active = q->tiles_slots = q->tiles_sort_hist = 0;
        for (int i = 0; i < 4; ++i) q->tiles_sort[i] = 0;
        q->sort_arrived = 0;
        q->error = 0;
        q->num_with_verts = q->num_verts = 0;
        q->grow_needed = 0;
        q->vert_overflow = 0;
        for (int i = 0; i < 4; ++i) q->sort_run[i] = q->sort_src[i] = 0;  // the plan of zero keys
        q->sort_first = 4;
        q->sort_final = 1;
        q->sort_key16 = q->sort_wide = 0;
    }
    for (int i = t; i < 1536; i += blockDim.x) (&q->sort_hist[0][0])[i] = 0;  // and sort_hist16
}

void prim_begin(QueryState* q, cudaStream_t s)
{
    k_prim_begin<<<1, 256, 0, s>>>(q);
    count_launches(1);
    BCMC_CUDA(cudaGetLastError());
}

// A CTA owns one contiguous range of tiles: it adds them up, publishes the sum,
// adds up the sums of the CTAs before it in one round trip (their ranks are
// claimed in order, so all of them run), and scans its tiles again from there --
// out of its registers when the range is one tile, which it is up to 5 M
// elements, else out of L2.  Tiles claimed one by one with a look-back each took
// 25 us on 4 M elements, most of it in the chain from tile to tile.
// Loads and stores are 16 bytes where the arrays allow it (kWide).
constexpr int kRangeThreads = 512;
constexpr int kRangeItems = 16;  // consecutive elements per thread
constexpr uint32_t kRangeTile = kRangeThreads * kRangeItems;
constexpr int kRangePerSm = 3;
static_assert(kRangeTile % kScanTile == 0, "the status words are sized by kScanTile");

template <bool kWide>
__device__ __forceinline__ void load_items(const uint32_t* in, uint64_t first, uint32_t n, uint32_t v[kRangeItems])
{
    if (kWide && first + kRangeItems <= n) {
#pragma unroll
        for (int j = 0; j < kRangeItems / 4; ++j) {
            const uint4 x = reinterpret_cast<const uint4*>(in + first)[j];
            v[4 * j] = x.x;
            v[4 * j + 1] = x.y;
            v[4 * j + 2] = x.z;
            v[4 * j + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int j = 0; j < kRangeItems; ++j) v[j] = first + j < n ? in[first + j] : 0u;
    }
}

// kSelect: the input is flags, the output the indices of the nonzero ones;
// otherwise the output is the exclusive scan.
template <bool kSelect, bool kWide>
__global__ void __launch_bounds__(kRangeThreads, kRangePerSm) k_scan(QueryState* q, const uint32_t* in, uint32_t* out,
                                                                     uint32_t n, uint32_t per_cta, ScanTotals tot,
                                                                     uint64_t* status)
{
    __shared__ uint32_t s_warp[kRangeThreads / 32 + 1];
    __shared__ uint32_t s_rank, s_sum, s_prefix;
    const uint32_t t = threadIdx.x;
    if (t == 0) {
        s_rank = atomicAdd(&q->tiles_active, 1u);
        s_sum = s_prefix = 0;
    }
    __syncthreads();
    const uint32_t rank = s_rank, ntiles = div_up(n, kRangeTile);
    const uint32_t first = rank * per_cta, end = min(ntiles, first + per_cta);
    uint32_t v[kRangeItems], sum = 0, all = 0;
    for (uint32_t tile = first; tile < end; ++tile) {
        load_items<kWide>(in, (uint64_t)tile * kRangeTile + t * kRangeItems, n, v);
        sum = 0;
#pragma unroll
        for (int j = 0; j < kRangeItems; ++j) sum += kSelect ? (v[j] != 0u ? 1u : 0u) : v[j];
        all += sum;
    }
    all = __reduce_add_sync(0xffffffffu, all);
    if ((t & 31u) == 0u && all) atomicAdd(&s_sum, all);
    __syncthreads();
    const bool late = cta_prefix_sum<kRangeThreads>(status, rank, s_sum, q->epoch, &q->error, kSelect ? 2u : 1u,
                                                    &s_prefix, lb_dropped(q, rank));
    if (late && tot.host) tot.host[1] = 1u;
    __syncthreads();
    uint32_t run = s_prefix;
    if (end == ntiles && t == 0) {
        const uint32_t total = run + s_sum;
        if (tot.device) *tot.device = total;
        if (tot.after) *tot.after = total;
        if (tot.host) tot.host[0] = total;
    }
    for (uint32_t tile = first; tile < end; ++tile) {
        const uint64_t at = (uint64_t)tile * kRangeTile + t * kRangeItems;
        if (end - first > 1u) {
            load_items<kWide>(in, at, n, v);
            sum = 0;
#pragma unroll
            for (int j = 0; j < kRangeItems; ++j) sum += kSelect ? (v[j] != 0u ? 1u : 0u) : v[j];
        }
        uint32_t total;
        uint32_t pos = run + cta_exclusive_scan<kRangeThreads>(sum, s_warp, &total);
        run += total;
        if (kSelect) {
#pragma unroll
            for (int j = 0; j < kRangeItems; ++j)
                if (v[j] != 0u) {
                    if (pos < n) out[pos] = (uint32_t)at + j;  // pos < n unless a wait timed out
                    ++pos;
                }
        } else if (kWide && at + kRangeItems <= n) {
#pragma unroll
            for (int j = 0; j < kRangeItems / 4; ++j) {
                uint4 x;
                x.x = pos;
                x.y = x.x + v[4 * j];
                x.z = x.y + v[4 * j + 1];
                x.w = x.z + v[4 * j + 2];
                pos = x.w + v[4 * j + 3];
                reinterpret_cast<uint4*>(out + at)[j] = x;
            }
        } else {
#pragma unroll
            for (int j = 0; j < kRangeItems; ++j)
                if (at + j < n) {
                    out[at + j] = pos;
                    pos += v[j];
                }
        }
    }
}

// Four elements a thread where the arrays allow 16-byte loads (16 -> 7 us on 4 M).
__global__ void __launch_bounds__(256) k_compact(uint32_t n, const uint32_t* __restrict__ flags,
                                                 const uint32_t* __restrict__ offsets, uint32_t* out, bool wide)
{
    const uint32_t step = gridDim.x * blockDim.x, t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t fours = wide ? n / 4u : 0u;
    for (uint32_t i = t; i < fours; i += step) {
        const uint4 f = __ldg(reinterpret_cast<const uint4*>(flags) + i);
        if (!(f.x | f.y | f.z | f.w)) continue;
        const uint4 o = __ldg(reinterpret_cast<const uint4*>(offsets) + i);
        if (f.x) out[o.x] = 4u * i;
        if (f.y) out[o.y] = 4u * i + 1u;
        if (f.z) out[o.z] = 4u * i + 2u;
        if (f.w) out[o.w] = 4u * i + 3u;
    }
    for (uint32_t i = 4u * fours + t; i < n; i += step)
        if (flags[i] != 0u) out[offsets[i]] = i;
}

static bool aligned16(const void* a, const void* b)
{
    return (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) % 16u == 0;
}

template <bool kSelect>
static cudaError_t launch_ranges(int num_sms, QueryState* q, const uint32_t* in, uint32_t* out, uint32_t n,
                                 const ScanTotals& tot, uint64_t* status, cudaStream_t s)
{
    const uint32_t tiles = div_up(n, kRangeTile), most = (uint32_t)num_sms * kRangePerSm;
    const uint32_t per_cta = div_up(tiles, most), grid = div_up(tiles, per_cta);
    // (a select's output is written element by element: its alignment is not asked for)
    if (aligned16(in, kSelect ? in : out)) k_scan<kSelect, true><<<grid, kRangeThreads, 0, s>>>(q, in, out, n, per_cta, tot, status);
    else k_scan<kSelect, false><<<grid, kRangeThreads, 0, s>>>(q, in, out, n, per_cta, tot, status);
    count_launches(1);
    return cudaGetLastError();
}

void scan_launch(bcmc_ctx* ctx, QueryState* q, const uint32_t* in, uint32_t* out, uint32_t n,
                 const ScanTotals& tot, uint64_t* status, cudaStream_t s)
{
    BCMC_CUDA(launch_ranges<false>(ctx->num_sms, q, in, out, n, tot, status, s));
}

cudaError_t scan_launch_sms(int num_sms, QueryState* q, const uint32_t* in, uint32_t* out, uint32_t n,
                            uint32_t* d_total, uint64_t* status, cudaStream_t s)
{
    return launch_ranges<false>(num_sms, q, in, out, n, ScanTotals{d_total}, status, s);
}

void select_launch(bcmc_ctx* ctx, QueryState* q, const uint32_t* flags, uint32_t* out, uint32_t n,
                   uint32_t* d_count, uint64_t* status, cudaStream_t s)
{
    BCMC_CUDA(launch_ranges<true>(ctx->num_sms, q, flags, out, n, ScanTotals{d_count}, status, s));
}

void compact_launch(bcmc_ctx* ctx, uint32_t n, const uint32_t* flags, const uint32_t* offsets, uint32_t* out,
                    cudaStream_t s)
{
    if (n == 0) return;
    const int grid = (int)min(div_up(n, 1024u), (uint32_t)ctx->num_sms * 8u);
    k_compact<<<grid, 256, 0, s>>>(n, flags, offsets, out, aligned16(flags, offsets));
    count_launches(1);
    BCMC_CUDA(cudaGetLastError());
}

}  // namespace bcmc
