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
        q->sort_arrived = q->sort_set = q->sort_clear = 0;
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
// out of its registers when the range is one tile, which it is up to 3.7 M
// elements, else out of L2 (tiles of up to 12288, one to a CTA up to 5.6 M, were no
// faster on 4 M).  Tiles claimed one by one with a look-back each took
// 25 us on 4 M elements, most of it in the chain from tile to tile.
// A warp has 512 consecutive elements of a tile, in four groups of four to a lane,
// so that its loads and stores are contiguous, 16 bytes a lane where the arrays
// allow it (kWide): sixteen elements to a thread take one scan instead of four,
// but 16-byte pieces of 64 (18.8 -> 15.1 us on 4 M elements).
constexpr int kRangeThreads = 512;
constexpr uint32_t kRangeGroups = 4;
constexpr uint32_t kRangeTile = kRangeThreads * 4u * kRangeGroups;
constexpr int kRangePerSm = 3;
static_assert(kRangeTile % kScanTile == 0, "the status words are sized by kScanTile");

// The lane's elements of the warp's 512 from `first` on.
template <bool kWide>
__device__ __forceinline__ void load_items(const uint32_t* in, uint64_t first, uint32_t n, uint4 v[kRangeGroups])
{
#pragma unroll
    for (uint32_t j = 0; j < kRangeGroups; ++j) {
        const uint64_t i = first + 128u * j + 4u * (threadIdx.x & 31u);
        if (kWide && i + 4u <= n) {
            v[j] = *reinterpret_cast<const uint4*>(in + i);
        } else {
            v[j].x = i < n ? in[i] : 0u;
            v[j].y = i + 1u < n ? in[i + 1u] : 0u;
            v[j].z = i + 2u < n ? in[i + 2u] : 0u;
            v[j].w = i + 3u < n ? in[i + 3u] : 0u;
        }
    }
}

// What the scan adds up: the elements, or (kSelect) how many are not 0.
template <bool kSelect>
__device__ __forceinline__ uint4 addends(uint4 v)
{
    if (kSelect) return make_uint4(v.x ? 1u : 0u, v.y ? 1u : 0u, v.z ? 1u : 0u, v.w ? 1u : 0u);
    return v;
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
    const uint32_t lane = t & 31u, warp = t >> 5;
    uint4 v[kRangeGroups];
    uint32_t all = 0;
    for (uint32_t tile = first; tile < end; ++tile) {
        load_items<kWide>(in, (uint64_t)tile * kRangeTile + 128u * kRangeGroups * warp, n, v);
#pragma unroll
        for (uint32_t j = 0; j < kRangeGroups; ++j) {
            const uint4 x = addends<kSelect>(v[j]);
            all += x.x + x.y + x.z + x.w;
        }
    }
    all = __reduce_add_sync(0xffffffffu, all);
    if ((t & 31u) == 0u && all) atomicAdd(&s_sum, all);
    __syncthreads();
    const bool late = cta_prefix_sums<kRangeThreads>({{status, s_sum, kSelect ? 2u : 1u, &s_prefix}}, rank, status_tag(q),
                                                     &q->error, lb_dropped(q, rank));
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
        const uint64_t base = (uint64_t)tile * kRangeTile + 128u * kRangeGroups * warp;
        if (end - first > 1u) load_items<kWide>(in, base, n, v);
        uint32_t before[kRangeGroups], sum = 0;  // of the warp's elements
#pragma unroll
        for (uint32_t j = 0; j < kRangeGroups; ++j) {
            const uint4 x = addends<kSelect>(v[j]);
            const uint32_t mine = x.x + x.y + x.z + x.w, inc = warp_inclusive_scan(mine);
            before[j] = sum + inc - mine;
            sum += __shfl_sync(0xffffffffu, inc, 31);
        }
        uint32_t total;
        const uint32_t warps = cta_exclusive_scan<kRangeThreads>(lane == 0 ? sum : 0u, s_warp, &total);
        const uint32_t start = run + __shfl_sync(0xffffffffu, warps, 0);
        run += total;
#pragma unroll
        for (uint32_t j = 0; j < kRangeGroups; ++j) {
            const uint64_t i = base + 128u * j + 4u * lane;
            const uint4 x = addends<kSelect>(v[j]);
            uint4 p;
            p.x = start + before[j];
            p.y = p.x + x.x;
            p.z = p.y + x.y;
            p.w = p.z + x.z;
            if (kSelect) {  // positions are below n unless a wait timed out
                if (x.x && p.x < n) out[p.x] = (uint32_t)i;
                if (x.y && p.y < n) out[p.y] = (uint32_t)i + 1u;
                if (x.z && p.z < n) out[p.z] = (uint32_t)i + 2u;
                if (x.w && p.w < n) out[p.w] = (uint32_t)i + 3u;
            } else if (kWide && i + 4u <= n) {
                *reinterpret_cast<uint4*>(out + i) = p;
            } else {
                if (i < n) out[i] = p.x;
                if (i + 1u < n) out[i + 1u] = p.y;
                if (i + 2u < n) out[i + 2u] = p.z;
                if (i + 3u < n) out[i + 3u] = p.w;
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
    // A select's ids go to places at or before their flags.  Where these are the
    // flags' own words, a CTA must not read a tile again after others may have
    // written: one tile to a CTA, which then keeps it in registers.
    const bool overlap = kSelect && in < out + n && out < in + n;
    const uint32_t per_cta = overlap ? 1u : div_up(tiles, most), grid = div_up(tiles, per_cta);
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
    // a thread's four elements are one load each of flags and offsets, or (bases that
    // are not on 16 bytes) four in turn, which more CTAs take side by side: 4.2 -> 3.3
    // us up to 300,000 elements
    const bool wide = aligned16(flags, offsets);
    const int grid = (int)(wide ? min(div_up(n, 1024u), (uint32_t)ctx->num_sms * 8u)
                                : min(div_up(n, 256u), (uint32_t)ctx->num_sms * 16u));
    k_compact<<<grid, 256, 0, s>>>(n, flags, offsets, out, wide);
    count_launches(1);
    BCMC_CUDA(cudaGetLastError());
}

}  // namespace bcmc
