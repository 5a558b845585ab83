// mc_common.cuh -- the marching-cubes work of one warp, shared by the
// per-query MC kernel (pipeline.cu) and the batched one (engine.cu): the case
// tables of mc_triangle.cuh in device memory, a block's corner mask, cases and
// triangle counts, and the emit of a few blocks' vertices.
//
// A warp works alone, on up to four blocks at a time, without CTA barriers:
//   lookup  lane 8j + o reads what neighbour o (x|y<<1|z<<2) of block j is:
//           active, and in which cache slot;
//   voxels  a block's 5^3 grid is four loads per lane (voxel lane + 32r), and
//           four ballots of `value <= iso` are its 125-bit corner mask in
//           registers; a ghost voxel that the grid does not take is read as
//           some voxel of the block itself, which changes no cell in the grid;
//   cases   a lane takes the cells lane and lane + 32: a cell's eight corners
//           are bits 0, 1, 5, 6, 25, 26, 30 and 31 of the 32-bit window of the
//           mask at its corner 0, so one funnel shift yields them all; a block
//           whose mask is all zeros or all ones has no cases to look up.
// Instructions bound these kernels, not bytes: half a warp per block with its
// rows tested through shared memory, and CTA-wide scans, took 240 warp
// instructions to count a block; this takes 60 to 90.
// The tables are static: each translation unit has its own copy.
#pragma once

#include "bcmc_internal.cuh"
#include "mc_triangle.cuh"

namespace bcmc {

constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kMcBlocks = 4;  // blocks a warp works on at a time

// copied into shared memory by every CTA (16-byte asynchronous copies)
struct McTables {
    mc_detail::TriRows rows;
    mc_detail::EdgeBases edges;
};
static_assert(sizeof(McTables) % 16 == 0, "copied in 16-byte pieces");
static __device__ const __align__(16) McTables c_mc = {mc_detail::make_tri_rows(), mc_detail::make_edge_bases()};
// for the few vertices that take the exact expression: read where it lies
static __device__ const __align__(16) mc_detail::CornerPack c_corner_pack = mc_detail::make_corner_pack();

// shared memory of one warp's emit
struct McWarpMem {
    float vol[kMcBlocks][128];      // the blocks' 5^3 grids
    uint32_t list[kMcBlocks * 64];  // cells with triangles, in order: cell | case << 8 | first triangle << 16
    uint2 out[128];                 // vertices on their way to a coalesced store
    uint8_t flag[kMcBlocks * 320];  // 1 where a triangle is its cell's first; zero between emits
};
static_assert(sizeof(McWarpMem) % 16 == 0, "16-byte aligned in an array");

template <int kThreads>
struct McShared {
    McTables tab;
    McWarpMem warp[kThreads / 32];
};

// Starts the copy of the tables (mc_tables_wait before their first use, then a
// barrier) and clears the warp's flags.  The counts are stored at once.
template <int kThreads>
__device__ __forceinline__ void mc_shared_begin(McShared<kThreads>& s)
{
    constexpr uint32_t n = sizeof(McTables) / 16;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&s.tab);
    const char* src = reinterpret_cast<const char*>(&c_mc);
    for (uint32_t i = threadIdx.x; i < n; i += kThreads)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * i), "l"(src + 16u * i) : "memory");
    asm volatile("cp.async.commit_group;" ::: "memory");
    uint32_t* f = reinterpret_cast<uint32_t*>(s.warp[threadIdx.x >> 5].flag);
    for (uint32_t i = threadIdx.x & 31u; i < sizeof(McWarpMem::flag) / 4; i += 32u) f[i] = 0u;
}
__device__ __forceinline__ void mc_tables_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// A lane's part of every block: where its four grid voxels come from
// (neighbour o, voxel within that block), and its two cells.
struct McLane {
    const float* src[4];  // the voxel in slot 0 of the cache
    uint32_t nb;          // neighbour of voxel r in byte r
    uint32_t g;           // corner 0 of cell `lane` in the grid; cell lane + 32's is at g + 50
    uint32_t need;        // axes on which cell `lane` needs the ghost layer, and from bit 3 cell lane + 32
};
__device__ __forceinline__ McLane mc_lane(const float* cache)
{
    const uint32_t lane = threadIdx.x & 31u;
    McLane m;
    m.nb = 0;
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) {
        uint32_t v = lane + 32u * r;
        if (v >= 125u) v = 0u;
        const uint32_t x = v % 5u, y = (v / 5u) % 5u, z = v / 25u;
        m.nb |= ((x >> 2) | ((y >> 2) << 1) | ((z >> 2) << 2)) << (8u * r);
        m.src[r] = cache + ((x & 3u) + 4u * ((y & 3u) + 4u * (z & 3u)));
    }
    const uint32_t x = lane & 3u, y = (lane >> 2) & 3u, z = lane >> 4;
    m.g = x + 5u * (y + 5u * z);
    const uint32_t xy = (x == 3u ? 1u : 0u) | (y == 3u ? 2u : 0u);
    m.need = xy | ((xy | (z == 1u ? 4u : 0u)) << 3);
    return m;
}

// compute_vertex_values.comp:96-156: the axes on which a block's grid takes the
// ghost layer of its +x/+y/+z neighbours.  `exist`: axes on which there is a
// neighbour; bit o of `act`: neighbour o (x|y<<1|z<<2) exists and is active.
__device__ __forceinline__ uint32_t mc_ghost_axes(uint32_t exist, uint32_t act)
{
    uint32_t h = exist;
    if (h == 7u && !(act >> 7 & 1u)) h = 0u;
    if ((h & 3u) == 3u && !(act >> 3 & 1u)) h &= ~3u;
    if ((h & 5u) == 5u && !(act >> 5 & 1u)) h &= ~5u;
    if ((h & 6u) == 6u && !(act >> 6 & 1u)) h &= ~6u;
    if ((h & 1u) && !(act >> 1 & 1u)) h &= ~1u;
    if ((h & 2u) && !(act >> 2 & 1u)) h &= ~2u;
    if ((h & 4u) && !(act >> 4 & 1u)) h &= ~4u;
    return h;
}

// The lane's neighbour of its block: lane 8j + o, block j, neighbour o; a lane
// of no block passes valid = false.  `active(nid)` says whether a block is
// active.  On return `slot` is where the lane's neighbour is cached (the
// block's own slot if its grid does not reach into that neighbour) and `has`
// the axes of the block's ghost layer.  A needed block that no slot holds
// cannot happen with a consistent cache: it is reported (`self_err` for the
// block itself, `nb_err` for a neighbour), and slot 0 is read.
template <typename Active>
__device__ __forceinline__ void mc_lookup(bool valid, uint32_t id, const BlockGrid& grid, const int32_t* item_slots,
                                          uint32_t slots, Active active, uint32_t* error, uint32_t self_err,
                                          uint32_t nb_err, uint32_t& slot, uint32_t& has)
{
    const uint32_t lane = threadIdx.x & 31u, o = lane & 7u;
    uint32_t exist = 0, act = 0;
    slot = 0xffffffffu;
    if (valid) {
        const uint3 c = block_coords(id, grid), nb = grid.nb;
        exist = (c.x + 1u < nb.x ? 1u : 0u) | (c.y + 1u < nb.y ? 2u : 0u) | (c.z + 1u < nb.z ? 4u : 0u);
        if ((o & ~exist) == 0u) {
            const uint32_t nid = id + (o & 1u) + nb.x * (((o >> 1) & 1u) + nb.y * (o >> 2));
            slot = (uint32_t)__ldg(item_slots + nid);
            act = o == 0u || active(nid) ? 1u : 0u;
        }
    }
    const uint32_t bits = __ballot_sync(kFull, act != 0u);
    has = mc_ghost_axes(exist, (bits >> (lane & 24u)) & 0xffu);
    const uint32_t self = __shfl_sync(kFull, slot, lane & 24u);
    if ((o & ~has) != 0u) slot = self;
    if (slot >= slots) {
        if (valid) atomicCAS(error, 0u, o == 0u ? self_err : nb_err);
        slot = 0u;
    }
}

// The grid voxels of blocks 0 .. n - 1, all loads in flight together.
__device__ __forceinline__ void mc_voxels(const McLane& m, uint32_t slot, uint32_t n, float f[kMcBlocks][4])
{
#pragma unroll
    for (uint32_t j = 0; j < kMcBlocks; ++j)
        if (j < n) {
#pragma unroll
            for (uint32_t r = 0; r < 4; ++r) {
                const uint32_t s = __shfl_sync(kFull, slot, 8u * j + ((m.nb >> (8u * r)) & 7u));
                f[j][r] = __ldg(m.src[r] + (uint64_t)s * 64u);
            }
        }
}

// A cell's case from the corner mask's window at its corner 0.
__device__ __forceinline__ uint32_t mc_case(uint32_t w)
{
    return (w & 0x03u) | ((w >> 3) & 0x0cu) | ((w >> 21) & 0x30u) | ((w >> 24) & 0xc0u);
}

// The cases of the lane's two cells (compute_block_has_vertices.comp:28-51);
// false when no cell of the block can have one (uniform over the warp).
__device__ __forceinline__ bool mc_cases(const McLane& m, const float f[4], float iso, uint32_t has, uint32_t& c0,
                                         uint32_t& c1)
{
    const uint32_t m0 = __ballot_sync(kFull, f[0] <= iso), m1 = __ballot_sync(kFull, f[1] <= iso),
                   m2 = __ballot_sync(kFull, f[2] <= iso), m3 = __ballot_sync(kFull, f[3] <= iso);
    c0 = c1 = 0u;
    if ((m0 | m1 | m2 | m3) == 0u || (m0 & m1 & m2 & m3) == 0xffffffffu) return false;
    const bool lo = m.g < 32u, lo1 = m.g < 14u;  // g + 50 < 64
    const uint32_t w0 = __funnelshift_r(lo ? m0 : m1, lo ? m1 : m2, m.g & 31u);
    const uint32_t w1 = __funnelshift_r(lo1 ? m1 : m2, lo1 ? m2 : m3, (m.g + 50u) & 31u);
    if ((m.need & 7u & ~has) == 0u) c0 = mc_case(w0);
    if (((m.need >> 3) & ~has) == 0u) c1 = mc_case(w1);
    return true;
}

__device__ __forceinline__ uint32_t mc_tri_count(const uint32_t* ntri, uint32_t c)
{
    return (ntri[c >> 3] >> (4u * (c & 7u))) & 15u;
}

// Where an emit's vertices go.  Device memory: straight from the warp's staging
// in coalesced stores.  Page-locked host memory (kHost): held back until a
// 256-byte-aligned window of 32 is full -- stores over the host link run about
// 20 % faster so -- with the rest carried on to the next emit, whose vertices
// follow; `finish` stores what is left.
template <bool kHost>
struct McSink {
    uint2* at;          // where the next vertex goes
    uint32_t held = 0;  // vertices waiting in the staging buffer (kHost)

    // n new vertices lie at stage[held ..]
    __device__ __forceinline__ void put(uint2* stage, uint32_t n)
    {
        const uint32_t lane = threadIdx.x & 31u;
        __syncwarp();
        if constexpr (!kHost) {
#pragma unroll
            for (uint32_t k = 0; k < 3; ++k)
                if (lane + 32u * k < n) at[lane + 32u * k] = stage[lane + 32u * k];
            at += n;
            __syncwarp();
        } else {
            held += n;
            flush(stage, false);
        }
    }
    __device__ __forceinline__ void flush(uint2* stage, bool all)
    {
        const uint32_t lane = threadIdx.x & 31u;
        uint32_t done = 0;
        while (done < held) {
            const uint32_t room = 32u - ((uint32_t)(reinterpret_cast<uintptr_t>(at) >> 3) & 31u);
            const uint32_t n = min(room, held - done);
            if (n < room && !all) break;
            if (lane < n) at[lane] = stage[done + lane];
            at += n;
            done += n;
        }
        held -= done;  // fewer than 32 are left
        if (done) {
            const uint2 v = lane < held ? stage[done + lane] : make_uint2(0u, 0u);
            __syncwarp();
            if (lane < held) stage[lane] = v;
        }
        __syncwarp();
    }
    __device__ __forceinline__ void finish(uint2* stage)
    {
        if constexpr (kHost) flush(stage, true);
    }
};

// The vertices of blocks 0 .. n - 1 (their lookups in `slot` and `has`, ids and
// isovalues in lane 8j) to the sink, in block, cell and table order.  A lane
// takes one triangle: the triangle's cell is the last with a start flag at or
// before it, counted by ballot; the three vertices share the cell's lookup and
// its row of the case table, and leave through the staging buffer so that the
// stores are contiguous.
template <bool kHost>
__device__ __forceinline__ void mc_emit(const McLane& m, const McTables& tab, McWarpMem& s, uint32_t n, uint32_t id,
                                        uint32_t slot, uint32_t has, float iso, McSink<kHost>& sink)
{
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    uint32_t tris = 0, cells = 0;
    {
        float f[kMcBlocks][4];
        mc_voxels(m, slot, n, f);
#pragma unroll
        for (uint32_t j = 0; j < kMcBlocks; ++j)
            if (j < n) {
#pragma unroll
                for (uint32_t r = 0; r < 4; ++r) s.vol[j][lane + 32u * r] = f[j][r];
                uint32_t c0, c1;
                if (!mc_cases(m, f[j], __shfl_sync(kFull, iso, 8u * j), __shfl_sync(kFull, has, 8u * j), c0, c1))
                    continue;
                const uint32_t t0 = mc_tri_count(tab.rows.ntri, c0), t1 = mc_tri_count(tab.rows.ntri, c1);
                const uint32_t inc = warp_inclusive_scan(t0 | (t1 << 16));
                const uint32_t tot = __shfl_sync(kFull, inc, 31);
                const uint32_t e0 = __ballot_sync(kFull, t0 != 0u), e1 = __ballot_sync(kFull, t1 != 0u);
                if (t0) {
                    const uint32_t first = tris + (inc & 0xffffu) - t0;
                    s.list[cells + __popc(e0 & below)] = (64u * j + lane) | (c0 << 8) | (first << 16);
                    s.flag[first] = 1;
                }
                if (t1) {
                    const uint32_t first = tris + (tot & 0xffffu) + (inc >> 16) - t1;
                    s.list[cells + __popc(e0) + __popc(e1 & below)] = (64u * j + 32u + lane) | (c1 << 8) | (first << 16);
                    s.flag[first] = 1;
                }
                tris += (tot & 0xffffu) + (tot >> 16);
                cells += __popc(e0) + __popc(e1);
            }
    }
    __syncwarp();
    uint32_t before = 0;  // cells that start before the window of 32 triangles
    for (uint32_t w = 0; w < tris; w += 32u) {
        const uint32_t starts = __ballot_sync(kFull, s.flag[w + lane] != 0);
        s.flag[w + lane] = 0;
        const uint32_t e = s.list[before + __popc(starts & (below | (1u << lane))) - 1u];
        before += __popc(starts);
        const uint32_t cell = e & 63u, j = (e >> 6) & 3u;
        const uint32_t bid = __shfl_sync(kFull, id, 8u * j);
        const float biso = __shfl_sync(kFull, iso, 8u * j);
        const uint32_t left = tris - w;
        if (lane < left) {
            const uint4 te = *reinterpret_cast<const uint4*>(tab.rows.t[(e >> 8) & 255u][w + lane - (e >> 16)]);
            const uint32_t g = cell + ((cell >> 2) & 3u) + 9u * (cell >> 4);  // the cell's corner 0 in the grid
            const float* vol = s.vol[j] + g;
            const mc_detail::EdgeBase* eb = &tab.edges.b[0][g];
            bool again = false;
            uint32_t p0 = mc_vertex_fast(te.x, vol, eb, biso, &again), p1 = mc_vertex_fast(te.y, vol, eb, biso, &again),
                     p2 = mc_vertex_fast(te.z, vol, eb, biso, &again);
            if (again) {
                const uint32_t* cp = &c_corner_pack.p[0][0];
                p0 = mc_vertex(mc_word_entry(te.x), cell, s.vol[j], cp, biso);
                p1 = mc_vertex(mc_word_entry(te.y), cell, s.vol[j], cp, biso);
                p2 = mc_vertex(mc_word_entry(te.z), cell, s.vol[j], cp, biso);
            }
            uint2* o = s.out + (kHost ? sink.held : 0u) + 3u * lane;
            o[0] = make_uint2(p0, bid);
            o[1] = make_uint2(p1, bid);
            o[2] = make_uint2(p2, bid);
        }
        sink.put(s.out, 3u * min(left, 32u));
    }
}

// The sum over the CTAs before `rank` of the two counts each published in its
// status words (aggregates of this epoch), to *sum_a and *sum_b in shared
// memory, zero before.  Every thread takes a share of the predecessors, so all
// are read in one round trip; the wait is for the slowest of them.
template <int kThreads>
__device__ __forceinline__ void cta_prefix_sums(uint64_t* status_a, uint64_t* status_b, uint32_t rank, uint32_t a,
                                                uint32_t b, uint32_t epoch, uint32_t* err, uint32_t site_a,
                                                uint32_t site_b, uint32_t* sum_a, uint32_t* sum_b)
{
    if (threadIdx.x == 0) {
        lb_store(status_a + rank, lb_pack(epoch, kFlagAggregate, a));
        lb_store(status_b + rank, lb_pack(epoch, kFlagAggregate, b));
    }
    uint32_t sa = 0, sb = 0;
    for (uint32_t p = threadIdx.x; p < rank; p += kThreads) {
        uint64_t va, vb;
        uint32_t spins = 0;
        for (;;) {
            va = lb_load(status_a + p);
            vb = lb_load(status_b + p);
            const bool ra = (uint32_t)(va >> 34) == epoch, rb = (uint32_t)(vb >> 34) == epoch;
            if (ra && rb) break;
            if (++spins > kSpinLimit) {
                atomicCAS(err, 0u, ra ? site_b : site_a);
                break;
            }
            if (spins > 8) __nanosleep(100);
        }
        sa += (uint32_t)va;
        sb += (uint32_t)vb;
    }
    sa = __reduce_add_sync(kFull, sa);
    sb = __reduce_add_sync(kFull, sb);
    if ((threadIdx.x & 31u) == 0u) {
        if (sa) atomicAdd(sum_a, sa);
        if (sb) atomicAdd(sum_b, sb);
    }
}

}  // namespace bcmc
