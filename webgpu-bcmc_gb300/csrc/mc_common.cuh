// mc_common.cuh -- the marching-cubes work of one warp, shared by the
// per-query MC kernel (pipeline.cu) and the batched one (engine.cu): the case
// tables of mc_triangle.cuh in device memory, a block's corner mask, cases and
// triangle counts, and the emit of a few blocks' vertices.
//
// A warp works alone, on up to four blocks at a time, without CTA barriers:
//   lookup  lane 8j + o reads what neighbour o (x|y<<1|z<<2) of block j is:
//           active, and in which cache slot; begun one round ahead, so that its
//           loads are in flight while the round before is worked on;
//   voxels  a block's 5^3 grid is four loads per lane (voxel lane + 32r), and
//           four ballots of `value <= iso` are its 125-bit corner mask in
//           registers; a ghost voxel that the grid does not take is read as
//           some voxel of the block itself, which changes no cell in the grid;
//   cases   a lane takes the cells lane and lane + 32: a cell's eight corners
//           are in the 32-bit window of the mask at its corner 0, so a funnel
//           shift and a product give its case; a block whose mask is all zeros
//           or all ones has no cases to look up.
// Instructions bound these kernels, not bytes: half a warp per block with its
// rows tested through shared memory, and CTA-wide scans, took 240 warp
// instructions to count a block.
// The tables are static: each translation unit has its own copy.
#pragma once

#include "bcmc_internal.cuh"
#include "mc_triangle.cuh"

namespace bcmc {

constexpr uint32_t kFull = 0xffffffffu;
constexpr uint32_t kMcBlocks = 4;  // blocks a warp works on at a time

// copied into shared memory by every CTA, the first part for the count pass
struct McTables {
    mc_detail::TriCounts count;
    mc_detail::GhostAxes ghost;
    mc_detail::TriRows rows;
    mc_detail::CellRecs cells;
};
constexpr uint32_t kMcFirstTables = (sizeof(mc_detail::TriCounts) + sizeof(mc_detail::GhostAxes)) / 16;
static_assert(sizeof(McTables) % 16 == 0 && offsetof(McTables, rows) == 16 * kMcFirstTables, "16-byte pieces");
static __device__ const __align__(16) McTables c_mc = {mc_detail::make_tri_counts(), mc_detail::make_ghost_axes(),
                                                       mc_detail::make_tri_rows(), mc_detail::make_cell_recs()};
// for the few vertices that take the exact expression: read where it lies
static __device__ const __align__(16) mc_detail::CornerPack c_corner_pack = mc_detail::make_corner_pack();

// shared memory of one warp's emit (`out`: only for stores to host memory).  Kept
// small: what shared memory leaves of an SM's 256 KB is its L1 cache, which
// neighbouring blocks' ghost layers are read through.
template <bool kHost>
struct McWarpMem {
    // cells and triangles listed at a time (one block has up to 64 and 320)
    static constexpr uint32_t kCells = 128, kTris = 512;
    float vol[kMcBlocks][128];  // the blocks' 5^3 grids
    // cells with triangles, in order: x is, from bit 16, where triangle 0 of the list
    // would be in the cell's row of the case table, and below where the cell is in
    // the cells' table; y its corner 0 in vol, and from bit 30 the block (all but
    // the last in bytes from the table's or array's start)
    uint2 list[kCells];
    uint8_t flag[kTris];  // 1 where a triangle is its cell's first; zero between emits
    uint32_t slot[32];    // the lookups' slots, lane 8j + o
    uint2 out[kHost ? 64 : 2];
};
static_assert(sizeof(McWarpMem<false>) % 16 == 0 && sizeof(McWarpMem<true>) % 16 == 0, "16-byte aligned in an array");

template <int kThreads, bool kHost>
struct McShared {
    McTables tab;
    McWarpMem<kHost> warp[kThreads / 32];
};

__device__ __forceinline__ void async_copy16(void* dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void async_copy4(void* dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kLeft>
__device__ __forceinline__ void async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(kLeft) : "memory");
}

// Starts the copy of the tables, in two groups (async_wait<1> and a barrier
// before the first tables' use, async_wait<0> and a barrier before the
// others'), and clears the warp's flags.
template <int kThreads, bool kHost>
__device__ __forceinline__ void mc_shared_begin(McShared<kThreads, kHost>& s)
{
    char* dst = reinterpret_cast<char*>(&s.tab);
    const char* src = reinterpret_cast<const char*>(&c_mc);
    for (uint32_t i = threadIdx.x; i < kMcFirstTables; i += kThreads) async_copy16(dst + 16u * i, src + 16u * i);
    async_commit();
    for (uint32_t i = kMcFirstTables + threadIdx.x; i < sizeof(McTables) / 16; i += kThreads)
        async_copy16(dst + 16u * i, src + 16u * i);
    async_commit();
    uint32_t* f = reinterpret_cast<uint32_t*>(s.warp[threadIdx.x >> 5].flag);
    for (uint32_t i = threadIdx.x & 31u; i < sizeof(s.warp[0].flag) / 4; i += 32u) f[i] = 0u;
}

// A lane's part of every block: where its four grid voxels come from
// (neighbour o, voxel within that block), and its two cells.
struct McLane {
    const float* src[4];       // the voxel in slot 0 of the cache
    const uint32_t* where[4];  // the slot of its neighbour of block 0, in the warp's memory
    uint32_t g;           // corner 0 of cell `lane` in the grid; cell lane + 32's is at g + 50
    uint32_t need;        // axes on which cell `lane` needs the ghost layer, and from bit 3 cell lane + 32
    // the emit's turn of 32 triangles into 96 vertices in order (mc_emit)
    uint32_t from, turn;  // the lane whose first vertex comes here, and which of the three it then is
    uint32_t tri[3];      // the lanes whose triangles vertices lane, 32 + lane and 64 + lane are of
};
__device__ __forceinline__ McLane mc_lane(const float* cache, const uint32_t* slots)
{
    const uint32_t lane = threadIdx.x & 31u;
    McLane m;
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) {
        uint32_t v = lane + 32u * r;
        if (v >= 125u) v = 0u;
        const uint32_t x = v % 5u, y = (v / 5u) % 5u, z = v / 25u;
        m.where[r] = slots + ((x >> 2) | ((y >> 2) << 1) | ((z >> 2) << 2));
        m.src[r] = cache + ((x & 3u) + 4u * ((y & 3u) + 4u * (z & 3u)));
    }
    const uint32_t x = lane & 3u, y = (lane >> 2) & 3u, z = lane >> 4;
    m.g = x + 5u * (y + 5u * z);
    const uint32_t xy = (x == 3u ? 1u : 0u) | (y == 3u ? 2u : 0u);
    m.need = xy | ((xy | (z == 1u ? 4u : 0u)) << 3);
    m.from = (11u * lane) & 31u;
    m.turn = (3u * m.from) >> 5;
#pragma unroll
    for (uint32_t k = 0; k < 3; ++k) m.tri[k] = (lane + 32u * k) / 3u;
    return m;
}

// The lane's neighbour of its block, as read: lane 8j + o, block j, neighbour o.
struct McLook {
    uint32_t id, slot, act, exist;
};
// Starts the loads of a lookup; a lane of no block passes valid = false.
// `active(nid)` says whether a block is active.
template <typename Active>
__device__ __forceinline__ McLook mc_look(bool valid, uint32_t id, const BlockGrid& grid, const int32_t* item_slots,
                                          Active active)
{
    const uint32_t o = threadIdx.x & 7u;
    McLook l{id, 0u, 0u, 0u};
    if (valid) {
        const uint3 c = block_coords(id, grid), nb = grid.nb;
        l.exist = (c.x + 1u < nb.x ? 1u : 0u) | (c.y + 1u < nb.y ? 2u : 0u) | (c.z + 1u < nb.z ? 4u : 0u);
        if ((o & ~l.exist) == 0u) {
            const uint32_t nid = id + (o & 1u) + nb.x * (((o >> 1) & 1u) + nb.y * (o >> 2));
            l.slot = (uint32_t)__ldg(item_slots + nid);
            l.act = active(nid);
        }
    }
    return l;
}
// Ends it: `slots_of` takes where each lane's neighbour is cached (the block's
// own slot if its grid does not reach into that neighbour), and `has` is the
// axes of the block's ghost layer.  A needed block that no slot holds cannot
// happen with a consistent cache: it is reported (`self_err` for the block
// itself, the next code for a neighbour), and slot 0 is read.
__device__ __forceinline__ void mc_look_end(const McLook& l, const McTables& tab, uint32_t slots, uint32_t* error,
                                            uint32_t self_err, uint32_t* slots_of, uint32_t& has)
{
    const uint32_t lane = threadIdx.x & 31u, o = lane & 7u;
    const uint32_t bits = __ballot_sync(kFull, l.act != 0u) >> (lane & 24u);
    has = tab.ghost.h[(l.exist << 7) | ((bits >> 1) & 127u)];
    uint32_t slot = l.slot;
    const uint32_t self = __shfl_sync(kFull, slot, lane & 24u);
    if ((o & ~has) != 0u) slot = self;
    if (slot >= slots) {
        atomicCAS(error, 0u, o == 0u ? self_err : self_err + 1u);
        slot = 0u;
    }
    __syncwarp();  // the last round's slots have been read
    slots_of[lane] = slot;
    __syncwarp();
}

// The grid voxels of blocks 0 .. n - 1, all loads in flight together.
__device__ __forceinline__ void mc_voxels(const McLane& m, uint32_t n, float f[kMcBlocks][4])
{
#pragma unroll
    for (uint32_t j = 0; j < kMcBlocks; ++j)
        if (j < n) {
#pragma unroll
            for (uint32_t r = 0; r < 4; ++r) f[j][r] = __ldg(m.src[r] + (uint64_t)m.where[r][8u * j] * 64u);
        }
}

// warp_inclusive_scan in two instructions a step: the shuffle itself says
// whether there was a lane to add
__device__ __forceinline__ uint32_t mc_scan(uint32_t v)
{
#pragma unroll
    for (uint32_t o = 1; o < 32u; o <<= 1)
        asm volatile(
            "{ .reg .u32 t; .reg .pred p; shfl.sync.up.b32 t|p, %0, %1, 0, 0xffffffff; @p add.u32 %0, %0, t; }"
            : "+r"(v)
            : "r"(o));
    return v;
}

// A cell's case from the corner mask's window at its corner 0.
__device__ __forceinline__ uint32_t mc_case(uint32_t w) { return mc_detail::case_index(w); }

// The cases of the lane's two cells (compute_block_has_vertices.comp:28-51).
// kSkip: false when no cell of the block can have one (uniform over the warp).
template <bool kSkip>
__device__ __forceinline__ bool mc_cases(const McLane& m, const float f[4], float iso, uint32_t has, uint32_t& c0,
                                         uint32_t& c1)
{
    const uint32_t m0 = __ballot_sync(kFull, f[0] <= iso), m1 = __ballot_sync(kFull, f[1] <= iso),
                   m2 = __ballot_sync(kFull, f[2] <= iso), m3 = __ballot_sync(kFull, f[3] <= iso);
    c0 = c1 = 0u;
    if (kSkip && ((m0 | m1 | m2 | m3) == 0u || (m0 & m1 & m2 & m3) == 0xffffffffu)) return false;
    const bool lo = m.g < 32u, lo1 = m.g < 14u;  // g + 50 < 64
    c0 = mc_case(__funnelshift_r(lo ? m0 : m1, lo ? m1 : m2, m.g & 31u));
    c1 = mc_case(__funnelshift_r(lo1 ? m1 : m2, lo1 ? m2 : m3, (m.g + 50u) & 31u));
    if (has != 7u) {  // uniform; most blocks have their whole ghost layer
        if ((m.need & 7u & ~has) != 0u) c0 = 0u;
        if (((m.need >> 3) & ~has) != 0u) c1 = 0u;
    }
    return true;
}

// Where an emit's vertices go.  Device memory: at once, lane by lane.
// Page-locked host memory (kHost): held back until a 256-byte-aligned window of
// 32 is full -- stores over the host link run about 20 % faster so -- with the
// rest carried on to the next emit, whose vertices follow; `finish` stores what
// is left.
template <bool kHost>
struct McSink {
    uint2* at;          // where the next vertex goes (device memory: the lane's next)
    uint32_t held = 0;  // vertices waiting in the staging buffer (kHost)

    __device__ __forceinline__ explicit McSink(uint2* first) { start(first); }
    __device__ __forceinline__ void start(uint2* first) { at = first + (kHost ? 0u : threadIdx.x & 31u); }
    // vertices 32k + lane of a window's nv (up to 96)
    __device__ __forceinline__ void put(uint2* stage, uint32_t k, uint32_t nv, uint2 v)
    {
        const uint32_t lane = threadIdx.x & 31u;
        if constexpr (!kHost) {
            if (lane + 32u * k < nv) at[32u * k] = v;
        } else {
            const uint32_t n = nv - min(nv, 32u * k);
            if (lane < n) stage[held + lane] = v;
            __syncwarp();
            held += min(n, 32u);
            flush(stage, false);
        }
    }
    __device__ __forceinline__ void next_window(uint32_t n)
    {
        if constexpr (!kHost) at += n;
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

// Starts the copies of the grids of blocks 0 .. n - 1 into the warp's memory.
template <typename Mem>
__device__ __forceinline__ void mc_grids(const McLane& m, Mem& s, uint32_t n)
{
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (uint32_t j = 0; j < kMcBlocks; ++j)
        if (j < n) {
#pragma unroll
            for (uint32_t r = 0; r < 4; ++r)
                async_copy4(&s.vol[j][lane + 32u * r], m.src[r] + (uint64_t)m.where[r][8u * j] * 64u);
        }
    async_commit();
}

// The vertices of blocks 0 .. n - 1 (mc_grids done; ids, isovalues and `has` in
// lane 8j) to the sink, in block, cell and table order.  The cells with
// triangles are listed first, with a flag at each one's first triangle, as many
// blocks' as the list holds (in most cases all).  Then, 32 triangles at a time,
// a ballot of the flags tells a lane which cell its triangle is of: the last that
// starts at or before it.  What is the cell's is so looked up once for three
// vertices; for stores that are contiguous the 96 then change lanes: vertex
// 3 s + r of lane s's triangle belongs in lane (3 s + r) mod 32, for one r a
// different lane for each s, so three shuffles move them, and a lane's three
// arrive turned by 0, 1 or 2 places, which is the same in every window.
// Issue slots (75 % taken) and the shared-memory pipe (79 %) bind this loop alike:
// with a vertex to a lane the kernel took 868 us of the 512^3 volume's query (165 M
// vertices, 812 M warp instructions), now 789 us (720 M).  A shuffle takes two
// turns of that pipe; still, staging the 96 in shared memory instead, and a table
// of the edges' or fixed axes' positions, took over twice the accesses.
// `ahead` is called once, when the grids are there, to start loads for what
// comes next.
template <bool kHost, bool kOneIso, typename Ahead>
__device__ __forceinline__ void mc_emit(const McLane& m, const McTables& tab, McWarpMem<kHost>& s, uint32_t n,
                                        uint32_t id, uint32_t has, float iso, McSink<kHost>& sink, Ahead ahead)
{
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    const char *rows = reinterpret_cast<const char*>(&tab.rows), *cell_recs = reinterpret_cast<const char*>(&tab.cells);
    async_wait<0>();
    __syncwarp();
    ahead();
    uint32_t b = 0;
    do {
        uint32_t tris = 0, cells = 0;
#pragma unroll 1
        for (; b < n; ++b) {
            float f[4];
#pragma unroll
            for (uint32_t r = 0; r < 4; ++r) f[r] = s.vol[b][lane + 32u * r];
            uint32_t c0, c1;
            mc_cases<false>(m, f, kOneIso ? iso : __shfl_sync(kFull, iso, 8u * b), __shfl_sync(kFull, has, 8u * b), c0, c1);
            const uint32_t t0 = tab.count.n[c0], t1 = tab.count.n[c1];
            const uint32_t inc = mc_scan(t0 | (t1 << 16));
            const uint32_t tot = __shfl_sync(kFull, inc, 31), sum = (tot & 0xffffu) + (tot >> 16);
            const uint32_t e0 = __ballot_sync(kFull, t0 != 0u), e1 = __ballot_sync(kFull, t1 != 0u);
            const uint32_t n0 = __popc(e0), n01 = n0 + __popc(e1);
            if (cells + n01 > s.kCells || tris + sum > s.kTris) break;
            const uint32_t where = 4u * m.g + 512u * b + (b << 30);  // cell lane + 32 lies two layers up
            if (t0) {
                const uint32_t first = tris + (inc & 0xffffu) - t0;
                s.list[cells + __popc(e0 & below)] = make_uint2(((80u * c0 - 16u * first) << 16) + 8u * lane, where);
                s.flag[first] = 1;
            }
            if (t1) {
                const uint32_t first = tris + (tot & 0xffffu) + (inc >> 16) - t1;
                s.list[cells + n0 + __popc(e1 & below)] =
                    make_uint2(((80u * c1 - 16u * first) << 16) + 8u * lane + 256u, where + 200u);
                s.flag[first] = 1;
            }
            tris += sum;
            cells += n01;
        }
        __syncwarp();
        uint32_t before = 0;  // cells that start before the window of 32 triangles
#pragma unroll 1
        for (uint32_t w = 0; w < tris; w += 32u) {
            const uint32_t starts = __ballot_sync(kFull, s.flag[w + lane] != 0);
            s.flag[w + lane] = 0;
            const uint32_t nt = min(tris - w, 32u), nv = 3u * nt;
            const uint2 e = s.list[before + __popc(starts & (2u * below + 1u)) - 1u];
            const uint32_t block = e.y >> 27;  // the lane that has the block's values: 8j
            const uint32_t bid = __shfl_sync(kFull, id, block);
            const float biso = kOneIso ? iso : __shfl_sync(kFull, iso, block);
            // lanes past the last triangle work on that, which is not kept
            const uint4 row = *reinterpret_cast<const uint4*>(rows + ((int32_t)e.x >> 16) +
                                                              (int32_t)(16u * (w + min(lane, nt - 1u))));
            const uint2 rec2 = *reinterpret_cast<const uint2*>(cell_recs + (e.x & 0xffffu));
            const mc_detail::CellRec rec{rec2.x, rec2.y};
            const float* vol = reinterpret_cast<const float*>(reinterpret_cast<const char*>(&s.vol[0][0]) + (e.y & 0x7ffu));
            bool a0, a1, a2;
            uint32_t v0 = mc_vertex_fast(row.x, vol, rec, biso, &a0), v1 = mc_vertex_fast(row.y, vol, rec, biso, &a1),
                     v2 = mc_vertex_fast(row.z, vol, rec, biso, &a2);
            if ((a0 || a1 || a2) && lane < nt) {
                const uint32_t c = (e.x & 0xffffu) >> 3, cell = ((c & 3u) << 20) | (((c >> 2) & 3u) << 10) | (c >> 4);
                uint32_t redo = (a0 ? 1u : 0u) | (a1 ? 2u : 0u) | (a2 ? 4u : 0u);
#pragma unroll 1
                for (; redo; redo &= redo - 1u) {
                    const uint32_t v = mc_vertex_exact(redo & 1u ? row.x : redo & 2u ? row.y : row.z, s.vol[block >> 3], cell,
                                                       &c_corner_pack.p[0][0], biso);
                    if (redo & 1u) v0 = v;
                    else if (redo & 2u) v1 = v;
                    else v2 = v;
                }
            }
            __syncwarp();
            v0 = __shfl_sync(kFull, v0, m.from);
            v1 = __shfl_sync(kFull, v1, m.from - 11u);
            v2 = __shfl_sync(kFull, v2, m.from - 22u);
            const bool one = m.turn == 1u, two = m.turn == 2u;
            sink.put(s.out, 0u, nv, make_uint2(one ? v1 : two ? v2 : v0, __shfl_sync(kFull, bid, m.tri[0])));
            sink.put(s.out, 1u, nv, make_uint2(one ? v0 : two ? v1 : v2, __shfl_sync(kFull, bid, m.tri[1])));
            sink.put(s.out, 2u, nv, make_uint2(one ? v2 : two ? v0 : v1, __shfl_sync(kFull, bid, m.tri[2])));
            sink.next_window(nv);
            before += __popc(starts);
        }
        __syncwarp();  // the next grids and lists overwrite these
    } while (b < n);
}

}  // namespace bcmc
