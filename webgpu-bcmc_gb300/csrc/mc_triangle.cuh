// mc_triangle.cuh -- vertices as the MC kernels emit them: the case table in
// their numbering of the cases, and mc_vertex's position without its division
// for nearly every vertex.  Free of the CUDA runtime, like
// mc_vertex.cuh, so that a host build of it can be checked against mc_vertex.
#pragma once

#include "mc_vertex.cuh"

namespace bcmc {

constexpr uint32_t kAxisOnes = (1u << 20) | (1u << 10) | 1u;  // of a position packed x << 20 | y << 10 | z

namespace mc_detail {
// A cell's corners in its block's bit mask (x + 5y + 25z): bits 0, 1, 5, 6, 25,
// 26, 30 and 31 of the 32-bit window at its corner 0.  The product gathers the
// eight in the top byte, a different byte for each of the 256 cases (checked
// below); this is the number that the kernels know a case by.
constexpr uint32_t kCaseBits = 0xc6000063u, kCaseMul = 0x08800001u;
constexpr uint32_t case_index(uint32_t window) { return ((window & kCaseBits) * kCaseMul) >> 24; }
constexpr uint32_t case_window(uint32_t natural)  // natural: bit x|y<<1|z<<2 per corner
{
    uint32_t w = 0;
    for (uint32_t o = 0; o < 8; ++o) w |= ((natural >> o) & 1u) << grid_off(o);
    return w;
}
constexpr bool case_index_is_unique()
{
    bool seen[256] = {};
    for (uint32_t c = 0; c < 256; ++c) {
        const uint32_t i = case_index(case_window(c));
        if (seen[i]) return false;
        seen[i] = true;
    }
    return case_index(0) == 0;
}
static_assert(case_index_is_unique(), "each case has a number of its own, no corner set is 0");

// The case table as the kernels read it, by case_index: a word to each of up to
// fifteen vertices, for its edge taken from the corner nearer the origin:
//   bits 0, 10, 20  that corner's z, y and x offset (none along the edge)
//   bits 8, 18, 28  the same
//   bits 2-6        its offset in the grid (grid_off)
//   bit 29          the table's first corner is the edge's other end
//   bits 30-31      the edge's axis: 0, 1, 2 for z, y, x
struct CaseRows {
    uint32_t w[256][15];
};
struct TriCounts {
    uint8_t n[256];  // triangles
};
constexpr uint32_t reference_case(uint32_t natural)
{
    uint32_t c = 0;
    for (int i = 0; i < 8; ++i) c |= ((natural >> kCorner[i]) & 1u) << i;
    return c;
}
constexpr uint32_t vertex_word(uint32_t e)  // from an entry of TriEdges
{
    if (e == 0xffffu) return 0u;
    const uint32_t d = (e >> 10) & 3u, oa = (e >> 12) & 7u, ga = e & 31u, gb = (e >> 5) & 31u;
    const uint32_t o = oa & ~(1u << d), spread = ((o & 1u) << 20) | (((o >> 1) & 1u) << 10) | (o >> 2);
    return spread | (spread << 8) | ((ga < gb ? ga : gb) << 2) | (((oa >> d) & 1u) << 29) | ((2u - d) << 30);
}
constexpr CaseRows make_case_rows()
{
    CaseRows t{};
    const TriEdges e = make_tri_edges();
    for (uint32_t c = 0; c < 256; ++c)
        for (int k = 0; k < 15; ++k) t.w[case_index(case_window(c))][k] = vertex_word(e.e[reference_case(c)][k]);
    return t;
}
constexpr TriCounts make_tri_counts()
{
    TriCounts t{};
    const TriCorners n = make_tri_corners();
    for (uint32_t c = 0; c < 256; ++c) t.n[case_index(case_window(c))] = (uint8_t)(n.count[reference_case(c)] / 3);
    return t;
}
constexpr bool whole_triangles()
{
    const TriCorners n = make_tri_corners();
    for (int c = 0; c < 256; ++c)
        if (n.count[c] % 3 != 0 || n.count[c] > 15) return false;
    return true;
}
static_assert(whole_triangles(), "a case is up to five triangles");
// What the emit needs to know of a cell, by its number x + 4y + 16z.
struct CellRec {
    uint32_t pack;  // its coordinates quantized, x << 20 | y << 10 | z: floor(255.75 c), odd where c > 0
    uint32_t frac;  // by axis (z, y, x from the low byte): the second byte of the float 3.5 + 255.75 c - floor(255.75 c)
};
struct CellRecs {
    CellRec r[64];
};
constexpr CellRec cell_rec(uint32_t x, uint32_t y, uint32_t z)
{
    constexpr uint32_t frac[4] = {0x60u, 0x88u, 0x80u, 0x70u};  // 3.5, 4.25, 4, 3.75, whose first byte is 0x40
    return CellRec{(q10(x) << 20) | (q10(y) << 10) | q10(z), frac[z] | (frac[y] << 8) | (frac[x] << 16)};
}
constexpr CellRecs make_cell_recs()
{
    CellRecs t{};
    for (uint32_t c = 0; c < 64; ++c) t.r[c] = cell_rec(c & 3u, (c >> 2) & 3u, c >> 4);
    return t;
}
// The case table with a triangle's three words together.
struct TriRows {
    uint32_t w[256][5][4];
};
constexpr TriRows make_tri_rows()
{
    TriRows t{};
    const CaseRows r = make_case_rows();
    for (int c = 0; c < 256; ++c)
        for (int k = 0; k < 15; ++k) t.w[c][k / 3][k % 3] = r.w[c][k];
    return t;
}
// compute_vertex_values.comp:96-156: the axes on which a block's grid takes the
// ghost layer of its +x/+y/+z neighbours, tested corner, edges, faces.  `exist`:
// axes on which there is a neighbour; bit o of `act`: neighbour o (x|y<<1|z<<2)
// exists and is active.
constexpr uint32_t ghost_axes(uint32_t exist, uint32_t act)
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
struct GhostAxes {
    uint8_t h[1024];  // by exist << 7 | act >> 1
};
constexpr GhostAxes make_ghost_axes()
{
    GhostAxes t{};
    for (uint32_t i = 0; i < 1024; ++i) t.h[i] = (uint8_t)ghost_axes(i >> 7, (i & 127u) << 1);
    return t;
}
}  // namespace mc_detail

// 1 / b to 1 ulp (a host build may put its own in)
#ifndef BCMC_HOST_RCP
#define BCMC_HOST_RCP(b) (1.0f / (b))
#endif
__device__ __forceinline__ float mc_rcp(float b)
{
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
    return r;
#else
    return BCMC_HOST_RCP(b);
#endif
}

// mc_vertex without its division, for nearly every vertex.  `w`: the vertex's
// word of CaseRows; `vol`: the grid at the cell's corner 0; `c`: the cell.
// Returns the packed position, or sets *again when the exact expression has to
// decide.
//
// The edge is taken from its corner nearer the origin, whichever the table puts
// first; that corner has the cell's coordinate c along the edge's axis, and the
// vertex lies at t = (iso - fl) / (fu - fl) from it.  Coordinates quantize to
// floor(255.75 c) = 256 c - (c > 0), all fields at once; along the axis,
// floor(255.75 (c + t)) is that plus floor(z), z the fraction 255.75 c leaves
// plus 255.75 t.
//
// The reference's rounded chain is within 2.5e-4 of the exact 255.75 (c + t) (t
// to 2^-24, the sums p + v + 0.5 - 0.5 below 5 to 7e-7 in all, times 255.75, and
// the last product to 2^-24 of 1023), and the product with an approximate
// reciprocal here within 1e-4 (t to 2^-22.2, the sum to 2^-16); so where this
// lies more than 4e-4 from a whole number, both have the same floor.  u = z +
// 3.5 is rounded by adding 1.5 * 2^23 - 4, which leaves the floor in the low
// bits, and |u - rounded| < 1/2 - 4e-4 says it is safe.  The vertices near a
// whole number (0.08 % of them), edges the reference puts at t = 0 (ends closer
// than 0.001), and ends too large for the reciprocal are left to mc_vertex.
__device__ __forceinline__ uint32_t mc_vertex_fast(uint32_t w, const float* vol, const mc_detail::CellRec& c, float iso,
                                                   bool* again)
{
    const uint32_t axis = w >> 30;
    const char* lower = reinterpret_cast<const char*>(vol) + (w & 0x7cu);
    const float fl = *reinterpret_cast<const float*>(lower);
    const float fu = *reinterpret_cast<const float*>(lower + __byte_perm(0x00041464u, 0u, 0x4440u + axis));  // 25, 5, 1 floats on
    const float from = __int_as_float((int32_t)__byte_perm(c.frac, 0x40000000u, 0x7044u + 256u * axis));
    const float b = __fsub_rn(fu, fl);
    const float t = __fmul_rn(__fsub_rn(iso, fl), mc_rcp(b));
    const float u = fmaf(255.75f, t, from);
    const float y = __fadd_rn(u, 12582908.0f);
    const float d = __fsub_rn(u, __fsub_rn(y, 12582908.0f));
    *again = !(fabsf(d) < 0.4996f && fabsf(b) >= 0.001f && fabsf(b) < 1e37f);
    return c.pack + (w & (kAxisOnes << 8)) - (w & ~c.pack & kAxisOnes) + ((__float_as_uint(y) & 0x3ffu) << (10u * axis));
}
__device__ __forceinline__ uint32_t mc_vertex_fast(uint32_t w, const float* vol, uint32_t cell, float iso, bool* again)
{
    return mc_vertex_fast(w, vol, mc_detail::cell_rec((cell >> 20) & 3u, (cell >> 10) & 3u, cell & 3u), iso, again);
}

// the entry of TriEdges that a word of CaseRows was made from
__device__ __forceinline__ uint32_t mc_word_entry(uint32_t w)
{
    const uint32_t axis = 2u - (w >> 30), far = (w >> 29) & 1u;
    const uint32_t lower = (w >> 2) & 31u, upper = lower + (axis == 0u ? 1u : axis == 1u ? 5u : 25u);
    const uint32_t o = ((w >> 20) & 1u) | (((w >> 10) & 1u) << 1) | ((w & 1u) << 2);
    return (far ? upper | (lower << 5) : lower | (upper << 5)) | (axis << 10) | ((o | (far << axis)) << 12);
}
// mc_vertex by the same arguments (`grid`: the whole grid; `cell`: x << 20 | y << 10 | z)
__device__ __forceinline__ uint32_t mc_vertex_exact(uint32_t w, const float* grid, uint32_t cell, const uint32_t* cp,
                                                    float iso)
{
    const uint32_t cc = ((cell >> 20) & 3u) | (((cell >> 10) & 3u) << 2) | ((cell & 3u) << 4);
    return mc_vertex(mc_word_entry(w), cc, grid, cp, iso);
}

}  // namespace bcmc
