// mc_triangle.cuh -- vertices as the MC kernels emit them: the case table in
// their numbering of the cases, and mc_vertex's position without its division
// for nearly every vertex.  Free of the CUDA runtime, like
// mc_vertex.cuh, so that a host build of it can be checked against mc_vertex.
#pragma once

#include "mc_vertex.cuh"

namespace bcmc {

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
// fifteen vertices:
//   bits 0, 10, 20  the z, y and x offset of the edge's first corner
//   bits 2-6        that corner's offset in the grid (grid_off)
//   bits 11-15      the second corner's
//   bits 26-30      where the edge's axis lies in a packed position (20, 10, 0)
//   bit 31          the first corner is the edge's far end
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
    const uint32_t d = (e >> 10) & 3u, oa = (e >> 12) & 7u;
    return ((oa & 1u) << 20) | (((oa >> 1) & 1u) << 10) | (oa >> 2) | ((e & 31u) << 2) | (((e >> 5) & 31u) << 11) |
           ((20u - 10u * d) << 26) | (((oa >> d) & 1u) << 31);
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

constexpr uint32_t kAxisOnes = (1u << 20) | (1u << 10) | 1u;

// mc_vertex without its division, for nearly every vertex.  `w`: the vertex's
// word of CaseRows; `vol`: the grid at the cell's corner 0; `cell`: the cell's
// position, x << 20 | y << 10 | z.  Returns the packed position, or sets *again
// when the exact expression has to decide.
//
// The two axes that the edge does not vary along are exact: coordinate c in 0..4
// quantizes to floor(255.75 c) = 256 c - (c > 0), all fields at once.
//
// Along the edge's axis the vertex quantizes to floor(x), x = 255.75 * (c +- t)
// with c the first corner's coordinate and t = (iso - fa) / (fb - fa).  The
// reference's rounded chain is within 2.5e-4 of the exact x (t to 2^-24, the
// sums p + v + 0.5 - 0.5 below 5 to 7e-7 in all, times 255.75, and the last
// product to 2^-24 of 1023), and the product with an approximate reciprocal
// here within 8e-5 (t to 2^-22.4, the sum to 2^-15); so where this x lies more
// than 4e-4 from a whole number, both have the same floor.  u = x - 1/2 is
// rounded by adding 1.5 * 2^23, whose low bits are then the floor, and |u -
// rounded| < 1/2 - 4e-4 says it is safe.  The vertices near a whole number
// (0.08 % of them), edges the reference puts at t = 0 (ends closer than
// 0.001), and ends too large for the reciprocal are left to mc_vertex.
__device__ __forceinline__ uint32_t mc_vertex_fast(uint32_t w, const float* vol, uint32_t cell, float iso, bool* again)
{
    const char* vb = reinterpret_cast<const char*>(vol);
    const float fa = *reinterpret_cast<const float*>(vb + (w & 0x7cu));
    const float fb = *reinterpret_cast<const float*>(vb + ((w >> 9) & 0x7cu));
    const uint32_t sh = (w >> 26) & 31u;
    const uint32_t corner = cell + (w & kAxisOnes);
    const float base = fmaf((float)((corner >> sh) & 7u), 255.75f, -0.5f);  // exact
    const uint32_t fixed = corner & ~(7u << sh);
    const uint32_t pack = 256u * fixed - (((fixed + 7u * kAxisOnes) >> 3) & kAxisOnes);
    const float b = __fsub_rn(fb, fa);
    const float t = __fmul_rn(__fsub_rn(iso, fa), mc_rcp(b));
    const float u = fmaf((w >> 31) ? -255.75f : 255.75f, t, base);
    const float y = __fadd_rn(u, 12582912.0f);
    const float d = __fsub_rn(u, __fsub_rn(y, 12582912.0f));
    *again = !(fabsf(d) < 0.4996f && fabsf(b) >= 0.001f && fabsf(b) < 1e37f);
    return pack | ((__float_as_uint(y) & 0x3ffu) << sh);
}

// the entry of TriEdges that a word of CaseRows was made from
__device__ __forceinline__ uint32_t mc_word_entry(uint32_t w)
{
    const uint32_t axis = 2u - ((w >> 26) & 31u) / 10u;
    return ((w >> 2) & 31u) | (((w >> 11) & 31u) << 5) | (axis << 10) | (((w >> 20) & 1u) << 12) |
           (((w >> 10) & 1u) << 13) | ((w & 1u) << 14);
}
// mc_vertex by the same arguments (`grid`: the whole grid)
__device__ __forceinline__ uint32_t mc_vertex_exact(uint32_t w, const float* grid, uint32_t cell, const uint32_t* cp,
                                                    float iso)
{
    const uint32_t cc = ((cell >> 20) & 3u) | (((cell >> 10) & 3u) << 2) | ((cell & 3u) << 4);
    return mc_vertex(mc_word_entry(w), cc, grid, cp, iso);
}

}  // namespace bcmc
