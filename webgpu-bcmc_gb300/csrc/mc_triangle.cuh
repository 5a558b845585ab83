// mc_triangle.cuh -- a triangle's vertices as the MC kernels emit them: the
// case table by triangle, the grid's edge table, and mc_vertex's position
// without its division for nearly every vertex.  Free of the CUDA runtime, like
// mc_vertex.cuh, so that a host build of it can be checked against mc_vertex.
#pragma once

#include "mc_vertex.cuh"

namespace bcmc {

namespace mc_detail {
// The case table as the kernels read it.  Cases are numbered by the corners in
// natural order (bit x|y<<1|z<<2), which is how a cell's corners fall out of
// its block's bit mask (mc_case).  A row holds up to five triangles, a word to
// each vertex:
//   bits 0-7    4 * the edge's first corner's offset in the grid (grid_off)
//   bits 8-15   4 * its second corner's
//   bits 16-20  where the edge's axis lies in a packed position (20, 10, 0)
//   bits 24-25  the axis
//   bits 26-28  the first corner
//   bit 31      the first corner is the edge's far end
// The counts are triangles, four bits to a case, so that the 32 words of the
// table lie on the 32 banks.
struct TriRows {
    uint32_t t[256][5][4];
    uint32_t ntri[32];
};
constexpr uint32_t reference_case(uint32_t natural)
{
    uint32_t c = 0;
    for (int i = 0; i < 8; ++i) c |= ((natural >> kCorner[i]) & 1u) << i;
    return c;
}
constexpr uint32_t tri_word(uint32_t e)  // from an entry of TriEdges
{
    if (e == 0xffffu) return 0u;
    const uint32_t d = (e >> 10) & 3u, oa = (e >> 12) & 7u;
    return (4u * (e & 31u)) | (4u * ((e >> 5) & 31u) << 8) | ((20u - 10u * d) << 16) | (d << 24) | (oa << 26) |
           (((oa >> d) & 1u) << 31);
}
constexpr TriRows make_tri_rows()
{
    TriRows t{};
    const TriEdges e = make_tri_edges();
    const TriCorners n = make_tri_corners();
    for (uint32_t c = 0; c < 256; ++c) {
        const uint32_t r = reference_case(c);
        for (int k = 0; k < 15; ++k) t.t[c][k / 3][k % 3] = tri_word(e.e[r][k]);
        t.ntri[c >> 3] |= (uint32_t)(n.count[r] / 3) << (4u * (c & 7u));
    }
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
// Per axis d and grid index v (x + 5y + 25z): the packed position of grid point
// v on the two other axes, and 255.75 times its coordinate on d, less a half.
struct EdgeBase {
    uint32_t pack;
    float base;
};
struct EdgeBases {
    EdgeBase b[3][128];
};
constexpr EdgeBases make_edge_bases()
{
    EdgeBases t{};
    for (uint32_t d = 0; d < 3; ++d)
        for (uint32_t v = 0; v < 125; ++v) {
            const uint32_t c[3] = {v % 5u, (v / 5u) % 5u, v / 25u};
            for (uint32_t ax = 0; ax < 3; ++ax)
                if (ax != d) t.b[d][v].pack |= q10(c[ax]) << (20u - 10u * ax);
            t.b[d][v].base = (float)c[d] * 255.75f - 0.5f;
        }
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
// word of TriRows; `vol` and `eb`: the grid and the edge table at the cell's
// corner 0.  Returns the packed position, or sets *again when the exact
// expression has to decide.
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
__device__ __forceinline__ uint32_t mc_vertex_fast(uint32_t w, const float* vol, const mc_detail::EdgeBase* eb,
                                                   float iso, bool* again)
{
    const char* vb = reinterpret_cast<const char*>(vol);
    const float fa = *reinterpret_cast<const float*>(vb + (w & 0xffu));
    const float fb = *reinterpret_cast<const float*>(vb + ((w >> 8) & 0xffu));
    const mc_detail::EdgeBase e = *reinterpret_cast<const mc_detail::EdgeBase*>(
        reinterpret_cast<const char*>(eb) + 2u * (w & 0xffu) + ((w >> 14) & 0xc00u));
    const float b = __fsub_rn(fb, fa);
    const float t = __fmul_rn(__fsub_rn(iso, fa), mc_rcp(b));
    const float u = fmaf((w >> 31) ? -255.75f : 255.75f, t, e.base);
    const float y = __fadd_rn(u, 12582912.0f);
    const float d = __fsub_rn(u, __fsub_rn(y, 12582912.0f));
    if (!(fabsf(d) < 0.4996f && fabsf(b) >= 0.001f && fabsf(b) < 1e37f)) *again = true;
    return e.pack | ((__float_as_uint(y) & 0x3ffu) << ((w >> 16) & 31u));
}

// the entry of TriEdges that a word of TriRows was made from
__device__ __forceinline__ uint32_t mc_word_entry(uint32_t w)
{
    return ((w >> 2) & 31u) | (((w >> 10) & 31u) << 5) | (((w >> 24) & 3u) << 10) | (((w >> 26) & 7u) << 12);
}

}  // namespace bcmc
