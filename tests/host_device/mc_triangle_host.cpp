// The case table and the division-free vertex of the MC kernels
// (mc_triangle.cuh) built as host code beside mc_vertex, for the CPU test that
// holds the one to the other.
#include "cuda_host_shim.h"

static int g_rcp_ulps = 0;  // the approximate reciprocal's error, in units of the last place
static inline float host_rcp(float b)
{
    float r = 1.0f / b;
    uint32_t u;
    memcpy(&u, &r, 4);
    u += (uint32_t)g_rcp_ulps;
    memcpy(&r, &u, 4);
    return r;
}
static inline uint32_t __float_as_uint(float f)
{
    uint32_t u;
    memcpy(&u, &f, 4);
    return u;
}
#define BCMC_HOST_RCP(b) host_rcp(b)
#include "mc_triangle.cuh"

namespace {
const bcmc::mc_detail::TriEdges kEdges = bcmc::mc_detail::make_tri_edges();
const bcmc::mc_detail::CornerPack kPack = bcmc::mc_detail::make_corner_pack();
const bcmc::mc_detail::TriCorners kTri = bcmc::mc_detail::make_tri_corners();
const bcmc::mc_detail::CaseRows kRows = bcmc::mc_detail::make_case_rows();
const bcmc::mc_detail::TriCounts kCounts = bcmc::mc_detail::make_tri_counts();
// the kernels' number of a case, from a mask with bits of other cells set too
uint32_t index_of(uint32_t natural) { return bcmc::mc_detail::case_index(bcmc::mc_detail::case_window(natural) | 0x39ffff9cu); }
}  // namespace

extern "C" uint32_t tri_count(uint32_t natural) { return kCounts.n[index_of(natural)]; }
extern "C" uint32_t ref_count(uint32_t natural) { return kTri.count[bcmc::mc_detail::reference_case(natural)]; }
extern "C" uint32_t word_entry(uint32_t natural, uint32_t k) { return bcmc::mc_word_entry(kRows.w[index_of(natural)][k]); }
extern "C" uint32_t ref_entry(uint32_t natural, uint32_t k)
{
    return kEdges.e[bcmc::mc_detail::reference_case(natural)][k];
}

// n vertices: natural case, vertex, cell, 8 corner values (natural order) and
// isovalue each; the fast result, whether it asked for the exact one, and the
// exact one
extern "C" void vertices(uint32_t n, const uint32_t* natural, const uint32_t* k, const uint32_t* cell,
                         const float* corners, const float* iso, int rcp_ulps, uint32_t* fast, uint8_t* again,
                         uint32_t* exact)
{
    g_rcp_ulps = rcp_ulps;
    for (uint32_t i = 0; i < n; ++i) {
        float vol[128];
        for (float& v : vol) v = NAN;
        const uint32_t cc = cell[i], g = (cc & 3u) + 5u * ((cc >> 2) & 3u) + 25u * (cc >> 4);
        for (uint32_t o = 0; o < 8; ++o) vol[g + bcmc::mc_detail::grid_off(o)] = corners[8 * i + o];
        const uint32_t w = kRows.w[index_of(natural[i])][k[i]];
        bool a = false;
        fast[i] = bcmc::mc_vertex_fast(w, vol + g, ((cc & 3u) << 20) | (((cc >> 2) & 3u) << 10) | (cc >> 4), iso[i], &a);
        again[i] = a;
        exact[i] = bcmc::mc_vertex_exact(w, vol, ((cc & 3u) << 20) | (((cc >> 2) & 3u) << 10) | (cc >> 4), &kPack.p[0][0], iso[i]);
    }
}
