// active_test.cuh -- the active-block test of compute_block_active.comp in words
// of 32 blocks, for the per-query pipeline (pipeline.cu) and the batched engine
// (engine.cu).
//
// compute_block_active.comp:24-61 tests, for each of the 26 neighbours n, iso in
// [min(lo_b, lo_n), max(hi_b, hi_n)].  With A = (iso >= lo), B = (iso <= hi) that
// is (A_b || A_n) && (B_b || B_n), so over all neighbours (and b itself, which
// adds nothing new):
//   active = (A_b && anyB) || (B_b && anyA) || any(A_n && B_n)
// -- the same booleans.  The bits of A, B and A && B are ORed along x (spread),
// then over the nine (y, z) rows of a word's blocks, those that the volume has
// (word_rows).
#pragma once

#include "bcmc_internal.cuh"
#include "bcmc_pipeline.h"

namespace bcmc {

// Of the 32 blocks from b0 on: those with a row before and after them in y and in z.
struct WordRows {
    uint32_t ym, yp, zm, zp;
    uint32_t sound;  // those whose coordinates are below SoundRanges'

    __device__ __forceinline__ uint32_t mask(int dy, int dz) const
    {
        return (dz < 0 ? zm : dz > 0 ? zp : 0xffffffffu) & (dy < 0 ? ym : dy > 0 ? yp : 0xffffffffu);
    }
};

__device__ __forceinline__ WordRows word_rows(uint32_t b0, const BlockGrid& g, const SoundRanges& sound)
{
    WordRows r{0u, 0u, 0u, 0u, 0u};
    uint3 c = block_coords(b0, g);
    for (uint32_t p = 0; p < 32u;) {  // the pieces of rows in the word
        const uint32_t len = min(g.nb.x - c.x, 32u - p);
        const uint32_t m = (0xffffffffu >> (32u - len)) << p;
        r.ym |= c.y > 0u ? m : 0u;
        r.yp |= c.y + 1u < g.nb.y ? m : 0u;
        r.zm |= c.z > 0u ? m : 0u;
        r.zp |= c.z + 1u < g.nb.z ? m : 0u;
        const uint32_t n = c.y < sound.y && c.z < sound.z && c.x < sound.x ? min(len, sound.x - c.x) : 0u;
        r.sound |= n ? (0xffffffffu >> (32u - n)) << p : 0u;
        p += len;
        c.x = 0;
        if (++c.y == g.nb.y) {
            c.y = 0;
            ++c.z;
        }
    }
    return r;
}

// Of the 32 blocks from b0 on: those at x = 0 and at x = nx - 1, which have no neighbour there.
struct WordEnds {
    uint32_t no_left, no_right;

    // The word's bits ORed with those of the block after each along x.
    __device__ __forceinline__ uint32_t up(uint32_t v, uint32_t next) const
    {
        return v | (__funnelshift_r(v, next, 1) & ~no_right);
    }
    // The word's bits ORed with those of the blocks before and after each along x;
    // the last bit of `prev` and the first of `next` are those beside the word.
    __device__ __forceinline__ uint32_t spread(uint32_t v, uint32_t prev, uint32_t next) const
    {
        return up(v, next) | (__funnelshift_l(prev, v, 1) & ~no_left);
    }
};

__device__ __forceinline__ WordEnds word_ends(uint32_t b0, const BlockGrid& g)
{
    const uint32_t nx = g.nb.x, x0 = b0 - fdiv(b0, g.dx) * nx;
    WordEnds e{0u, 0u};
    for (uint32_t p = x0 ? nx - x0 : 0u; p < 32u; p += nx) e.no_left |= 1u << p;
    for (uint32_t p = nx - 1u - x0; p < 32u; p += nx) e.no_right |= 1u << p;
    return e;
}

}  // namespace bcmc
