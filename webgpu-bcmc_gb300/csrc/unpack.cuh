// unpack.cuh -- a packed vertex's world and clip position: the vertex stage's
// math (shaders/mc_isosurface.vert:51-60 with block_vertex_position.comp:19-26),
// shared by bcmc_unpack_vertices (unpack.cu) and the render pass (render.cu),
// which works positions out where it needs them instead of storing them.
#pragma once

#include "bcmc_internal.cuh"
#include "exact_div.cuh"

namespace bcmc {

struct VertexStage {
    BlockGrid grid;
    float dims[3], inv_dims[3], scale[3];
    float m[16];  // column-major view-projection
};

inline VertexStage make_vertex_stage(const uint32_t dims[3], const float scale[3], const float* proj_view)
{
    VertexStage v{};
    v.grid = make_block_grid(make_uint3(div_up(dims[0], 4u), div_up(dims[1], 4u), div_up(dims[2], 4u)));
    for (int k = 0; k < 3; ++k) {
        v.dims[k] = (float)dims[k];
        v.inv_dims[k] = 1.0f / v.dims[k];
        v.scale[k] = scale ? scale[k] : 1.0f;
    }
    for (int k = 0; k < 16; ++k) v.m[k] = proj_view ? proj_view[k] : (k % 5 == 0 ? 1.0f : 0.0f);
    return v;
}

// block: the coordinates of the vertex's block (block_coords of its id)
__device__ __forceinline__ void vertex_world(const VertexStage& s, uint32_t packed, uint3 block, float w[3])
{
    const float q[3] = {(float)((packed & 0x3ff00000u) >> 20), (float)((packed & 0x000ffc00u) >> 10),
                        (float)(packed & 0x000003ffu)};
    const float bp[3] = {__fmul_rn(4.0f, (float)block.x), __fmul_rn(4.0f, (float)block.y),
                         __fmul_rn(4.0f, (float)block.z)};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        // decompress_position: (quantized * 4.0) / 1023 + 0.5
        const float d = __fadd_rn(exact_div(__fmul_rn(q[k], 4.0f), 1023.0f, 1.0f / 1023.0f), 0.5f);
        // world = scale * ((block_pos + d) / dims - 0.5)
        w[k] = __fmul_rn(s.scale[k], __fsub_rn(exact_div(__fadd_rn(bp[k], d), s.dims[k], s.inv_dims[k]), 0.5f));
    }
}

__device__ __forceinline__ void vertex_clip(const VertexStage& s, const float w[3], float c[4])
{
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        float acc = __fmul_rn(s.m[r], w[0]);
        acc = __fadd_rn(acc, __fmul_rn(s.m[4 + r], w[1]));
        acc = __fadd_rn(acc, __fmul_rn(s.m[8 + r], w[2]));
        c[r] = __fadd_rn(acc, s.m[12 + r]);  // * 1.0
    }
}

}  // namespace bcmc
