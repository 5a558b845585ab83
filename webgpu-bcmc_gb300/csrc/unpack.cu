// unpack.cu -- world-space positions of packed vertices: the position math of
// the reference's vertex stage (shaders/mc_isosurface.vert:51-60 with
// block_vertex_position.comp:19-26), as a CUDA kernel for consumers of the
// mesh that do not decode the packed form themselves.
#include "bcmc_impl.h"
#include "unpack.cuh"

namespace bcmc {
namespace {

struct UnpackArgs {
    const uint2* verts;
    uint64_t n;
    VertexStage stage;
    int has_clip;
    float* world;  // 3 floats per vertex
    float* clip;   // 4 floats per vertex
};

__global__ void __launch_bounds__(256) k_unpack(UnpackArgs a)
{
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < a.n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint2 v = __ldg(a.verts + i);
        float w[3];
        vertex_world(a.stage, v.x, block_coords(v.y, a.stage.grid), w);
#pragma unroll
        for (int k = 0; k < 3; ++k) a.world[3 * i + k] = w[k];
        if (a.has_clip) {
            float c[4];
            vertex_clip(a.stage, w, c);
#pragma unroll
            for (int r = 0; r < 4; ++r) a.clip[4 * i + r] = c[r];
        }
    }
}

}  // namespace

void unpack_launch(bcmc_ctx* ctx, const uint2* verts, uint64_t n, const uint32_t dims[3], const float scale[3],
                   const float* proj_view, float* world, float* clip, cudaStream_t s)
{
    if (n == 0) return;
    const UnpackArgs a{verts, n, make_vertex_stage(dims, scale, proj_view), proj_view && clip ? 1 : 0, world, clip};
    const uint64_t want = (n + 255) / 256, cap = (uint64_t)ctx->num_sms * 16;
    k_unpack<<<(int)(want < cap ? want : cap), 256, 0, s>>>(a);
    count_launches(1);
    BCMC_CUDA(cudaGetLastError());
}

}  // namespace bcmc
