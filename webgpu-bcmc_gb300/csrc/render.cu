// render.cu -- headless rendering of an isosurface mesh into a device image:
// the reference's render pass (js/bcmc.js:174-190,237-265,377-391) with the
// shading of shaders/mc_isosurface.vert/.frag, as CUDA kernels instead of a
// graphics pipeline (no window, swapchain or graphics API).
//
//   k_raster      one thread per triangle: its three vertices' clip positions
//                 (unpack.cuh) -> NDC -> pixels (WebGPU conventions: y up in
//                 NDC, depth in [0, 1]), edge functions with a top-left rule at
//                 pixel centres, depth "less" against a buffer cleared to 1.0 --
//                 each covered pixel takes the 64-bit atomicMin of (depth bits,
//                 triangle id), so the result does not depend on thread order
//   k_resolve     one thread per pixel: the winning triangle's fragment shading
//                 (mc_isosurface.frag:15-40: flat normal, Blinn-Phong, optional
//                 fog with mc_isosurface.vert:35-49's entry distances),
//                 background (1, 1, 1, 1) where no triangle won
// Positions are worked out from the packed vertices where they are needed: 24
// bytes a triangle, and a covered pixel again, where stored world and clip
// positions were 84 written and read back.
// Triangles with a vertex at w <= 1e-6 (behind the eye) or more than 2^21
// pixels off the image are not drawn: there is no clipping.  Every float
// operation is an explicitly rounded IEEE operation (no contraction), so the
// CPU restatement in the oracle reproduces the depth/triangle buffers bit for
// bit.
#include "bcmc_impl.h"
#include "unpack.cuh"

namespace bcmc {
namespace {

struct RenderArgs {
    const uint2* verts;
    VertexStage stage;
    uint64_t ntri;
    uint32_t w, h;
    float eye[3];
    float half[3];  // the volume's box is [-half, half]
    int fog;
    unsigned long long* keys;  // per pixel
    float* rgba;               // 4 per pixel
    float* depth;              // 1 per pixel, or null
    uint32_t* triangle;        // 1 per pixel, or null
    uint32_t* big;             // triangles left to k_raster_big
    unsigned int* nbig;        // their number less one
};

// a triangle whose pixel box holds more than this many pixels, or is wider or
// higher than kBigSide, is rasterised by a whole CTA (k_raster_big) instead of
// one thread: below it the edge functions fit 32 bits
constexpr long long kBigBox = 256;
constexpr int kBigSide = 64;

// Screen positions are snapped to 1/256 pixel (the sub-pixel precision
// WebGPU's rasterisers use) and the edge functions are evaluated in 64-bit
// integers, exactly: the shared edge of two triangles gives opposite values
// in the two, so with the top-left rule every pixel centre on it is covered
// by exactly one of them (no cracks, no double coverage).
constexpr float kSub = 256.0f;          // sub-pixel steps per pixel
constexpr float kGuard = 2097152.0f;    // |screen coordinate| limit in pixels (2^21)

struct Tri {
    int x[3], y[3];   // fixed-point screen positions, positive winding
    float z[3];       // NDC depth
    int idx[3];       // which input vertex each of the three is
    long long area;   // twice the area in fixed-point units, > 0
};

__device__ __forceinline__ long long edge_fn(int ax, int ay, int bx, int by, int px, int py)
{
    return (long long)(bx - ax) * (long long)(py - ay) - (long long)(by - ay) * (long long)(px - ax);
}

// top-left rule (screen y down, positive winding): a pixel centre exactly on
// an edge belongs to the triangle when the edge is a top edge (horizontal,
// running in +x) or a left edge (running in -y)
__device__ __forceinline__ bool top_left(int ax, int ay, int bx, int by) { return (ay == by && bx > ax) || (by < ay); }

// the world and clip positions of triangle t's vertices
__device__ __forceinline__ void load_triangle(const RenderArgs& a, uint64_t t, float world[9], float clip[12])
{
    uint2 v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) v[k] = __ldg(a.verts + 3 * t + k);
    uint3 b = block_coords(v[0].y, a.stage.grid);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (k && v[k].y != v[k - 1].y) b = block_coords(v[k].y, a.stage.grid);  // a mesh's triangles lie in one block
        vertex_world(a.stage, v[k].x, b, world + 3 * k);
        vertex_clip(a.stage, world + 3 * k, clip + 4 * k);
    }
}

// false when the triangle is not drawn: a vertex at w <= 1e-6, a vertex
// beyond the guard band (or not finite), or zero area
__device__ __forceinline__ bool tri_setup(const float* c, uint32_t w, uint32_t h, Tri& t)
{
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float cw = c[4 * k + 3];
        if (!(cw > 1e-6f)) return false;
        const float nx = __fdiv_rn(c[4 * k], cw), ny = __fdiv_rn(c[4 * k + 1], cw);
        const float sx = __fmul_rn(__fadd_rn(__fmul_rn(nx, 0.5f), 0.5f), (float)w);
        const float sy = __fmul_rn(__fsub_rn(0.5f, __fmul_rn(ny, 0.5f)), (float)h);
        if (!(fabsf(sx) <= kGuard && fabsf(sy) <= kGuard)) return false;
        t.x[k] = (int)rintf(__fmul_rn(sx, kSub));
        t.y[k] = (int)rintf(__fmul_rn(sy, kSub));
        t.z[k] = __fdiv_rn(c[4 * k + 2], cw);
        t.idx[k] = k;
    }
    t.area = edge_fn(t.x[0], t.y[0], t.x[1], t.y[1], t.x[2], t.y[2]);
    if (t.area == 0) return false;
    if (t.area < 0) {  // make the winding positive
        int tmp = t.x[1]; t.x[1] = t.x[2]; t.x[2] = tmp;
        tmp = t.y[1]; t.y[1] = t.y[2]; t.y[2] = tmp;
        const float tz = t.z[1]; t.z[1] = t.z[2]; t.z[2] = tz;
        t.idx[1] = 2;
        t.idx[2] = 1;
        t.area = -t.area;
    }
    return true;
}

// floor(v / 256) for any sign
__device__ __forceinline__ int floor_div256(int v) { return v >= 0 ? v / 256 : -((255 - v) / 256); }

__device__ __forceinline__ void edges_at(const Tri& t, int px, int py, long long e[3])
{
    const int cx = px * 256 + 128, cy = py * 256 + 128;  // pixel centre
    e[0] = edge_fn(t.x[1], t.y[1], t.x[2], t.y[2], cx, cy);
    e[1] = edge_fn(t.x[2], t.y[2], t.x[0], t.y[0], cx, cy);
    e[2] = edge_fn(t.x[0], t.y[0], t.x[1], t.y[1], cx, cy);
}

// depth test of a covered pixel with edge values e: the 64-bit atomicMin of
// (depth bits, triangle index) keeps the nearest fragment, the earlier triangle
// on ties (depth >= 0, so its bits order as the values do)
__device__ __forceinline__ void put_fragment(const RenderArgs& a, const float e[3], const float tz[3], float area,
                                             float inv_area, uint32_t ti, int px, int py)
{
    // depth: NDC z interpolated linearly in screen space (the area is at least 1)
    const float num = __fadd_rn(__fadd_rn(__fmul_rn(e[0], tz[0]), __fmul_rn(e[1], tz[1])), __fmul_rn(e[2], tz[2]));
    const float z = num > 1e-20f && num < 1e30f ? exact_div(num, area, inv_area) : __fdiv_rn(num, area);
    if (!(z >= 0.0f && z < 1.0f)) return;  // outside the depth range, or not less than the clear value
    const unsigned long long key = ((unsigned long long)__float_as_uint(z) << 32) | ti;
    atomicMin(a.keys + (uint64_t)py * a.w + px, key);
}

// pixels whose centre (256 p + 128) lies in the triangle's box, clamped to the
// image: x0 > x1 or y0 > y1 when there are none
__device__ __forceinline__ int4 pixel_box(const RenderArgs& a, const Tri& t)
{
    const int xmin = min(t.x[0], min(t.x[1], t.x[2])), xmax = max(t.x[0], max(t.x[1], t.x[2]));
    const int ymin = min(t.y[0], min(t.y[1], t.y[2])), ymax = max(t.y[0], max(t.y[1], t.y[2]));
    return make_int4(max(0, floor_div256(xmin - 128 + 255)), max(0, floor_div256(ymin - 128 + 255)),
                     min((int)a.w - 1, floor_div256(xmax - 128)), min((int)a.h - 1, floor_div256(ymax - 128)));
}

// A lane of k_raster's triangle, as its fragments need it.  48 bytes: eight lanes'
// 16-byte reads at different triangles fall on different banks.
struct __align__(16) SmallTri {
    int at[3];       // the edge functions at the box's first pixel
    uint32_t d[3];   // each edge's dx and (from bit 16) dy, in sub-pixel steps
    float z[3], inv_area;
    int x, y;        // the box's first pixel
};

// A warp takes 32 triangles, one to a lane.  A small triangle's edge functions are
// exact in 32 bits (corners within 2^15 of each other and of the box's pixel
// centres), each less the top-left rule's one, so that a pixel is covered when no
// value is negative: its box is gone through once with an add per edge and pixel,
// four pixels of a row at a time.  Covered pixels are listed and take the depth
// test a lane each, whichever triangle they are of: the most that a warp's
// triangles cover is several times the mean.  With 64-bit products per pixel and
// the depth test inside the loop this took 203 us on 1.27 M triangles at 1080p,
// with each lane testing its own triangle's pixels 115 us, now 88 us.
constexpr int kRasterThreads = 256;
struct RasterWarp {
    SmallTri tri[32];
    uint32_t covered[1024];  // lane, and from bits 5 and 12 the pixel in the box; 32 of each lane at a time
};

__global__ void __launch_bounds__(kRasterThreads) k_raster(RenderArgs a)
{
    __shared__ RasterWarp s_warp[kRasterThreads / 32];
    const uint32_t lane = threadIdx.x & 31u;
    RasterWarp& s = s_warp[threadIdx.x >> 5];
    for (uint64_t t0 = blockIdx.x * (uint64_t)kRasterThreads + (threadIdx.x & ~31u); t0 < a.ntri;
         t0 += (uint64_t)gridDim.x * kRasterThreads) {
        const uint64_t ti = t0 + lane;
        int row[3] = {}, e[3] = {}, right[3] = {}, down[3] = {};
        uint32_t per_row = 1, groups = 0, last = 0;  // the box in groups of four pixels of a row
        if (ti < a.ntri) {
            float world[9], clip[12];
            load_triangle(a, ti, world, clip);
            Tri t;
            if (tri_setup(clip, a.w, a.h, t)) {
                const int4 box = pixel_box(a, t);
                const int bw = box.z - box.x + 1, bh = box.w - box.y + 1;
                if (bw <= 0 || bh <= 0) {
                } else if ((long long)bw * bh > kBigBox ||
                           max(max(t.x[0], t.x[1]), t.x[2]) - min(min(t.x[0], t.x[1]), t.x[2]) > 256 * kBigSide ||
                           max(max(t.y[0], t.y[1]), t.y[2]) - min(min(t.y[0], t.y[1]), t.y[2]) > 256 * kBigSide) {
                    a.big[atomicAdd(a.nbig, 1u) + 1u] = (uint32_t)ti;
                } else {
                    // edge k runs from corner k + 1 to corner k + 2; its value at the
                    // first pixel's centre, its steps to the right and down, and
                    // whether a centre on it is outside
                    const int cx = box.x * 256 + 128, cy = box.y * 256 + 128;
                    SmallTri r;
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const int p = (k + 1) % 3, q = (k + 2) % 3;
                        const int dx = t.x[q] - t.x[p], dy = t.y[q] - t.y[p];
                        r.at[k] = dx * (cy - t.y[p]) - dy * (cx - t.x[p]);
                        r.d[k] = (uint32_t)(dx & 0xffff) | ((uint32_t)dy << 16);
                        r.z[k] = t.z[k];
                        right[k] = -256 * dy;
                        down[k] = 256 * dx;
                        row[k] = e[k] = r.at[k] - (top_left(t.x[p], t.y[p], t.x[q], t.y[q]) ? 0 : 1);
                    }
                    r.inv_area = __frcp_rn(__ll2float_rn(t.area));
                    r.x = box.x;
                    r.y = box.y;
                    s.tri[lane] = r;
                    per_row = (uint32_t)(bw + 3) >> 2;
                    groups = per_row * (uint32_t)bh;
                    last = 15u & (15u << (4 * (int)per_row - bw));  // pixels of a row's last group, as `covered` has them
                }
            }
        }
        const uint32_t inv = (65535u + per_row) / per_row;  // g / per_row = g * inv >> 16 for g < 1024
        const uint32_t most = __reduce_max_sync(0xffffffffu, groups);
        uint32_t gx = 0;
        for (uint32_t first = 0; first < most; first += 8u) {
            uint32_t covered = 0;
            for (uint32_t i = 0; i < 8u && first + i < groups; ++i) {
                uint32_t outside = 0;  // sign bits shifted in: the group's first pixel ends at bit 3
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    outside = __funnelshift_l((uint32_t)(e[0] | e[1] | e[2]), outside, 1);
#pragma unroll
                    for (int k = 0; k < 3; ++k) e[k] += right[k];
                }
                const bool end = ++gx == per_row;
                covered |= (~outside & (end ? last : 15u)) << (4u * i);
                if (end) {
                    gx = 0;
#pragma unroll
                    for (int k = 0; k < 3; ++k) e[k] = row[k] += down[k];
                }
            }
            const uint32_t n = (uint32_t)__popc(covered), inc = warp_inclusive_scan(n);
            const uint32_t total = __shfl_sync(0xffffffffu, inc, 31);
            for (uint32_t at = inc - n; covered; ++at) {
                const uint32_t i = (uint32_t)__ffs(covered) - 1u, g = first + (i >> 2), r = g * inv >> 16;
                covered &= covered - 1u;
                s.covered[at] = lane | ((4u * (g - r * per_row) + (~i & 3u)) << 5) | (r << 12);
            }
            __syncwarp();
            for (uint32_t i = lane; i < total; i += 32u) {
                const uint32_t c = s.covered[i], px = (c >> 5) & 127u, py = c >> 12;
                const SmallTri r = s.tri[c & 31u];
                float f[3];
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    f[k] = __int2float_rn(r.at[k] + 256 * ((int)py * (int)(int16_t)(r.d[k] & 0xffffu) - (int)px * ((int)r.d[k] >> 16)));
                put_fragment(a, f, r.z, __int2float_rn(r.at[0] + r.at[1] + r.at[2]), r.inv_area, (uint32_t)t0 + (c & 31u),
                             r.x + (int)px, r.y + (int)py);
            }
            __syncwarp();
        }
    }
}

// the triangles k_raster set aside, one CTA each, its threads striding over
// the pixel box (up to 2^28 pixels).  One thread sets the triangle up, and a
// thread's pixel moves on without a division: set up by every thread, with 64-bit
// quotients per pixel, a frame of a hundred triangles across all of a 1080p image
// took 1.85 ms, now 1.27, one of 20,000 37.6, now 30.9; a mesh of 35,199 at 2560 x
// 1600 325 us, now 291.
__global__ void __launch_bounds__(256) k_raster_big(RenderArgs a)
{
    __shared__ Tri s_tri;
    const unsigned int nbig = *a.nbig + 1u;
    for (unsigned int b = blockIdx.x; b < nbig; b += gridDim.x) {
        const uint32_t ti = a.big[b];
        __syncthreads();  // the last triangle has been read
        if (threadIdx.x == 0) {
            float world[9], clip[12];
            load_triangle(a, ti, world, clip);
            tri_setup(clip, a.w, a.h, s_tri);
        }
        __syncthreads();
        const Tri t = s_tri;
        const int4 box = pixel_box(a, t);
        const uint32_t bw = box.z - box.x + 1, npix = bw * (uint32_t)(box.w - box.y + 1);
        const uint32_t down = blockDim.x / bw, right = blockDim.x - down * bw;
        uint32_t y = threadIdx.x / bw, x = threadIdx.x - y * bw;
        const float area = __ll2float_rn(t.area), inv_area = __frcp_rn(area);
        for (uint32_t p = threadIdx.x; p < npix; p += blockDim.x) {
            const int px = box.x + (int)x, py = box.y + (int)y;
            x += right;
            y += down;
            if (x >= bw) {
                x -= bw;
                ++y;
            }
            long long e[3];
            edges_at(t, px, py, e);
            const bool in0 = e[0] > 0 || (e[0] == 0 && top_left(t.x[1], t.y[1], t.x[2], t.y[2]));
            const bool in1 = e[1] > 0 || (e[1] == 0 && top_left(t.x[2], t.y[2], t.x[0], t.y[0]));
            const bool in2 = e[2] > 0 || (e[2] == 0 && top_left(t.x[0], t.y[0], t.x[1], t.y[1]));
            if (!(in0 && in1 && in2)) continue;
            const float f[3] = {__ll2float_rn(e[0]), __ll2float_rn(e[1]), __ll2float_rn(e[2])};
            put_fragment(a, f, t.z, area, inv_area, ti, px, py);
        }
    }
}

__device__ __forceinline__ float3 f3(const float* p) { return make_float3(p[0], p[1], p[2]); }
__device__ __forceinline__ float3 sub3(float3 a, float3 b)
{
    return make_float3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z));
}
__device__ __forceinline__ float dot3(float3 a, float3 b)
{
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ float3 scale3(float3 a, float s)
{
    return make_float3(__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s));
}
// GLSL's definitions: normalize(x) = x / length(x), min(x, y) = y < x ? y : x,
// max(x, y) = x < y ? y : x, clamp(x, a, b) = min(max(x, a), b)
__device__ __forceinline__ float3 norm3(float3 a)
{
    const float len = __fsqrt_rn(dot3(a, a));
    return make_float3(__fdiv_rn(a.x, len), __fdiv_rn(a.y, len), __fdiv_rn(a.z, len));
}
__device__ __forceinline__ float gmin(float x, float y) { return y < x ? y : x; }
__device__ __forceinline__ float gmax(float x, float y) { return x < y ? y : x; }
__device__ __forceinline__ float3 cross3(float3 a, float3 b)
{
    return make_float3(__fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(a.z, b.y)),
                       __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(a.x, b.z)),
                       __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float clamp01(float x) { return gmin(gmax(x, 0.0f), 1.0f); }

// mc_isosurface.vert:35-49: distance along the eye ray where it enters the
// volume's box [-scale/2, scale/2], clamped at 0
__device__ __forceinline__ float fog_enter(const RenderArgs& a, const float* world, float3 eye)
{
    const float3 d = norm3(sub3(f3(world), eye));
    const float o[3] = {eye.x, eye.y, eye.z}, dd[3] = {d.x, d.y, d.z};
    float tmin[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float inv = __frcp_rn(dd[k]);
        const float ta = __fmul_rn(__fsub_rn(-a.half[k], o[k]), inv), tb = __fmul_rn(__fsub_rn(a.half[k], o[k]), inv);
        tmin[k] = gmin(ta, tb);
    }
    return gmax(gmax(tmin[0], gmax(tmin[1], tmin[2])), 0.0f);
}

__global__ void __launch_bounds__(256) k_resolve(RenderArgs a)
{
    const uint64_t npix = (uint64_t)a.w * a.h;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < npix; i += (uint64_t)gridDim.x * blockDim.x) {
        const unsigned long long key = a.keys[i];
        float4 out = make_float4(1.0f, 1.0f, 1.0f, 1.0f);  // clearValue (js/bcmc.js:179)
        float depth = 1.0f;
        uint32_t tri = 0xffffffffu;
        if (key != ~0ull) {
            const uint64_t t = key & 0xffffffffull;
            tri = (uint32_t)t;
            depth = __uint_as_float((uint32_t)(key >> 32));
            float world[9], clip[12];
            load_triangle(a, t, world, clip);
            Tri tr;
            tri_setup(clip, a.w, a.h, tr);  // drawn, so set up as in k_raster
            long long ee[3];
            edges_at(tr, (int)(i % a.w), (int)(i / a.w), ee);
            const float3 eye = make_float3(a.eye[0], a.eye[1], a.eye[2]);
            // perspective-correct weights of the varyings: (e_k / w_k) / sum.  The
            // edges come in the winding's order: corners 1 and 2 may be exchanged
            const bool flip = tr.idx[1] == 2;
            float pw[3], psum = 0.0f;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float cw = k == 0 ? clip[3] : ((k == 1) != flip ? clip[7] : clip[11]);
                pw[k] = __fdiv_rn(__ll2float_rn(ee[k]), cw);
                psum = __fadd_rn(psum, pw[k]);
            }
            float3 wp = make_float3(0.0f, 0.0f, 0.0f);
            float te = 0.0f;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float b = __fdiv_rn(pw[k], psum);
                float wk[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) wk[c] = k == 0 ? world[c] : ((k == 1) != flip ? world[3 + c] : world[6 + c]);
                wp = make_float3(__fadd_rn(wp.x, __fmul_rn(b, wk[0])), __fadd_rn(wp.y, __fmul_rn(b, wk[1])),
                                 __fadd_rn(wp.z, __fmul_rn(b, wk[2])));
                if (a.fog) te = __fadd_rn(te, __fmul_rn(b, fog_enter(a, wk, eye)));
            }
            // mc_isosurface.frag:15-40
            float3 v = sub3(wp, eye);
            const float dist = __fsqrt_rn(dot3(v, v));
            v = scale3(norm3(v), -1.0f);
            const float3 light = v;
            float3 n = norm3(cross3(sub3(f3(world + 3), f3(world)), sub3(f3(world + 6), f3(world))));
            if (dot3(n, light) < 0.0f) n = scale3(n, -1.0f);
            const float3 base = make_float3(0.3f, 0.3f, 0.9f);
            const float3 hv = norm3(make_float3(__fadd_rn(v.x, light.x), __fadd_rn(v.y, light.y), __fadd_rn(v.z, light.z)));
            const float diff = __fmul_rn(0.6f, clamp01(dot3(light, n)));
            const float sp = clamp01(dot3(n, hv));
            const float sp2 = __fmul_rn(sp, sp);
            const float spec = __fmul_rn(0.1f, powf(sp, 5.0f));
            float3 col = make_float3(__fadd_rn(__fadd_rn(__fmul_rn(base.x, 0.2f), __fmul_rn(diff, base.x)), spec),
                                     __fadd_rn(__fadd_rn(__fmul_rn(base.y, 0.2f), __fmul_rn(diff, base.y)), spec),
                                     __fadd_rn(__fadd_rn(__fmul_rn(base.z, 0.2f), __fmul_rn(diff, base.z)), spec));
            if (a.fog) {
                const float fog = expf(__fmul_rn(-1.0f, gmax(__fsub_rn(dist, __fadd_rn(te, 0.1f)), 0.0f)));
                const float rest = __fsub_rn(1.0f, fog);
                col = make_float3(__fadd_rn(__fmul_rn(fog, col.x), rest), __fadd_rn(__fmul_rn(fog, col.y), rest),
                                  __fadd_rn(__fmul_rn(fog, col.z), rest));
            }
            out = make_float4(col.x, col.y, col.z, 1.0f);
        }
        reinterpret_cast<float4*>(a.rgba)[i] = out;
        if (a.depth) a.depth[i] = depth;
        if (a.triangle) a.triangle[i] = tri;
    }
}

int grid_of(bcmc_ctx* ctx, uint64_t n)
{
    const uint64_t want = (n + 255) / 256, cap = (uint64_t)ctx->num_sms * 16;
    return (int)(want == 0 ? 1 : (want < cap ? want : cap));
}

}  // namespace

void render_launch(bcmc_ctx* ctx, const uint2* verts, uint64_t n, const uint32_t dims[3], const float scale[3],
                   const bcmc_render_params& p, float* rgba, float* depth, uint32_t* triangle, cudaStream_t s)
{
    const uint64_t ntri = n / 3, npix = (uint64_t)p.width * p.height;
    // working buffers, carved from one grow-only context allocation: the
    // per-pixel keys, the list of large triangles and its counter
    const uint64_t b_keys = (npix * 8 + 255) & ~uint64_t(255), need = b_keys + (ntri + 1) * 4;
    if (need > ctx->render_bytes) {
        dev_free(ctx, ctx->d_render, ctx->render_bytes);
        ctx->d_render = nullptr;
        ctx->render_bytes = 0;
        ctx->d_render = dev_alloc(ctx, need);
        ctx->render_bytes = need;
    }
    unsigned long long* keys = static_cast<unsigned long long*>(ctx->d_render);
    uint32_t* big = reinterpret_cast<uint32_t*>(static_cast<char*>(ctx->d_render) + b_keys);
    try {
        BCMC_CUDA(cudaMemsetAsync(keys, 0xff, b_keys + 4, s));  // the keys, and the counter at -1
        RenderArgs a{};
        a.verts = verts;
        a.stage = make_vertex_stage(dims, scale, p.proj_view);
        a.ntri = ntri;
        a.w = p.width;
        a.h = p.height;
        for (int k = 0; k < 3; ++k) {
            a.eye[k] = p.eye_pos[k];
            a.half[k] = (scale ? scale[k] : 1.0f) * 0.5f;
        }
        a.fog = p.fog ? 1 : 0;
        a.keys = keys;
        a.rgba = rgba;
        a.depth = depth;
        a.triangle = triangle;
        a.nbig = big;
        a.big = big + 1;
        if (ntri) {
            k_raster<<<grid_of(ctx, ntri), kRasterThreads, 0, s>>>(a);
            k_raster_big<<<ctx->num_sms * 4, 256, 0, s>>>(a);
            count_launches(2);
        }
        k_resolve<<<grid_of(ctx, npix), 256, 0, s>>>(a);
        count_launches(1);
        BCMC_CUDA(cudaGetLastError());
        BCMC_CUDA(cudaStreamSynchronize(s));  // the working buffers are free again when this returns
    } catch (...) {
        cudaStreamSynchronize(s);
        throw;
    }
}

}  // namespace bcmc
