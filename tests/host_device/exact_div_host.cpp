// exact_div (exact_div.cuh) as host code, for every packed position along an
// axis of `dim` voxels: the count of quotients that differ from a / b.
#include "cuda_host_shim.h"
#include "exact_div.cuh"

extern "C" uint64_t differing(uint32_t dim)
{
    const float b = (float)dim, inv = 1.0f / b;
    uint64_t bad = 0;
    for (uint32_t q = 0; q < 1024; ++q) {
        volatile float n = (float)q * 4.0f;
        volatile float d = n / 1023.0f;
        if (bcmc::exact_div(n, 1023.0f, 1.0f / 1023.0f) != d) ++bad;
        volatile float p = d + 0.5f;
        const uint32_t blocks = (dim + 3) / 4, step = blocks > 4096 ? blocks / 1024 : 1;
        for (uint32_t i = 0; i < blocks; i += step) {
            volatile float a = 4.0f * (float)i + p;
            volatile float want = a / b;
            if (bcmc::exact_div(a, b, inv) != want) ++bad;
        }
    }
    return bad;
}
