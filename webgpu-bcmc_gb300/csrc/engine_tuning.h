// engine_tuning.h -- the batched engine's launch parameters and which of them its
// autotuner times.  Free of the CUDA runtime, so that a host build of it can be
// checked.
#pragma once

#include <algorithm>
#include <vector>

namespace bcmc {

constexpr int kBmcPerSm = 6;  // k_bmc CTAs per SM that a configuration may ask for at 16 blocks

// Launch parameters the autotuner chooses per batch-size bucket (the kernels'
// tile shapes are compile-time; these are the runtime knobs).
struct EngConfig {
    int act_per_sm = 8;      // k_bactive and k_bentries CTAs per SM
    int dec_threads = 128;   // k_bdecode threads per CTA (64, 128, 256)
    int dec_per_sm = 16;     // k_bdecode CTAs per SM
    int mc_per_sm = kBmcPerSm;  // k_bmc CTAs per SM at 16 blocks (4, 5, 6), scaled by 16 / mc_blocks at
                                // the other sizes, and no more than fit (mc_ctas)
    int mc_blocks = 32;         // k_bmc "tile blocks", 16 threads each (8, 16, 32)
};

// The k_bmc CTAs per SM that a configuration gets where `resident` fit.
inline int mc_ctas(const EngConfig& c, int resident)
{
    return std::max(1, std::min(std::min(c.mc_per_sm, kBmcPerSm) * 16 / c.mc_blocks, resident));
}

// `c` with each other CTA size of k_bmc.
inline std::vector<EngConfig> other_mc_sizes(const EngConfig& c)
{
    std::vector<EngConfig> r;
    for (int blocks : {8, 16, 32})
        if (blocks != c.mc_blocks) {
            r.push_back(c);
            r.back().mc_blocks = blocks;
        }
    return r;
}

// `c` with fewer k_bmc CTAs per SM: one configuration for each grid that 5 and 4
// give where `resident` CTAs fit.  None, today: six, four and two CTAs of 8, 16 and
// 32 blocks fit, and 4 asks for no fewer.
inline std::vector<EngConfig> other_mc_ctas(const EngConfig& c, int resident)
{
    std::vector<EngConfig> r;
    int last = mc_ctas(c, resident);
    for (int per_sm : {5, 4}) {
        EngConfig d = c;
        d.mc_per_sm = per_sm;
        if (mc_ctas(d, resident) == last) continue;
        last = mc_ctas(d, resident);
        r.push_back(d);
    }
    return r;
}

}  // namespace bcmc
