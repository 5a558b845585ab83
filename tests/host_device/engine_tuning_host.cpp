// The autotuner's candidates (csrc/engine_tuning.h) as host code.
#include "engine_tuning.h"

static int put(const std::vector<bcmc::EngConfig>& v, int (*of)(const bcmc::EngConfig&), int* out)
{
    int n = 0;
    for (const auto& c : v) out[n++] = of(c);
    return n;
}

extern "C" int default_size() { return bcmc::EngConfig{}.mc_blocks; }
extern "C" int sizes(int mc_blocks, int* out)
{
    bcmc::EngConfig c;
    c.mc_blocks = mc_blocks;
    return put(bcmc::other_mc_sizes(c), [](const bcmc::EngConfig& x) { return x.mc_blocks; }, out);
}
extern "C" int per_sm(int mc_blocks, int resident, int* out)
{
    bcmc::EngConfig c;
    c.mc_blocks = mc_blocks;
    return put(bcmc::other_mc_ctas(c, resident), [](const bcmc::EngConfig& x) { return x.mc_per_sm; }, out);
}
extern "C" int ctas(int mc_blocks, int mc_per_sm, int resident)
{
    bcmc::EngConfig c;
    c.mc_blocks = mc_blocks;
    c.mc_per_sm = mc_per_sm;
    return bcmc::mc_ctas(c, resident);
}
