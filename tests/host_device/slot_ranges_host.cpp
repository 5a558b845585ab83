// The share-out of the LRU's slots (csrc/slot_ranges.cuh) as host code.
#include "cuda_host_shim.h"
#include "slot_ranges.cuh"

// 0 when the CTAs that publish a count are ranks 0 .. k - 1, all with a status
// word, and their ranges are the slots, one after the other; else what is wrong.
extern "C" int check_ranges(uint32_t slots, uint32_t ctas)
{
    uint32_t at = 0;
    bool ended = false;
    for (uint32_t rank = 0; rank < ctas; ++rank) {
        const bcmc::SlotRange r = bcmc::slot_range(slots, ctas, rank);
        if (!r.any()) {
            ended = true;
            continue;
        }
        if (ended) return 1;
        if (rank >= bcmc::slot_tiles(slots)) return 2;
        if (r.first != at || r.end > slots) return 3;
        at = r.end;
    }
    return at == slots ? 0 : 4;
}
