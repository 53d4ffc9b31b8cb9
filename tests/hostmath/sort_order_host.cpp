// Host build of the check and the exchange by which a sort tile puts right what its ranks left out of order (the
// header compiles as plain C++).  The threads of a phase run one after the other, in the order asked for.
#include "../../pointtransformerv3_b200/csrc/sort_order.cuh"

using namespace ptv3;

// whether any thread finds a neighbour out of order as the tile is written
extern "C" int host_out_of_order(const uint64_t* words, int count, int shift, uint32_t mask)
{
    const OsOrder o{shift, mask};
    bool bad = false;
    for (int i = 1; i < count; ++i) bad |= os_wrong(o, words[i - 1], words[i]);
    return bad;
}

// the kernel's loop; rounds that it took, or -1 where they did not suffice
extern "C" int host_put_right(uint64_t* words, int count, int shift, uint32_t mask, int threads, int backwards)
{
    const OsOrder o{shift, mask};
    for (int round = 0; round < os_rounds(count); ++round) {
        bool bad = false;
        for (int odd = 0; odd < 2; ++odd)
            for (int t = 0; t < threads; ++t)
                bad |= os_exchange(o, words, count, odd, backwards ? threads - 1 - t : t, threads);
        if (!bad) return round;
    }
    return host_out_of_order(words, count, shift, mask) ? -1 : os_rounds(count);
}
