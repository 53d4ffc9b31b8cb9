// The order among a tile's elements of one digit, and how a tile that is out of it is put right (sort.cu).  Plain
// integer code, usable from device code and (for the tests) from host code.
#pragma once
#include <stdint.h>
#ifndef PTV3_HD
#if defined(__CUDACC__)
#define PTV3_HD __host__ __device__ __forceinline__
#else
#define PTV3_HD static inline
#endif
#endif

namespace ptv3 {

// A packed word holds its digit at `shift` and, below it, everything that the order among equal digits goes by: the
// digits done, and the index.
struct OsOrder {
    int shift;
    uint32_t mask;       // of the digit
};

// whether neighbours x, y of an ordered tile are of one digit and the wrong way round
PTV3_HD bool os_wrong(const OsOrder& o, uint64_t x, uint64_t y)
{
    const uint64_t below = (1ull << o.shift) - 1ull;
    return (((x ^ y) >> o.shift) & o.mask) == 0 && (x & below) > (y & below);
}

// A thread's share of one phase of an odd-even exchange of neighbours, the pairs from `odd` (0 or 1) on: the pairs of a
// phase do not overlap, so its threads need no order; a barrier follows it.  True: it exchanged some.
PTV3_HD bool os_exchange(const OsOrder& o, uint64_t* words, int count, int odd, int thread, int threads)
{
    bool any = false;
    for (int i = 2 * thread + 1 + odd; i < count; i += 2 * threads) {
        const uint64_t x = words[i - 1], y = words[i];
        if (os_wrong(o, x, y)) {
            words[i - 1] = y;
            words[i] = x;
            any = true;
        }
    }
    return any;
}

// rounds of two phases after which any disorder is gone (an odd-even exchange sorts n elements in n phases)
PTV3_HD int os_rounds(int count) { return count / 2 + 1; }

}  // namespace ptv3
