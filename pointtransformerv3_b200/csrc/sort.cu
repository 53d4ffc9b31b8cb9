// Stable LSD radix argsort of k rows of n non-negative int64 codes, restricted
// to the significant low bits, with the inverse permutation written by the last
// pass.  Replaces torch.argsort + scatter_ at model.py:118-126 and :667-674
// (ties are resolved by original index, the canonical order).
//
// One-sweep form (Adinets and Merrill, "Onesweep: A Faster Least Significant Digit Radix Sort for GPUs",
// 2022; the look-back is Merrill and Garland's, 2016): one kernel reads every key once and builds the digit
// histograms of ALL passes; after that every pass is a single kernel.  A tile of
// a pass ranks its keys by digit in shared memory, publishes its per-digit counts
// in a status table and obtains its global offsets by looking back over the
// status words of the tiles before it (decoupled look-back), so a pass reads and
// writes every element exactly once.  Digits are up to 10 bits wide and spread
// evenly over the significant bits (29 bits -> 3 passes, 49 bits -> 5 passes).
//
// Between passes an element is ONE 64-bit word, its key above its index, where the significant bits
// and the bits of an index fit (37 + 23 at 8 M points): 8 bytes in and 8 out instead of 12 and 12, one
// shared-memory access instead of two, and runs of equal digits that fill sectors.  Longer keys travel
// beside their indices until enough of their digits are done.
// The first pass reads the caller's codes; the last one writes order / inverse as int64.
//
// Bytes per element: 8 (histograms) + 16 per pass + 8 in the last one.  What bounds a pass is a
// tile's chain of short phases separated by barriers, two tiles per SM, most of each phase scattered accesses to
// shared memory.  Of the 26 000 cycles of a tile of 8 192 with 512 bins: 1 700 until it has its number, 4 200 its loads,
// 4 400 counting, 3 500 the scan over warps and digits, 3 900 putting its elements in order, 2 800 the look-back, 4 300
// writing.  32 M elements take ~185 us a pass against 79 for the bytes (270 with ranks from masks, see below).
// The last pass adds ~350 us to that for the scattered 8-byte inverses, the rate at which L2 takes single sectors (the
// same in a kernel of its own; 25 us more without the hint that keeps them there).
// 8 M x 4 rows: 37 bits 1 548 -> 1 362 us, 36 bits (a single scene has no scene number) 1 383 -> 1 195; 1 M x 4 of 34
// bits 214 -> 164; 100 000 x 4 of 27 bits 47.  Measured and dropped: CTAs of 256 threads, four to an SM (1 367).
//
// Tiles take their number from a counter when they start, so every tile a tile
// waits for is already running or finished; all the same every wait is bounded
// and a wait that runs out sets PTV3_STATUS_WAIT_LIMIT.
#include "common.cuh"
#include "sort_order.cuh"
#include "../../include/ptv3_b200.h"

namespace ptv3 {

constexpr int OS_THREADS = 512;
constexpr int OS_WARPS = OS_THREADS / 32;
constexpr int OS_MAX_BITS = 10;
constexpr int OS_MAX_BINS = 1 << OS_MAX_BITS;
constexpr int OS_DPT = OS_MAX_BINS / OS_THREADS;  // digits a thread looks after
constexpr int OS_MAX_PASSES = 7;                  // 63 bits / 10 -> 7
constexpr uint32_t OS_COUNT_MASK = (1u << 28) - 1u;
constexpr uint32_t OS_SPIN_LIMIT = 1u << 20;
constexpr int64_t OS_L2_BYTES = (int64_t)96 << 20;   // of the 126 MB, what streams leave to be kept
constexpr int OS_WINDOW = 8;                     // earlier tiles inspected per round trip

struct SortPlan {
    int passes;
    int bits;      // digit width of every pass but possibly the last
    int val_bits;  // of an index
    int wide;      // passes whose elements are held as a key with its index beside it
    int items;     // per thread of a pass
    int ntiles;
    size_t bytes;
};

// Digit histograms of every pass in one read of the keys: hist[row][pass][digit].
// Four keys of a thread are under way at once: one at a time, a block waited for memory between its shared-memory
// atomics (8 M x 4 rows, 36 bits: 1 220 -> 1 195 us for the sort; eight keys, or a quarter of the blocks: the same).
constexpr int OS_HIST_KEYS = 4;
__global__ void __launch_bounds__(OS_THREADS) os_hist_kernel(const uint64_t* __restrict__ keys, int64_t n,
                                                            int sig_bits, int bits, int passes,
                                                            uint32_t* __restrict__ hist)
{
    extern __shared__ uint32_t os_smem[];      // [passes][OS_MAX_BINS]
    const int row = blockIdx.y;
    for (int i = threadIdx.x; i < passes * OS_MAX_BINS; i += OS_THREADS) os_smem[i] = 0;
    __syncthreads();
    const uint64_t* k = keys + (int64_t)row * n;
    const uint32_t mask = (1u << bits) - 1u;
    const int64_t stride = (int64_t)gridDim.x * OS_THREADS;
    for (int64_t idx = (int64_t)blockIdx.x * OS_THREADS + threadIdx.x; idx < n; idx += OS_HIST_KEYS * stride) {
        uint64_t key[OS_HIST_KEYS];
#pragma unroll
        for (int q = 0; q < OS_HIST_KEYS; ++q) key[q] = idx + q * stride < n ? k[idx + q * stride] : 0;
#pragma unroll
        for (int q = 0; q < OS_HIST_KEYS; ++q) {
            if (idx + q * stride >= n) break;
            for (int p = 0; p < passes; ++p)
                atomicAdd(&os_smem[p * OS_MAX_BINS + ((uint32_t)(key[q] >> (p * bits)) & mask)], 1u);
        }
    }
    __syncthreads();
    uint32_t* out = hist + (size_t)row * OS_MAX_PASSES * OS_MAX_BINS;
    for (int i = threadIdx.x; i < passes * OS_MAX_BINS; i += OS_THREADS) {
        const uint32_t c = os_smem[i];
        if (c) atomicAdd(&out[i], c);
    }
}

// exclusive scan over the block of one value per thread (two 32-bit sums packed in 64 bits)
__device__ __forceinline__ uint64_t os_block_excl_scan(uint64_t v, uint64_t* warp_sums)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t u = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += u;
    }
    if (lane == 31) warp_sums[warp] = inc;
    __syncthreads();
    uint64_t base = 0;
#pragma unroll
    for (int w = 0; w < OS_WARPS; ++w)
        if (w < warp) base += warp_sums[w];
    return base + inc - v;
}

// a store that L2 keeps rather than what streams past it
__device__ __forceinline__ void store_kept(int64_t* p, int64_t v)
{
    uint64_t policy;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(policy));
    asm volatile("st.global.L2::cache_hint.b64 [%0], %1, %2;" ::"l"(p), "l"(v), "l"(policy) : "memory");
}

// How elements enter and leave a pass: as the caller's codes, as packed words, as keys with their
// indices beside them, as the final order
enum { OS_PACKED = 0, OS_WIDE = 1, OS_FINAL = 2 };

struct OsPass {
    const uint64_t* in;      // RAW codes, packed words or keys
    const int32_t* vals_in;  // indices beside wide keys (nullptr: an element's index is its place)
    uint64_t* out;
    int32_t* vals_out;
    int64_t *order, *inverse;
    const uint32_t* hist;
    uint32_t *tile_status, *tile_counter, *status;
    int64_t n;
    int raw;                 // PACKED: `in` holds codes, the pass packs them
    int shift, bits;         // of the pass's digit in the key
    int val_bits;            // of an index inside a packed word
    int pass, ntiles, rows;
    int by_row;              // tiles in row-after-row order
};

// shared memory of a tile's elements (or of the masks that rank them)
__host__ __device__ constexpr size_t os_element_bytes(int items, int bins, bool wide, bool masks)
{
    const size_t elements = (size_t)OS_THREADS * items * (wide ? 12 : 8), words = masks ? (size_t)OS_WARPS * bins * 4 : 0;
    return elements > words ? elements : words;
}

// One pass over one tile of 512 * ITEMS elements.  Element order inside a tile is warp-major: warp w owns
// [w * 32 * ITEMS, (w + 1) * 32 * ITEMS), visited 32 consecutive elements at a time, so that
// (warp, item, lane) order is index order and ranks taken in that order are stable.
//
// Order of the steps: counts first (a histogram with shared-memory atomics) and their
// publication; then the ranking and the reordering in shared memory; the look-back last.  By
// then the tiles before this one, which started earlier, have mostly finished their own
// look-back, so the walk finds an inclusive prefix after one or two tiles.  (With the look-back
// first, a tile meets hundreds of tiles in the "counts only" state; that walk then takes longer
// than everything else and keeps itself long.)
//
// Ranks among the equal digits of a warp: the counters that the histogram adds to hand them out (atomicAdd
// returns the count so far).  That is the order of the elements except among lanes of one instruction with the same digit,
// whose order of service nobody promises.  But a packed word holds everything that the order among equal
// digits goes by, so neighbours in the ordered tile are compared as they are written, and exchanged until none is out
// of order (sort_order.cuh; on this hardware none has been seen, so the tests run it on the host).
// MASKS: sorts that dropped digits on the way (see `wide`) cannot tell; their ranks come from masks of the lanes with
// the same digit, one shared-memory word per warp and digit, which cost five accesses per element: of the 33 000 cycles
// of a tile of 8 192 that form spent 11 700 there (8 M x 4 rows of 36 bits: 1 383 us, 1 296 with ranks from the counters).
//
// WIDE: keys of 64 bits with indices beside them; else packed words.  OUT: see above.
template <int OS_ITEMS, bool WIDE, int OUT, bool MASKS>
__global__ void __launch_bounds__(OS_THREADS, 2) os_pass_kernel(const OsPass a)
{
    static_assert(MASKS || !WIDE, "the check reads packed words");
    extern __shared__ __align__(16) unsigned char os_raw[];
    constexpr int OS_TILE = OS_THREADS * OS_ITEMS;
    const int bins = 1 << a.bits;
    uint32_t* peer_masks = reinterpret_cast<uint32_t*>(os_raw);                  // [OS_WARPS][bins], until ranked
    uint64_t* skeys = reinterpret_cast<uint64_t*>(os_raw);                       // [OS_TILE], then
    int32_t* svals = reinterpret_cast<int32_t*>(skeys + OS_TILE);                // [WIDE ? OS_TILE : 0]
    uint16_t* whist = reinterpret_cast<uint16_t*>(os_raw + os_element_bytes(OS_ITEMS, bins, WIDE, MASKS));    // [OS_WARPS][bins]
    uint32_t* local_off = reinterpret_cast<uint32_t*>(whist + OS_WARPS * bins);  // [bins + 1]
    uint32_t* gbase = local_off + bins + 1;                                      // [bins]
    __shared__ uint64_t warp_sums[OS_WARPS];
    __shared__ uint32_t tile_s;
    __shared__ int give_up;

    const int row = a.by_row ? blockIdx.x / a.ntiles : blockIdx.x % a.rows;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t mask = (uint32_t)bins - 1u;
    if (threadIdx.x == 0) {
        tile_s = atomicAdd(&a.tile_counter[a.pass * a.rows + row], 1u);
        give_up = 0;
    }
    // (bins >= 2: the 16-bit counters are cleared and counted in pairs)
    for (int i = threadIdx.x; i < OS_WARPS * bins / 2; i += OS_THREADS) reinterpret_cast<uint32_t*>(whist)[i] = 0;
    if (MASKS)
        for (int i = threadIdx.x; i < OS_WARPS * bins; i += OS_THREADS) peer_masks[i] = 0;
    __syncthreads();
    const int tile = (int)tile_s;
    if (tile >= a.ntiles) return;    // cannot happen with a grid of ntiles blocks per row

    // (asked for now, wanted for the scan)
    uint2 ghist = make_uint2(0u, 0u);
    if (threadIdx.x * 2 < bins)
        ghist = reinterpret_cast<const uint2*>(a.hist + ((size_t)row * OS_MAX_PASSES + a.pass) * OS_MAX_BINS)[threadIdx.x];
    const int64_t rbase = (int64_t)row * a.n;
    const int64_t tbase = (int64_t)tile * OS_TILE;
    const int tile_count = (int)min((int64_t)OS_TILE, a.n - tbase);
    const int wlo = warp * (32 * OS_ITEMS) + lane;       // this lane's first element inside the tile
    // place of the pass's digit inside an element as it is held here
    const int shift = a.shift + (WIDE ? 0 : a.val_bits);

    // ---- load; count the digits per warp ------------------------------------------------------
    uint64_t key[OS_ITEMS];
    int32_t val[WIDE ? OS_ITEMS : 1];
    uint16_t pos[OS_ITEMS];              // place in the ordered tile; first the rank inside the warp
    uint16_t* wh = whist + warp * bins;
    {
        const uint64_t* in = a.in + rbase + tbase;
#pragma unroll
        for (int it = 0; it < OS_ITEMS; ++it) {
            const int i = wlo + it * 32;
            key[it] = i < tile_count ? in[i] : 0ull;
            if constexpr (WIDE)
                val[it] = !a.vals_in ? (int32_t)(tbase + i) : i < tile_count ? a.vals_in[rbase + tbase + i] : 0;
        }
        if (!WIDE && a.raw) {
#pragma unroll
            for (int it = 0; it < OS_ITEMS; ++it)
                key[it] = (key[it] << a.val_bits) | (uint64_t)(tbase + wlo + it * 32);
        }
        // a warp holds 512 elements, so two 16-bit counters share a word without carries
        uint32_t* wh32 = reinterpret_cast<uint32_t*>(wh);
#pragma unroll
        for (int it = 0; it < OS_ITEMS; ++it) {
            if (wlo + it * 32 < tile_count) {
                const uint32_t d = (uint32_t)(key[it] >> shift) & mask;
                const uint32_t old = atomicAdd(&wh32[d >> 1], (d & 1u) ? 0x10000u : 1u);
                pos[it] = (uint16_t)((d & 1u) ? old >> 16 : old);
            }
        }
    }
    __syncthreads();

    // ---- per digit: offsets of the warps and of the digit inside the tile -----------------------
    // For the scans thread t owns the digits 2 t and 2 t + 1, whose counters are one word; for the
    // status table (below) it owns t and t + 512, so that a warp's status reads and writes are
    // contiguous in memory.  The two views meet in shared memory.
    uint32_t* st_row = a.tile_status + ((size_t)row * a.ntiles) * OS_MAX_BINS;
    const uint32_t code_agg = (uint32_t)(2 * a.pass + 1) << 28, code_inc = (uint32_t)(2 * a.pass + 2) << 28;
    {
        const bool mine = threadIdx.x * 2 < bins;
        uint32_t* column = reinterpret_cast<uint32_t*>(whist) + threadIdx.x;
        uint32_t total = 0;            // both digits' counts, at most 8192 each
        const uint2 g = ghist;
        if (mine) {
#pragma unroll
            for (int w = 0; w < OS_WARPS; ++w) total += column[w * (bins >> 1)];
        }
        const uint32_t lo = total & 0xffffu, hi = total >> 16;
        // exclusive prefixes over the digits: of the tile's counts (low word) and of the global
        // histogram (high word: start of every digit's range in the output)
        const uint64_t both = os_block_excl_scan(((uint64_t)(g.x + g.y) << 32) | (lo + hi), warp_sums);
        const uint32_t excl = (uint32_t)both, gexcl = (uint32_t)(both >> 32);
        if (mine) {
            local_off[2 * threadIdx.x] = excl;
            local_off[2 * threadIdx.x + 1] = excl + lo;
            gbase[2 * threadIdx.x] = gexcl - excl;            // the look-back adds the earlier tiles' counts
            gbase[2 * threadIdx.x + 1] = gexcl + g.x - (excl + lo);
            uint32_t run = excl | ((excl + lo) << 16);
#pragma unroll
            for (int w = 0; w < OS_WARPS; ++w) {
                const uint32_t c = column[w * (bins >> 1)];
                column[w * (bins >> 1)] = run;
                run += c;
            }
        }
        if (threadIdx.x == 0) local_off[bins] = (uint32_t)tile_count;
    }
    __syncthreads();

    // ---- publish the tile's counts (the first tile's counts are inclusive prefixes already) ----
    uint32_t cnt[OS_DPT], look[OS_DPT];
#pragma unroll
    for (int j = 0; j < OS_DPT; ++j) {
        const int d = j * OS_THREADS + threadIdx.x;
        cnt[j] = look[j] = 0;
        if (d < bins) {
            cnt[j] = local_off[d + 1] - local_off[d];
            *reinterpret_cast<volatile uint32_t*>(&st_row[(size_t)tile * OS_MAX_BINS + d]) =
                (tile == 0 ? code_inc : code_agg) | cnt[j];
        }
    }

    // ---- rank inside the warp, then order the tile by digit in shared memory ------------------------
    // An element's place is its warp's running offset of the digit plus its rank among the equal digits
    // of the 32.  The lanes of a digit find each other in a word per digit and warp into which each sets its
    // bit (a ballot per digit bit, the form before, cost 10 ballots and 140 cycles per 32 elements of a scheduler's
    // time; match.any about a thousand); the lowest moves the offset on and clears the word.
    if constexpr (MASKS) {
        const uint32_t lt = (1u << lane) - 1u;
        uint32_t* masks = peer_masks + warp * bins;
#pragma unroll
        for (int it = 0; it < OS_ITEMS; ++it) {
            const bool valid = wlo + it * 32 < tile_count;
            const uint32_t d = (uint32_t)(key[it] >> shift) & mask;
            volatile uint32_t* group = masks + d;
            volatile uint16_t* off = wh + d;
            if (valid) atomicOr(masks + d, 1u << lane);
            __syncwarp();
            const uint32_t peers = *group, before = peers & lt, base = *off;
            pos[it] = (uint16_t)(base + __popc(before));
            __syncwarp();
            if (valid && before == 0) {
                *group = 0u;
                *off = (uint16_t)(base + __popc(peers));
            }
            __syncwarp();
        }
        __syncthreads();       // the masks make room for the elements
    } else {
#pragma unroll
        for (int it = 0; it < OS_ITEMS; ++it)
            if (wlo + it * 32 < tile_count) pos[it] += wh[(uint32_t)(key[it] >> shift) & mask];
    }
#pragma unroll
    for (int it = 0; it < OS_ITEMS; ++it) {
        if (wlo + it * 32 < tile_count) {
            skeys[pos[it]] = key[it];
            if constexpr (WIDE) svals[pos[it]] = val[it];
        }
    }
    // ---- look back over the earlier tiles: all of this thread's digits at once, and a window of
    //      tiles per digit and round trip (the loads of a window do not depend on each other)
    if (tile > 0) {
        int back[OS_DPT];
        bool done[OS_DPT];
#pragma unroll
        for (int j = 0; j < OS_DPT; ++j) {
            back[j] = tile - 1;
            done[j] = j * OS_THREADS + threadIdx.x >= bins;
        }
        uint32_t spins = 0;
        bool all = false;
        while (!all) {
            uint32_t s[OS_DPT][OS_WINDOW];
#pragma unroll
            for (int j = 0; j < OS_DPT; ++j) {
                const int d = j * OS_THREADS + threadIdx.x;
#pragma unroll
                for (int q = 0; q < OS_WINDOW; ++q) {
                    const int tb = back[j] - q;
                    s[j][q] = code_inc;      // before the first tile: an inclusive prefix of zero
                    if (!done[j] && tb >= 0)
                        s[j][q] = *reinterpret_cast<volatile uint32_t*>(&st_row[(size_t)tb * OS_MAX_BINS + d]);
                }
            }
            all = true;
#pragma unroll
            for (int j = 0; j < OS_DPT; ++j) {
                if (done[j]) continue;
                bool stop = false;
#pragma unroll
                for (int q = 0; q < OS_WINDOW; ++q) {
                    const uint32_t code = s[j][q] & ~OS_COUNT_MASK;
                    if (stop || done[j]) continue;
                    if (code == code_inc) {
                        look[j] += s[j][q] & OS_COUNT_MASK;
                        done[j] = true;
                    } else if (code == code_agg) {
                        look[j] += s[j][q] & OS_COUNT_MASK;
                        --back[j];
                    } else {
                        stop = true;        // not published yet: ask again from this tile on
                    }
                }
                if (!done[j]) all = false;
            }
            if (!all && (++spins > OS_SPIN_LIMIT || *reinterpret_cast<volatile int*>(&give_up))) {
                give_up = 1;
                break;
            }
        }
    }
    // publish the inclusive prefixes; global offset of the tile's share of every digit
#pragma unroll
    for (int j = 0; j < OS_DPT; ++j) {
        const int d = j * OS_THREADS + threadIdx.x;
        if (d < bins) {
            if (tile > 0)
                *reinterpret_cast<volatile uint32_t*>(&st_row[(size_t)tile * OS_MAX_BINS + d]) =
                    code_inc | ((look[j] + cnt[j]) & OS_COUNT_MASK);
            gbase[d] += look[j];
        }
    }
    __syncthreads();
    if (give_up) {
        if (threadIdx.x == 0 && a.status) atomicOr(a.status, PTV3_STATUS_WAIT_LIMIT);
        return;
    }
    // ---- write out: neighbours in shared memory with the same digit are neighbours in global
    const OsOrder in_digit{shift, mask};
    auto write = [&] {
        bool bad = false;
#pragma unroll 4
        for (int i = threadIdx.x; i < tile_count; i += OS_THREADS) {
            const uint64_t kx = skeys[i];
            if (!MASKS && i > 0) bad |= os_wrong(in_digit, skeys[i - 1], kx);
            const int64_t dst = rbase + (uint32_t)(gbase[(uint32_t)(kx >> shift) & mask] + (uint32_t)i);
            if constexpr (OUT == OS_FINAL) {
                const int64_t v = (int64_t)(kx & ((1ull << a.val_bits) - 1ull));
                __stcs(&a.order[dst], v);       // (streams past the inverses that L2 collects)
                store_kept(&a.inverse[rbase + v], dst - rbase);
            } else if constexpr (WIDE) {
                const int32_t v = svals[i];
                if (OUT == OS_WIDE) {
                    a.out[dst] = kx;
                    a.vals_out[dst] = v;
                } else {
                    // the digits done make room for the index; the later passes find theirs lower by as much
                    a.out[dst] = ((kx >> (a.shift + a.bits)) << a.val_bits) | (uint64_t)v;
                }
            } else {
                a.out[dst] = kx;
            }
        }
        return bad;
    };
    bool bad = write();
    if constexpr (!MASKS) {
        if (__syncthreads_or(bad)) {            // (nobody reads the output before this kernel has ended)
            for (int round = 0; round < os_rounds(tile_count); ++round) {
                bad = false;
                for (int odd = 0; odd < 2; ++odd) {
                    bad |= os_exchange(in_digit, skeys, tile_count, odd, threadIdx.x, OS_THREADS);
                    __syncthreads();
                }
                if (!__syncthreads_or(bad)) break;
            }
            write();
        }
    }
}

static size_t os_pass_smem(int items, int bits, bool wide, bool masks)
{
    const size_t bins = (size_t)1 << bits;
    return os_element_bytes(items, (int)bins, wide, masks) + OS_WARPS * bins * 2 + (2 * bins + 1) * 4;
}

template <int ITEMS, bool WIDE, int OUT, bool MASKS>
static int os_launch(const OsPass& a, cudaStream_t stream)
{
    if (allow_smem(os_pass_kernel<ITEMS, WIDE, OUT, MASKS>) != cudaSuccess)
        return check_launch("ptv3_argsort_inverse: shared memory attribute");
    os_pass_kernel<ITEMS, WIDE, OUT, MASKS><<<a.ntiles * a.rows, OS_THREADS, os_pass_smem(ITEMS, a.bits, WIDE, MASKS),
                                              stream>>>(a);
    return check_launch("ptv3_argsort_inverse");
}

static SortPlan sort_plan(int k, int64_t n, int sig_bits)
{
    SortPlan p;
    p.passes = sig_bits <= 0 ? 1 : (sig_bits + OS_MAX_BITS - 1) / OS_MAX_BITS;
    p.bits = sig_bits <= 0 ? 8 : (sig_bits + p.passes - 1) / p.passes;   // spread evenly
    p.val_bits = 1;
    while (((n - 1) >> p.val_bits) != 0) ++p.val_bits;
    p.wide = 0;
    while (sig_bits - p.wide * p.bits + p.val_bits > 64) ++p.wide;
    // tiles of 8192: half the look-back and status words per element; of 4096, with half the chain from start to
    // end, while those of all rows run at once (two to an SM)
    p.items = (int64_t)k * ((n + 8 * OS_THREADS - 1) / (8 * OS_THREADS)) <= 2 * SMS ? 8 : 16;
    p.ntiles = ceil_div(n, (int64_t)p.items * OS_THREADS);
    size_t b = 0;
    b += 2 * align_up((size_t)k * n * sizeof(uint64_t), 256);   // ping-pong of words or keys
    if (p.wide > 1) b += 2 * align_up((size_t)k * n * sizeof(int32_t), 256);    // and of indices beside keys
    // zeroed region: histograms, tile counters, tile status
    b += align_up((size_t)k * OS_MAX_PASSES * OS_MAX_BINS * sizeof(uint32_t), 256);
    b += align_up((size_t)k * OS_MAX_PASSES * sizeof(uint32_t), 256);
    b += align_up((size_t)k * p.ntiles * OS_MAX_BINS * sizeof(uint32_t), 256);
    p.bytes = b;
    return p;
}

}  // namespace ptv3

extern "C" size_t ptv3_argsort_workspace_bytes(int k, int64_t n, int sig_bits)
{
    if (k <= 0 || n <= 0) return 0;
    return ptv3::sort_plan(k, n, sig_bits).bytes;
}

extern "C" int ptv3_argsort_inverse(const int64_t* codes, int k, int64_t n, int sig_bits,
                                    int64_t* order, int64_t* inverse, uint32_t* status, void* workspace,
                                    size_t workspace_bytes, void* stream_)
{
    using namespace ptv3;
    PTV3_REQUIRE(k >= 1 && k <= 65535 && n >= 0, PTV3_ERR_INVALID_ARGUMENT, "ptv3_argsort_inverse: bad k/n");
    PTV3_REQUIRE(sig_bits >= 0 && sig_bits <= 63, PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_argsort_inverse: sig_bits %d outside [0, 63]", sig_bits);
    PTV3_REQUIRE(n <= (int64_t)OS_COUNT_MASK, PTV3_ERR_UNSUPPORTED,
                 "ptv3_argsort_inverse: more than 2^28 - 1 elements per row");
    if (n == 0) return PTV3_OK;
    PTV3_REQUIRE(codes && order && inverse && workspace, PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_argsort_inverse: null pointer");
    const SortPlan p = sort_plan(k, n, sig_bits);
    PTV3_REQUIRE(workspace_bytes >= p.bytes, PTV3_ERR_WORKSPACE,
                 "ptv3_argsort_inverse: workspace %zu < %zu bytes", workspace_bytes, p.bytes);
    cudaStream_t stream = (cudaStream_t)stream_;
    Carver cv(workspace);
    uint64_t* kbuf[2] = {cv.take<uint64_t>((size_t)k * n), cv.take<uint64_t>((size_t)k * n)};
    int32_t* vbuf[2] = {nullptr, nullptr};
    if (p.wide > 1)
        for (int32_t*& v : vbuf) v = cv.take<int32_t>((size_t)k * n);
    char* zero_lo = cv.base + cv.off;
    uint32_t* hist = cv.take<uint32_t>((size_t)k * OS_MAX_PASSES * OS_MAX_BINS);
    uint32_t* counters = cv.take<uint32_t>((size_t)k * OS_MAX_PASSES);
    uint32_t* tile_status = cv.take<uint32_t>((size_t)k * p.ntiles * OS_MAX_BINS);
    if (cudaMemsetAsync(zero_lo, 0, (size_t)(cv.base + cv.off - zero_lo), stream) != cudaSuccess)
        return check_launch("ptv3_argsort_inverse: memset");

    const uint64_t* kin = reinterpret_cast<const uint64_t*>(codes);
    {
        const int hb = (int)std::min<int64_t>(ceil_div(n, OS_THREADS * 8), 4 * SMS);
        os_hist_kernel<<<dim3(hb, k), OS_THREADS, (size_t)p.passes * OS_MAX_BINS * sizeof(uint32_t), stream>>>(
            kin, n, sig_bits, p.bits, p.passes, hist);
    }
    OsPass a;
    a.in = kin;
    a.vals_in = nullptr;
    a.order = order;
    a.inverse = inverse;
    a.hist = hist;
    a.tile_status = tile_status;
    a.tile_counter = counters;
    a.status = status;
    a.n = n;
    a.raw = 1;
    a.val_bits = p.val_bits;
    a.ntiles = p.ntiles;
    a.rows = k;
    // the histogram kernel cuts every digit with the full width; the last digit then only
    // holds the bits that are left, which is the same value (nothing is set above sig_bits)
    a.bits = p.bits;
    a.shift = 0;
    for (a.pass = 0; a.pass < p.passes; ++a.pass) {
        const bool wide = a.pass < p.wide, last = a.pass == p.passes - 1;
        a.out = kbuf[a.pass & 1];
        a.vals_out = vbuf[a.pass & 1];
        // rows take turns over the grid, so every row has the same share of the running tiles (a
        // tile waits only for tiles of its own row); only the last pass goes row after row where the inverses of
        // all rows together outgrow L2, which holds those of one (its scattered 8-byte writes then meet in L2)
        a.by_row = last && (int64_t)k * n * 8 > OS_L2_BYTES;
        const bool small = p.items == 8;
        int rc;
        if (wide && a.pass + 1 < p.wide) rc = (small ? os_launch<8, true, OS_WIDE, true> : os_launch<16, true, OS_WIDE, true>)(a, stream);
        else if (wide) rc = (small ? os_launch<8, true, OS_PACKED, true> : os_launch<16, true, OS_PACKED, true>)(a, stream);
        else if (p.wide > 0 && last) rc = (small ? os_launch<8, false, OS_FINAL, true> : os_launch<16, false, OS_FINAL, true>)(a, stream);
        else if (p.wide > 0) rc = (small ? os_launch<8, false, OS_PACKED, true> : os_launch<16, false, OS_PACKED, true>)(a, stream);
        else if (last) rc = (small ? os_launch<8, false, OS_FINAL, false> : os_launch<16, false, OS_FINAL, false>)(a, stream);
        else rc = (small ? os_launch<8, false, OS_PACKED, false> : os_launch<16, false, OS_PACKED, false>)(a, stream);
        if (rc != PTV3_OK) return rc;
        a.in = a.out;
        a.vals_in = a.vals_out;
        // (a wide pass that packs drops the digits that are done)
        a.shift = wide && a.pass + 1 == p.wide ? 0 : a.shift + a.bits;
        if (!wide || a.pass + 1 == p.wide) a.raw = 0;
    }
    count_launches(1 + p.passes);
    return PTV3_OK;
}
