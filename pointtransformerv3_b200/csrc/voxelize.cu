// Voxelisation front end: the step right before the serialized backbone.
//
//   ptv3_grid_coord    grid_coord = trunc((coord - min over all points) / grid_size)
//                      as the reference derives it when only coordinates are given
//                      (model.py:88-96, 156-158): batch-global minimum, fp32
//                      subtraction and division, truncation toward zero.
//   ptv3_voxel_dedup   one point per occupied voxel of every scene: the first
//                      point (lowest row) of each (scene, x, y, z) is kept, kept
//                      rows stay in input order (so scenes stay contiguous), and
//                      every input point learns the kept row of its voxel.  The
//                      reference leaves this to its data pipeline (grid sampling);
//                      the backbone assumes at most one point per voxel for its
//                      submanifold convolutions.
//
// The voxel hash table is the one of the kernel-map builder (lowest row wins on
// insertion); positions come from the flag scan used by the pooling plan.
#include <algorithm>

#include "common.cuh"
#include "kmap.cuh"
#include "scan.cuh"

namespace ptv3 {

// ---- grid coordinates ---------------------------------------------------------
__device__ __forceinline__ void atomic_min_float(float* addr, float v)
{
    // non-negative floats order like signed ints, negative ones in reverse like unsigned ints
    if (v >= 0.f)
        atomicMin(reinterpret_cast<int*>(addr), __float_as_int(v));
    else
        atomicMax(reinterpret_cast<unsigned int*>(addr), __float_as_uint(v));
}

__global__ void vox_origin_init_kernel(float* origin)
{
    if (threadIdx.x < 3) origin[threadIdx.x] = __int_as_float(0x7f800000);   // +inf
}

__global__ void __launch_bounds__(256) vox_min_kernel(const float* __restrict__ coord, int64_t n,
                                                      float* __restrict__ origin)
{
    float m[3] = {__int_as_float(0x7f800000), __int_as_float(0x7f800000), __int_as_float(0x7f800000)};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        m[0] = fminf(m[0], coord[3 * i + 0]);
        m[1] = fminf(m[1], coord[3 * i + 1]);
        m[2] = fminf(m[2], coord[3 * i + 2]);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m[a] = fminf(m[a], __shfl_xor_sync(0xffffffffu, m[a], o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomic_min_float(origin + 0, m[0]);
        atomic_min_float(origin + 1, m[1]);
        atomic_min_float(origin + 2, m[2]);
    }
}

__global__ void __launch_bounds__(256) vox_grid_kernel(const float* __restrict__ coord, int64_t n3,
                                                       float grid_size, const float* __restrict__ origin,
                                                       int32_t* __restrict__ grid)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n3) return;
    // IEEE subtraction and division (the build enables fast-math approximations elsewhere)
    const float d = __fsub_rn(coord[i], origin[i % 3]);
    grid[i] = (int32_t)truncf(__fdiv_rn(d, grid_size));
}

// ---- one point per voxel ----------------------------------------------------------
__global__ void __launch_bounds__(256) vox_first_kernel(const int32_t* __restrict__ indices, int64_t n,
                                                        const unsigned long long* __restrict__ keys,
                                                        const uint32_t* __restrict__ vals, uint64_t cap_mask,
                                                        uint32_t* __restrict__ first, uint32_t* __restrict__ status)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int4 v = reinterpret_cast<const int4*>(indices)[i];
    uint64_t key;
    uint32_t f = (uint32_t)i;   // a point outside the key range (reported through the status) keeps itself
    if (km_key(v.x, v.y, v.z, v.w, key)) {
        bool overflow = false;
        const int32_t r = km_lookup(keys, vals, cap_mask, key, &overflow);
        if (overflow) atomicOr(status, PTV3_STATUS_PROBE_LIMIT);
        if (r >= 0) f = (uint32_t)r;
    }
    first[i] = f;
}

struct FirstFlag {
    const uint32_t* first;
    __device__ bool operator()(int, int64_t j) const { return first[j] == (uint32_t)j; }
};

struct KeepSink {
    int64_t* keep;
    uint32_t* rank;
    __device__ void operator()(int, int64_t j, uint32_t pos, bool f) const
    {
        if (f) {
            keep[pos] = j;
            rank[j] = pos;
        }
    }
};

__global__ void __launch_bounds__(256) vox_inverse_kernel(const uint32_t* __restrict__ first,
                                                          const uint32_t* __restrict__ rank, int64_t n,
                                                          const uint32_t* __restrict__ total,
                                                          const int64_t* __restrict__ offset, int n_scenes,
                                                          int64_t* __restrict__ point2voxel,
                                                          int64_t* __restrict__ new_offset,
                                                          int64_t* __restrict__ count)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) point2voxel[i] = rank[first[i]];
    if (i == 0) *count = *total;
    if (i < n_scenes && new_offset) {
        // the first point of a scene is the first point of its voxel, so its rank is the number
        // of voxels kept before the scene
        const int64_t end = offset[i];
        new_offset[i] = end < n ? (int64_t)rank[end] : (int64_t)*total;
    }
}

static size_t dedup_scratch_bytes(int64_t n)
{
    const int ntiles = ceil_div(n, SC_TILE);
    return align_up((size_t)n * 4, 256) * 2 + align_up((size_t)ntiles * 4, 256) + 256;
}

// ---- raw points to one point per voxel, fused ----------------------------------------
// 2.4 M points took 0.68 ms through single operators (a library kernel for the scene ids alone 0.32 ms,
// the grid coordinates written and read back twice, a table of 3.5 slots per point with a cleared 12
// bytes each, two probes per point).  Here the grid coordinates are recomputed where they are needed, a
// point remembers its slot instead of probing again, and the voxel count reaches the host from the insertion,
// before the voxels are numbered and the outputs made.
//
// What bounds it: sectors of the table fetched at random from L2, one per point and kernel (claims, first rows,
// map), 14 us a pass at 2.4 M points; the claims take longer, since a point of a new voxel is a chain of two round
// trips.  A slot is therefore 16 bytes, key, first row and voxel number together: one sector answers a probe.
// With the keys and the rows in two arrays a point cost two sectors and always an atomic.
// 1.5 slots per point: the 57 MB of 2.4 M points stay in the 126 MB L2, and points that all lie in voxels
// of their own fill the table to two thirds.  2.4 M points into 410 000 voxels, with the host's read: 145 -> 115 us.
struct __align__(16) VoxelSlot {
    unsigned long long key;
    uint32_t first;      // lowest row of the voxel
    uint32_t rank;       // its number among the kept rows
};

constexpr uint32_t VZ_NO_SLOT = 0xffffffffu;
constexpr int VZ_ITEMS = 4;                                          // pieces of a thread in flight at once
constexpr int VZ_TILE_ITEMS = 16, VZ_TILE = 256 * VZ_TILE_ITEMS;     // points of a tile of the numbering
constexpr int VZ_WORDS = VZ_TILE / 32, VZ_GROUP = 256;
constexpr int VZ_COUNTERS = 64;                                      // of claimed slots, a sector each

// Loads of what an earlier kernel of the chain makes: in their place behind pdl_wait() (see common.cuh).
__device__ __forceinline__ uint32_t vz_made(const uint32_t* p)
{
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int64_t vz_made(const int64_t* p)
{
    int64_t v;
    asm volatile("ld.global.s64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float vz_made(const float* p)
{
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}

__global__ void vz_origin_init_kernel(float* origin)
{
    pdl_launch_next();
    if (threadIdx.x < 3) origin[threadIdx.x] = __int_as_float(0x7f800000);   // +inf
}

// Clears the table and the tile words (`clear` 16-byte pieces) and takes the minimum over the points, four
// points (three 16-byte loads) per step, one atomic per block and axis.  One kernel: the stores go to L2
// while the coordinates come from memory (2.4 M points: one launch of 14 us, apart 11 and 8 us and a gap).
__global__ void __launch_bounds__(256) vz_prepare_kernel(const float* coord, int64_t n, bool vec, float* origin,
                                                         uint4* table, int64_t clear)
{
    pdl_launch_next();
    const float inf = __int_as_float(0x7f800000);
    float m[3] = {inf, inf, inf};
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    const uint32_t ones = 0xffffffffu;
    for (int64_t i = t; i < clear; i += stride) table[i] = make_uint4(ones, ones, ones, ones);
    int64_t done = 0;
    if (vec) {
        done = n / 4 * 4;
        const float4* c4 = reinterpret_cast<const float4*>(coord);
        for (int64_t i = t; i < n / 4; i += stride) {
            const float4 a = c4[3 * i], b = c4[3 * i + 1], c = c4[3 * i + 2];
            m[0] = fminf(m[0], fminf(fminf(a.x, a.w), fminf(b.z, c.y)));
            m[1] = fminf(m[1], fminf(fminf(a.y, b.x), fminf(b.w, c.z)));
            m[2] = fminf(m[2], fminf(fminf(a.z, b.y), fminf(c.x, c.w)));
        }
    }
    for (int64_t i = done + t; i < n; i += stride)
#pragma unroll
        for (int a = 0; a < 3; ++a) m[a] = fminf(m[a], coord[3 * i + a]);
    __shared__ float warp_min[8][3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m[a] = fminf(m[a], __shfl_xor_sync(0xffffffffu, m[a], o));
        if ((threadIdx.x & 31) == 0) warp_min[threadIdx.x >> 5][a] = m[a];
    }
    __syncthreads();
    pdl_wait();
    if (threadIdx.x < 3) {
        float v = warp_min[0][threadIdx.x];
        for (int w = 1; w < 8; ++w) v = fminf(v, warp_min[w][threadIdx.x]);
        atomic_min_float(origin + threadIdx.x, v);
    }
}

__device__ __forceinline__ int32_t vz_cell(float coord, float origin, float grid_size)
{
    return (int32_t)truncf(__fdiv_rn(__fsub_rn(coord, origin), grid_size));
}

// a pair of slots (one 32-byte sector) as it stands, past L1; either word may be older than an update under way
__device__ __forceinline__ void vz_look(const VoxelSlot* pair, unsigned long long (&key)[2], uint32_t (&first)[2])
{
    unsigned long long r0, r1;
    asm volatile("ld.relaxed.gpu.global.v4.u64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(key[0]), "=l"(r0), "=l"(key[1]), "=l"(r1) : "l"(pair) : "memory");
    first[0] = (uint32_t)r0;
    first[1] = (uint32_t)r1;
}

// Every point claims a slot for its voxel; the lowest row wins.  A plain look comes first: most points of a
// voxel follow its first one, find key and row as they should be and need no atomic (an older row only costs
// one).  Probes go by pairs, so that few of them need a second round trip.  Claims are counted (a point without a
// slot counts as one): the number of voxels is known when this kernel ends.
// One point per thread: with two or four the looks of more points pass before their voxels' first claims (38,
// 42 and 49 us at 2.4 M points).
__global__ void __launch_bounds__(256) vz_insert_kernel(const float* coord, int64_t n, float grid_size,
                                                        const float* origin, const int64_t* offset,
                                                        int B, VoxelSlot* table, uint32_t pairs,
                                                        uint32_t* slot_of, uint32_t* claimed, uint32_t* status)
{
    extern __shared__ int64_t ends[];
    pdl_launch_next();
    for (int s = threadIdx.x; s < B; s += blockDim.x) ends[s] = offset[s];
    __syncthreads();
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    float c[3] = {};
    int lo = 0, hi = B - 1;              // first scene whose end lies beyond i
    if (i < n) {
#pragma unroll
        for (int a = 0; a < 3; ++a) c[a] = coord[3 * i + a];
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (ends[mid] > i) hi = mid; else lo = mid + 1;
        }
    }
    pdl_wait();                          // the minimum and the cleared table
    bool own = false;
    if (i < n) {
        uint64_t key;
        uint32_t at = VZ_NO_SLOT;        // outside the key range: reported, and the point keeps itself
        if (km_key(lo, vz_cell(c[0], vz_made(origin), grid_size), vz_cell(c[1], vz_made(origin + 1), grid_size),
                   vz_cell(c[2], vz_made(origin + 2), grid_size), key)) {
            uint32_t pair = (uint32_t)(((km_mix(key) >> 32) * pairs) >> 32), probe = 0;
            for (; probe < pairs && at == VZ_NO_SLOT; ++probe) {
                unsigned long long seen[2];
                uint32_t first[2];
                vz_look(table + 2 * (size_t)pair, seen, first);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (at != VZ_NO_SLOT) continue;
                    VoxelSlot* slot = table + 2 * (size_t)pair + h;
                    if (seen[h] == KM_EMPTY) {
                        seen[h] = atomicCAS(&slot->key, KM_EMPTY, key);
                        first[h] = VZ_NO_SLOT;
                        own = seen[h] == KM_EMPTY;
                    }
                    if (own || seen[h] == key) {
                        if (first[h] > (uint32_t)i) atomicMin(&slot->first, (uint32_t)i);
                        at = 2 * pair + h;
                    }
                }
                pair = pair + 1 == pairs ? 0 : pair + 1;
            }
            if (at == VZ_NO_SLOT) atomicOr(status, PTV3_STATUS_PROBE_LIMIT);
        } else {
            atomicOr(status, PTV3_STATUS_BAD_INDEX);
        }
        own |= at == VZ_NO_SLOT;
        slot_of[i] = at;
    }
    const int mine = __syncthreads_count(own);
    // (one counter for all blocks: their additions to one address alone take 10 us; cleared to all ones: one less)
    if (threadIdx.x == 0 && mine) atomicAdd(claimed + blockIdx.x % VZ_COUNTERS * 8, (uint32_t)mine);
}

// The kept points (the first of every voxel) of a tile as a bit mask, and how many they are: per tile, and
// summed over groups of VZ_GROUP tiles.  The first block hands the number of voxels and the status word to the
// host before anything else: the voxels are numbered while the host makes the outputs.
__global__ void __launch_bounds__(256) vz_first_kernel(const uint32_t* slot_of, int64_t n, const VoxelSlot* table,
                                                       uint32_t slots, uint32_t* kept, uint32_t* tile_sums,
                                                       uint32_t* group_sums, const uint32_t* claimed,
                                                       const uint32_t* status, int64_t* count, int64_t* host)
{
    __shared__ uint32_t sum;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_launch_next();
    if (threadIdx.x == 0) sum = 0;
    const int64_t base = (int64_t)blockIdx.x * VZ_TILE + threadIdx.x;
    pdl_wait();
    if (blockIdx.x == 0 && warp == 7) {
        static_assert(VZ_COUNTERS == 64, "two counters per lane");
        const uint32_t voxels =
            __reduce_add_sync(0xffffffffu, vz_made(claimed + lane * 8) + vz_made(claimed + (lane + 32) * 8) + 2u);
        if (lane == 0) {
            *count = voxels;
            host[0] = voxels;
            host[1] = vz_made(status);
            __threadfence_system();
            *reinterpret_cast<volatile int64_t*>(&host[2]) = 1;
            __threadfence_system();
        }
    }
    uint32_t s[VZ_TILE_ITEMS], f[VZ_TILE_ITEMS], word = 0;
#pragma unroll
    for (int it = 0; it < VZ_TILE_ITEMS; ++it) {
        const int64_t j = base + it * 256;
        s[it] = j < n ? vz_made(slot_of + j) : VZ_NO_SLOT;
    }
#pragma unroll
    for (int it = 0; it < VZ_TILE_ITEMS; ++it)
        f[it] = s[it] < slots ? vz_made(&table[s[it]].first) : (uint32_t)(base + it * 256);
#pragma unroll
    for (int it = 0; it < VZ_TILE_ITEMS; ++it) {
        const int64_t j = base + it * 256;
        const uint32_t set = __ballot_sync(0xffffffffu, j < n && f[it] == (uint32_t)j);
        if (lane == it) word = set;
    }
    if (lane < VZ_TILE_ITEMS) kept[(int64_t)blockIdx.x * VZ_WORDS + lane * 8 + warp] = word;
    const uint32_t c = __reduce_add_sync(0xffffffffu, __popc(word));
    __syncthreads();
    if (lane == 0 && c) atomicAdd(&sum, c);
    __syncthreads();
    if (threadIdx.x == 0) {
        tile_sums[blockIdx.x] = sum;
        if (sum) atomicAdd(&group_sums[blockIdx.x / VZ_GROUP], sum);     // cleared to all ones: one less
    }
}

// Numbers the kept points in input order.  A block adds up the groups and the tiles before its own (at most
// 2 048 and 255 words for 2^31 points), which takes no kernel between the two and waits for no other block;
// a kept point leaves its number in its slot, one without a slot (reported) in the map itself.
// (With the scan of the tile sums in a kernel of its own and first row and number of every point in arrays:
// 39 us at 2.4 M points; as one kernel with a look-back 30, and the host learned the count at its end.)
__global__ void __launch_bounds__(256) vz_number_kernel(const uint32_t* slot_of, int64_t n, const uint32_t* kept,
                                                        const uint32_t* tile_sums, const uint32_t* group_sums,
                                                        VoxelSlot* table, uint32_t slots, int64_t* keep,
                                                        int64_t* point2voxel)
{
    static_assert(VZ_WORDS == 128, "four words per lane of a warp");
    __shared__ __align__(16) uint32_t before[VZ_WORDS];
    __shared__ uint32_t sum;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tile = blockIdx.x, group = tile / VZ_GROUP;
    pdl_launch_next();
    if (threadIdx.x == 0) sum = 0;
    pdl_wait();
    uint32_t set[VZ_TILE_ITEMS], c = 0;
#pragma unroll
    for (int it = 0; it < VZ_TILE_ITEMS; ++it) set[it] = vz_made(kept + (int64_t)tile * VZ_WORDS + it * 8 + warp);
    for (int g = threadIdx.x; g < group; g += 256) c += vz_made(group_sums + g) + 1u;
    if (group * VZ_GROUP + (int)threadIdx.x < tile) c += vz_made(tile_sums + group * VZ_GROUP + threadIdx.x);
    if (lane == 0)
#pragma unroll
        for (int it = 0; it < VZ_TILE_ITEMS; ++it) before[it * 8 + warp] = __popc(set[it]);
    c = __reduce_add_sync(0xffffffffu, c);
    __syncthreads();
    if (lane == 0 && c) atomicAdd(&sum, c);
    if (warp == 0) {
        const uint4 v = reinterpret_cast<const uint4*>(before)[lane];
        uint32_t inc = v.x + v.y + v.z + v.w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        reinterpret_cast<uint4*>(before)[lane] =
            make_uint4(inc - v.w - v.z - v.y - v.x, inc - v.w - v.z - v.y, inc - v.w - v.z, inc - v.w);
    }
    __syncthreads();
    const uint32_t prefix = sum, earlier = (1u << lane) - 1;
    const int64_t base = (int64_t)tile * VZ_TILE + threadIdx.x;
    uint32_t s[VZ_TILE_ITEMS];
#pragma unroll
    for (int it = 0; it < VZ_TILE_ITEMS; ++it) {
        const int64_t j = base + it * 256;
        s[it] = j < n && (set[it] >> lane & 1) ? vz_made(slot_of + j) : VZ_NO_SLOT;
    }
#pragma unroll
    for (int it = 0; it < VZ_TILE_ITEMS; ++it) {
        const int64_t j = base + it * 256;
        const uint32_t pos = prefix + before[it * 8 + warp] + __popc(set[it] & earlier);
        if (!(set[it] >> lane & 1) || pos >= n) continue;
        keep[pos] = j;
        if (s[it] < slots)
            table[s[it]].rank = pos;
        else
            point2voxel[j] = pos;
    }
}

// every point's voxel number from its slot, and the scenes' ends among the kept points
__global__ void __launch_bounds__(256) vz_inverse_kernel(const uint32_t* slot_of, int64_t n, const VoxelSlot* table,
                                                         uint32_t slots, const int64_t* offset, int n_scenes,
                                                         const int64_t* count, int64_t* point2voxel,
                                                         int64_t* new_offset)
{
    pdl_launch_next();
    pdl_wait();
    const int64_t base = blockIdx.x * (int64_t)(256 * VZ_ITEMS) + threadIdx.x;
    uint32_t s[VZ_ITEMS], r[VZ_ITEMS];
#pragma unroll
    for (int q = 0; q < VZ_ITEMS; ++q) s[q] = base + q * 256 < n ? vz_made(slot_of + base + q * 256) : VZ_NO_SLOT;
#pragma unroll
    for (int q = 0; q < VZ_ITEMS; ++q) r[q] = s[q] < slots ? vz_made(&table[s[q]].rank) : 0u;
#pragma unroll
    for (int q = 0; q < VZ_ITEMS; ++q)
        if (s[q] < slots) point2voxel[base + q * 256] = r[q];
    for (int64_t i = blockIdx.x * (int64_t)256 + threadIdx.x; i < n_scenes; i += (int64_t)gridDim.x * 256) {
        // the first point of a scene is the first point of its voxel, so its number is the number of
        // voxels kept before the scene
        const int64_t end = offset[i];
        if (end >= n) {
            new_offset[i] = vz_made(count);
        } else {
            const uint32_t at = vz_made(slot_of + end);
            new_offset[i] = at < slots ? (int64_t)vz_made(&table[at].rank) : vz_made(point2voxel + end);
        }
    }
}

// Output rows: coordinates, grid coordinates (recomputed) and features of the kept points; a row of features
// is `words` pieces of W.  A block copies `block_rows` rows, about VZ_PIECES pieces and one per thread and step:
// the row of a piece comes from a 32-bit division and the source rows from shared memory (410 000 rows of 24
// feature bytes: 21 us with one piece per thread, a 64-bit division and a load of its source row each).
constexpr int VZ_ROWS = 128, VZ_PIECES = 1024;
template <typename W>
__global__ void __launch_bounds__(256) vz_gather_kernel(const int64_t* keep, int64_t m, const float* coord,
                                                        const float* origin, float grid_size, const W* feat,
                                                        uint32_t words, int block_rows, float* out_coord,
                                                        int32_t* out_grid, W* out_feat)
{
    __shared__ int64_t source[VZ_ROWS];
    pdl_launch_next();
    pdl_wait();
    const int64_t row0 = blockIdx.x * (int64_t)block_rows;
    const uint32_t rows = (uint32_t)(m - row0 < block_rows ? m - row0 : block_rows);
    if (threadIdx.x < rows) source[threadIdx.x] = vz_made(keep + row0 + threadIdx.x);
    __syncthreads();
    const float o0 = vz_made(origin), o1 = vz_made(origin + 1), o2 = vz_made(origin + 2);
    const uint32_t lanes = 3 + words;            // three axes, then the feature words
    const uint32_t pieces = rows * lanes;
    for (uint32_t e0 = threadIdx.x; e0 < pieces; e0 += 256 * VZ_ITEMS) {
        float c[VZ_ITEMS];
        W w[VZ_ITEMS];
        int64_t to[VZ_ITEMS];
        uint32_t axis[VZ_ITEMS];
#pragma unroll
        for (int q = 0; q < VZ_ITEMS; ++q) {
            const uint32_t e = e0 + q * 256;
            axis[q] = VZ_NO_SLOT;
            if (e >= pieces) continue;
            const uint32_t r = e / lanes, a = e - r * lanes;
            const int64_t src = source[r], row = row0 + r;
            axis[q] = a;
            to[q] = a < 3 ? 3 * row + a : row * words + (a - 3);
            if (a < 3)
                c[q] = coord[3 * src + a];
            else
                w[q] = feat[src * words + (a - 3)];
        }
#pragma unroll
        for (int q = 0; q < VZ_ITEMS; ++q) {
            if (axis[q] == VZ_NO_SLOT) continue;
            if (axis[q] < 3) {
                out_coord[to[q]] = c[q];
                out_grid[to[q]] = vz_cell(c[q], axis[q] == 0 ? o0 : axis[q] == 1 ? o1 : o2, grid_size);
            } else {
                out_feat[to[q]] = w[q];
            }
        }
    }
}

static uint32_t vz_pairs(int64_t n) { return (uint32_t)(n < 1024 ? 768 : (3 * n + 3) / 4); }

// the table, the count of voxels and the group sums (cleared together, up to `slot_of`), the slots of the
// points, the kept points of every tile as bits and as numbers
struct VoxelScratch {
    VoxelSlot* table;
    uint32_t *claimed, *group_sums, *slot_of, *kept, *tile_sums;
    size_t bytes;
};

static VoxelScratch vz_scratch(int64_t n, void* base)
{
    const int ntiles = ceil_div(n, VZ_TILE);
    Carver cv(base);
    VoxelScratch v;
    v.table = cv.take<VoxelSlot>(2 * (size_t)vz_pairs(n));
    v.claimed = cv.take<uint32_t>(VZ_COUNTERS * 8);
    v.group_sums = cv.take<uint32_t>(ceil_div(ntiles, VZ_GROUP));
    v.slot_of = cv.take<uint32_t>(n);
    v.kept = cv.take<uint32_t>((size_t)ntiles * VZ_WORDS);
    v.tile_sums = cv.take<uint32_t>(ntiles);
    v.bytes = cv.off;
    return v;
}

}  // namespace ptv3

using namespace ptv3;

extern "C" int ptv3_grid_coord(const float* coord, int64_t n, float grid_size, float* origin, int32_t* grid_coord,
                               void* stream_)
{
    PTV3_REQUIRE(n >= 0, PTV3_ERR_INVALID_ARGUMENT, "ptv3_grid_coord: n < 0");
    PTV3_REQUIRE(grid_size > 0.f, PTV3_ERR_INVALID_ARGUMENT, "ptv3_grid_coord: grid_size must be positive");
    if (n == 0) return PTV3_OK;
    PTV3_REQUIRE(coord && origin && grid_coord, PTV3_ERR_INVALID_ARGUMENT, "ptv3_grid_coord: null pointer");
    cudaStream_t stream = (cudaStream_t)stream_;
    vox_origin_init_kernel<<<1, 32, 0, stream>>>(origin);
    const unsigned blocks = (unsigned)std::min<int64_t>((n + 255) / 256, SMS * 8);
    vox_min_kernel<<<blocks, 256, 0, stream>>>(coord, n, origin);
    vox_grid_kernel<<<(unsigned)((3 * n + 255) / 256), 256, 0, stream>>>(coord, 3 * n, grid_size, origin, grid_coord);
    count_launches(3);
    return check_launch("ptv3_grid_coord");
}

extern "C" size_t ptv3_voxel_dedup_workspace_bytes(int64_t n)
{
    if (n <= 0) return 0;
    return km_table_bytes(n) + dedup_scratch_bytes(n);
}

extern "C" int ptv3_voxel_dedup(const int32_t* indices, int64_t n, const int64_t* offset, int n_scenes,
                                int64_t* keep, int64_t* point2voxel, int64_t* new_offset, int64_t* count,
                                uint32_t* status, void* workspace, size_t workspace_bytes, void* stream_)
{
    PTV3_REQUIRE(n >= 0 && n < (1ll << 31), PTV3_ERR_INVALID_ARGUMENT, "ptv3_voxel_dedup: bad n");
    PTV3_REQUIRE(n_scenes >= 0 && (n_scenes == 0 || offset), PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_voxel_dedup: offset missing");
    PTV3_REQUIRE(count != nullptr, PTV3_ERR_INVALID_ARGUMENT, "ptv3_voxel_dedup: null pointer");
    cudaStream_t stream = (cudaStream_t)stream_;
    if (n == 0) {
        cudaMemsetAsync(count, 0, sizeof(int64_t), stream);
        if (new_offset && n_scenes > 0) cudaMemsetAsync(new_offset, 0, sizeof(int64_t) * n_scenes, stream);
        return check_launch("ptv3_voxel_dedup");
    }
    PTV3_REQUIRE(indices && keep && point2voxel && status && workspace, PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_voxel_dedup: null pointer");
    PTV3_REQUIRE(((uintptr_t)indices & 15) == 0, PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_voxel_dedup: indices must be 16-byte aligned");
    PTV3_REQUIRE(n_scenes <= n, PTV3_ERR_INVALID_ARGUMENT, "ptv3_voxel_dedup: more scenes than points");
    const size_t need = ptv3_voxel_dedup_workspace_bytes(n);
    PTV3_REQUIRE(workspace_bytes >= need, PTV3_ERR_WORKSPACE, "ptv3_voxel_dedup: workspace %zu < %zu bytes",
                 workspace_bytes, need);
    unsigned long long* keys;
    uint32_t* vals;
    uint64_t cap_mask;
    int rc = km_build_table(indices, n, workspace, status, stream, &keys, &vals, &cap_mask);
    if (rc != PTV3_OK) return rc;
    Carver cv(static_cast<char*>(workspace) + km_table_bytes(n));
    const int ntiles = ceil_div(n, SC_TILE);
    uint32_t* first = cv.take<uint32_t>(n);
    uint32_t* rank = cv.take<uint32_t>(n);
    uint32_t* tile_sums = cv.take<uint32_t>(ntiles);
    uint32_t* total = cv.take<uint32_t>(1);
    const unsigned blocks = (unsigned)((n + 255) / 256);
    vox_first_kernel<<<blocks, 256, 0, stream>>>(indices, n, keys, vals, cap_mask, first, status);
    const FirstFlag flag{first};
    scan_tile_sums_kernel<FirstFlag><<<dim3(ntiles, 1), SC_THREADS, 0, stream>>>(flag, n, ntiles, tile_sums);
    scan_sums_kernel<<<1, SC_THREADS, 0, stream>>>(tile_sums, ntiles, total);
    scan_apply_kernel<FirstFlag, KeepSink><<<dim3(ntiles, 1), SC_THREADS, 0, stream>>>(
        flag, KeepSink{keep, rank}, n, ntiles, tile_sums);
    vox_inverse_kernel<<<blocks, 256, 0, stream>>>(first, rank, n, total, offset, n_scenes, point2voxel, new_offset,
                                                   count);
    count_launches(5);
    return check_launch("ptv3_voxel_dedup");
}

extern "C" size_t ptv3_voxelize_workspace_bytes(int64_t n)
{
    if (n <= 0) return 0;
    return vz_scratch(n, nullptr).bytes;
}

extern "C" int ptv3_voxelize(const float* coord, int64_t n, float grid_size, const int64_t* offset, int n_scenes,
                             float* origin, int64_t* keep, int64_t* point2voxel, int64_t* new_offset, int64_t* count_host,
                             int64_t* count, uint32_t* status, void* workspace, size_t workspace_bytes, void* stream_)
{
    PTV3_REQUIRE(n >= 1 && n < (1ll << 31) - 1, PTV3_ERR_INVALID_ARGUMENT, "ptv3_voxelize: bad n");
    PTV3_REQUIRE(grid_size > 0.f, PTV3_ERR_INVALID_ARGUMENT, "ptv3_voxelize: grid_size must be positive");
    PTV3_REQUIRE(n_scenes >= 1 && n_scenes <= 4096 && n_scenes <= n, PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_voxelize: %d scenes", n_scenes);
    PTV3_REQUIRE(coord && offset && origin && keep && point2voxel && new_offset && count_host && count && status &&
                     workspace,
                 PTV3_ERR_INVALID_ARGUMENT, "ptv3_voxelize: null pointer");
    const size_t need = ptv3_voxelize_workspace_bytes(n);
    PTV3_REQUIRE(workspace_bytes >= need, PTV3_ERR_WORKSPACE, "ptv3_voxelize: workspace %zu < %zu bytes",
                 workspace_bytes, need);
    cudaStream_t stream = (cudaStream_t)stream_;
    const VoxelScratch v = vz_scratch(n, workspace);
    const int64_t clear = (reinterpret_cast<char*>(v.slot_of) - reinterpret_cast<char*>(v.table)) / 16;
    const uint32_t slots = 2 * vz_pairs(n);
    const dim3 points((unsigned)((n + 255) / 256)), tiles(ceil_div(n, VZ_TILE));
    vz_origin_init_kernel<<<1, 32, 0, stream>>>(origin);
    launch_dependent(vz_prepare_kernel, dim3((unsigned)std::min<int64_t>((n + 1023) / 1024, SMS * 8)), dim3(256), 0,
                     stream, coord, n, ((uintptr_t)coord & 15) == 0, origin, reinterpret_cast<uint4*>(v.table), clear);
    launch_dependent(vz_insert_kernel, points, dim3(256), (size_t)n_scenes * sizeof(int64_t), stream, coord, n,
                     grid_size, origin, offset, n_scenes, v.table, vz_pairs(n), v.slot_of, v.claimed, status);
    launch_dependent(vz_first_kernel, tiles, dim3(256), 0, stream, v.slot_of, n, v.table, slots, v.kept,
                     v.tile_sums, v.group_sums, v.claimed, status, count, count_host);
    launch_dependent(vz_number_kernel, tiles, dim3(256), 0, stream, v.slot_of, n, v.kept, v.tile_sums,
                     v.group_sums, v.table, slots, keep, point2voxel);
    launch_dependent(vz_inverse_kernel, dim3((unsigned)((n + 256 * VZ_ITEMS - 1) / (256 * VZ_ITEMS))), dim3(256), 0,
                     stream, v.slot_of, n, v.table, slots, offset, n_scenes, count, point2voxel, new_offset);
    count_launches(6);
    return check_launch("ptv3_voxelize");
}

extern "C" int ptv3_voxelize_rows(const int64_t* keep, int64_t m, const float* coord, const float* origin, float grid_size,
                                  const void* feat, int64_t feat_row_bytes, float* out_coord, int32_t* out_grid,
                                  void* out_feat, void* stream_)
{
    PTV3_REQUIRE(m >= 0 && feat_row_bytes >= 0 && feat_row_bytes < (1 << 20), PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_voxelize_rows: bad sizes");
    if (m == 0) return PTV3_OK;
    PTV3_REQUIRE(keep && coord && origin && out_coord && out_grid && (feat_row_bytes == 0 || (feat && out_feat)),
                 PTV3_ERR_INVALID_ARGUMENT, "ptv3_voxelize_rows: null pointer");
    cudaStream_t stream = (cudaStream_t)stream_;
    const uintptr_t align = (uintptr_t)feat | (uintptr_t)out_feat | (uintptr_t)feat_row_bytes;
#define VZ_GATHER(W)                                                                                          \
    do {                                                                                                      \
        const uint32_t words = (uint32_t)(feat_row_bytes / (int64_t)sizeof(W));                               \
        const int rows = std::max(1, std::min<int>(VZ_ROWS, VZ_PIECES / (int)(3 + words)));                   \
        launch_dependent(vz_gather_kernel<W>, dim3((unsigned)((m + rows - 1) / rows)), dim3(256), 0, stream,   \
                         keep, m, coord, origin, grid_size, (const W*)feat, words, rows, out_coord,           \
                         out_grid, (W*)out_feat);                                                             \
    } while (0)
    if (align % 16 == 0)
        VZ_GATHER(uint4);
    else if (align % 8 == 0)
        VZ_GATHER(uint2);
    else if (align % 4 == 0)
        VZ_GATHER(uint32_t);
    else if (align % 2 == 0)
        VZ_GATHER(uint16_t);
    else
        VZ_GATHER(uint8_t);
#undef VZ_GATHER
    count_launches(1);
    return check_launch("ptv3_voxelize_rows");
}
