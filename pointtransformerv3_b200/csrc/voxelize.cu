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
// bytes each, two probes per point).  Here the grid coordinates are recomputed where they are needed,
// the table has exactly two slots per point (57 MB at 2.4 M points: it stays in the 126 MB L2), a point
// remembers its slot instead of probing again, and the voxel count reaches the host from the scan,
// before the point -> voxel map and the outputs are made.

// minimum over the points, four points (three 16-byte loads) per step, one atomic per block and axis
__global__ void __launch_bounds__(256) vz_min_kernel(const float* __restrict__ coord, int64_t n, bool vec,
                                                     float* __restrict__ origin)
{
    const float inf = __int_as_float(0x7f800000);
    float m[3] = {inf, inf, inf};
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
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

constexpr uint32_t VZ_NO_SLOT = 0xffffffffu;

// every point claims the slot of its voxel; the lowest row wins
__global__ void __launch_bounds__(256) vz_insert_kernel(const float* __restrict__ coord, int64_t n, float grid_size,
                                                        const float* __restrict__ origin,
                                                        const int64_t* __restrict__ offset, int B,
                                                        unsigned long long* __restrict__ keys,
                                                        uint32_t* __restrict__ vals, uint32_t cap,
                                                        uint32_t* __restrict__ slot_of, uint32_t* __restrict__ status)
{
    extern __shared__ int64_t ends[];
    for (int s = threadIdx.x; s < B; s += blockDim.x) ends[s] = offset[s];
    __syncthreads();
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    int lo = 0, hi = B - 1;          // first scene whose end lies beyond i
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (ends[mid] > i) hi = mid; else lo = mid + 1;
    }
    uint64_t key;
    uint32_t at = VZ_NO_SLOT;        // outside the key range: reported, and the point keeps itself
    if (km_key(lo, vz_cell(coord[3 * i], origin[0], grid_size), vz_cell(coord[3 * i + 1], origin[1], grid_size),
               vz_cell(coord[3 * i + 2], origin[2], grid_size), key)) {
        uint32_t slot = (uint32_t)(((km_mix(key) >> 32) * cap) >> 32);
        uint32_t probe = 0;
        for (; probe < cap; ++probe) {
            // a plain look first: most points of a voxel come after its first
            unsigned long long prev = *reinterpret_cast<volatile unsigned long long*>(&keys[slot]);
            if (prev == KM_EMPTY) prev = atomicCAS(&keys[slot], KM_EMPTY, key);
            if (prev == KM_EMPTY || prev == key) {
                atomicMin(&vals[slot], (uint32_t)i);
                at = slot;
                break;
            }
            slot = slot + 1 == cap ? 0 : slot + 1;
        }
        if (probe == cap) atomicOr(status, PTV3_STATUS_PROBE_LIMIT);
    } else {
        atomicOr(status, PTV3_STATUS_BAD_INDEX);
    }
    slot_of[i] = at;
}

// first row of every point's voxel (over its slot), and the number of kept points per scan tile
__global__ void __launch_bounds__(SC_THREADS) vz_first_kernel(uint32_t* __restrict__ slot_first, int64_t n,
                                                              const uint32_t* __restrict__ vals,
                                                              uint32_t* __restrict__ tile_sums)
{
    __shared__ uint32_t warp_sums[SC_THREADS / 32];
    const int64_t base = (int64_t)blockIdx.x * SC_TILE;
    uint32_t c = 0;
#pragma unroll
    for (int it = 0; it < SC_ITEMS; ++it) {
        const int64_t j = base + it * SC_THREADS + threadIdx.x;
        if (j < n) {
            const uint32_t s = slot_first[j];
            const uint32_t f = s == VZ_NO_SLOT ? (uint32_t)j : vals[s];
            slot_first[j] = f;
            c += f == (uint32_t)j ? 1u : 0u;
        }
    }
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t s = 0;
        for (int w = 0; w < SC_THREADS / 32; ++w) s += warp_sums[w];
        tile_sums[blockIdx.x] = s;
    }
}

// scan of the tile sums; the total and the status word go to the host at once
__global__ void __launch_bounds__(1024) vz_scan_kernel(uint32_t* __restrict__ tile_sums, int ntiles,
                                                       uint32_t* __restrict__ total, int64_t* host,
                                                       const uint32_t* __restrict__ status)
{
    __shared__ uint32_t warp_sums[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (int base = 0; base < ntiles; base += 1024) {
        const int t = base + threadIdx.x;
        const uint32_t v = t < ntiles ? tile_sums[t] : 0u;
        uint32_t inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += u;
        }
        if (lane == 31) warp_sums[warp] = inc;
        __syncthreads();
        uint32_t before = 0, all = 0;
        for (int w = 0; w < 32; ++w) {
            before += w < warp ? warp_sums[w] : 0u;
            all += warp_sums[w];
        }
        if (t < ntiles) tile_sums[t] = carry + before + inc - v;
        carry += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        *total = carry;
        host[0] = carry;
        host[1] = *status;
        __threadfence_system();
        *reinterpret_cast<volatile int64_t*>(&host[2]) = 1;
        __threadfence_system();
    }
}

// output rows: coordinates, grid coordinates (recomputed) and features of the kept points; a row of
// features is `words` pieces of W
template <typename W>
__global__ void __launch_bounds__(256) vz_gather_kernel(const int64_t* __restrict__ keep, int64_t m,
                                                        const float* __restrict__ coord,
                                                        const float* __restrict__ origin, float grid_size,
                                                        const W* __restrict__ feat, int words,
                                                        float* __restrict__ out_coord, int32_t* __restrict__ out_grid,
                                                        W* __restrict__ out_feat)
{
    const int lanes = 3 + words;                 // three axes, then the feature words
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= m * lanes) return;
    const int64_t row = e / lanes;
    const int a = (int)(e - row * lanes);
    const int64_t src = keep[row];
    if (a < 3) {
        const float c = coord[3 * src + a];
        out_coord[3 * row + a] = c;
        out_grid[3 * row + a] = vz_cell(c, origin[a], grid_size);
    } else {
        out_feat[row * words + a - 3] = feat[src * words + a - 3];
    }
}

static uint32_t vz_capacity(int64_t n) { return (uint32_t)(2 * n < 1024 ? 1024 : 2 * n); }

static size_t vz_scratch(int64_t n, void* base, unsigned long long** keys, uint32_t** vals, uint32_t** first,
                         uint32_t** rank, uint32_t** tile_sums, uint32_t** total)
{
    const uint32_t cap = vz_capacity(n);
    Carver cv(base);
    *keys = cv.take<unsigned long long>(cap);
    *vals = cv.take<uint32_t>(cap);              // cleared together with the keys
    *first = cv.take<uint32_t>(n);
    *rank = cv.take<uint32_t>(n);
    *tile_sums = cv.take<uint32_t>(ceil_div(n, SC_TILE));
    *total = cv.take<uint32_t>(1);
    return cv.off;
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
    unsigned long long* k;
    uint32_t* p[5];
    return vz_scratch(n, nullptr, &k, &p[0], &p[1], &p[2], &p[3], &p[4]);
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
    unsigned long long* keys;
    uint32_t *vals, *first, *rank, *tile_sums, *total;
    vz_scratch(n, workspace, &keys, &vals, &first, &rank, &tile_sums, &total);
    const uint32_t cap = vz_capacity(n);
    const size_t clear = (size_t)(reinterpret_cast<char*>(first) - reinterpret_cast<char*>(keys));
    if (cudaMemsetAsync(keys, 0xff, clear, stream) != cudaSuccess) return check_launch("ptv3_voxelize: table reset");
    vox_origin_init_kernel<<<1, 32, 0, stream>>>(origin);
    const unsigned blocks = (unsigned)((n + 255) / 256);
    vz_min_kernel<<<(unsigned)std::min<int64_t>((n + 1023) / 1024, SMS * 8), 256, 0, stream>>>(
        coord, n, ((uintptr_t)coord & 15) == 0, origin);
    vz_insert_kernel<<<blocks, 256, (size_t)n_scenes * sizeof(int64_t), stream>>>(
        coord, n, grid_size, origin, offset, n_scenes, keys, vals, cap, first, status);
    const int ntiles = ceil_div(n, SC_TILE);
    vz_first_kernel<<<ntiles, SC_THREADS, 0, stream>>>(first, n, vals, tile_sums);
    vz_scan_kernel<<<1, 1024, 0, stream>>>(tile_sums, ntiles, total, count_host, status);
    const FirstFlag flag{first};
    scan_apply_kernel<FirstFlag, KeepSink><<<dim3(ntiles, 1), SC_THREADS, 0, stream>>>(flag, KeepSink{keep, rank}, n,
                                                                                        ntiles, tile_sums);
    vox_inverse_kernel<<<blocks, 256, 0, stream>>>(first, rank, n, total, offset, n_scenes, point2voxel, new_offset,
                                                   count);
    count_launches(7);
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
        const int words = (int)(feat_row_bytes / (int64_t)sizeof(W));                                         \
        vz_gather_kernel<W><<<(unsigned)((m * (3 + words) + 255) / 256), 256, 0, stream>>>(                    \
            keep, m, coord, origin, grid_size, (const W*)feat, words, out_coord, out_grid, (W*)out_feat);     \
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
