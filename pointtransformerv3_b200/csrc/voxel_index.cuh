// Two-level voxel index: a hash table of 4 x 4 x 4 blocks whose values point at
// 64-entry cell tables (cell -> row of the voxel, VI_NO_ROW where empty).
// A (2r+1)^3 neighbourhood with r <= 2 touches at most 2 blocks per axis, so a voxel
// needs 8 hash probes instead of one per kernel offset; each offset then costs a
// few integer operations and one load from a 256-byte cell table.  Duplicate
// voxels resolve to the lowest row.
#pragma once
#include "common.cuh"
#include "kmap.cuh"

namespace ptv3 {

constexpr uint32_t VI_NO_ROW = 0xffffffffu;

__device__ __forceinline__ bool vi_block_key(int b, int bx, int by, int bz, uint64_t& key)
{
    if ((unsigned)b > 0xfffeu || (unsigned)bx > 0x3fffu || (unsigned)by > 0x3fffu || (unsigned)bz > 0x3fffu)
        return false;
    key = ((uint64_t)b << 48) | ((uint64_t)bx << 32) | ((uint64_t)by << 16) | (uint64_t)bz;
    return true;
}

// (plain pointers: kernels that start early read through them, see common.cuh)
__device__ __forceinline__ uint32_t vi_block_lookup(const unsigned long long* keys, const uint32_t* vals,
                                                    uint64_t cap_mask, uint64_t key, bool* overflow)
{
    uint64_t slot = km_mix(key) & cap_mask;
    for (uint64_t probe = 0; probe <= cap_mask; ++probe) {
        const unsigned long long kk = keys[slot];
        if (kk == key) return vals[slot];
        if (kk == KM_EMPTY) return VI_NO_ROW;
        slot = (slot + 1) & cap_mask;
    }
    *overflow = true;
    return VI_NO_ROW;
}


struct VoxelIndex {
    const unsigned long long* keys;   // block hash table
    const uint32_t* vals;             // block -> cell table id
    uint64_t cap_mask;
    const uint32_t* cells;            // 64 rows per table
};

// cell of coordinate (x, y, z) inside its block
__device__ __forceinline__ int vi_cell(int x, int y, int z) { return (x & 3) << 4 | (y & 3) << 2 | (z & 3); }

// The words that an index starts from: empty keys (pairs of them) and no block taken.  Any kernel ahead of
// `fill_voxel_index` may write them: `clear` by all its threads, nothing for a job of none.
struct VoxelClear {
    ulonglong2* keys;
    int64_t pairs;
    uint32_t* counter;
    __device__ void clear() const
    {
        const int64_t first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
        for (int64_t i = first; i < pairs; i += (int64_t)gridDim.x * blockDim.x)
            keys[i] = make_ulonglong2(KM_EMPTY, KM_EMPTY);
        if (first == 0 && counter) *counter = 0;
    }
};

// blocks of 256 threads for a kernel that does nothing else
inline unsigned voxel_clear_blocks(const VoxelClear& job)
{
    const int64_t blocks = (job.pairs + 255) / 256;
    return (unsigned)(blocks < SMS * 8 ? blocks : SMS * 8);
}

size_t voxel_index_bytes(int64_t n);
// lays the index of n voxels out in `workspace`
VoxelClear place_voxel_index(int64_t n, void* workspace, VoxelIndex* out);
// enters the n voxels (rows of (batch, x, y, z) int32) into a cleared index
int fill_voxel_index(const VoxelIndex& vi, const VoxelClear& cleared, const int32_t* indices, int64_t n, uint32_t* status,
                     cudaStream_t stream);
// all of it: places, clears and fills the index
int build_voxel_index(const int32_t* indices, int64_t n, void* workspace, uint32_t* status, cudaStream_t stream,
                      VoxelIndex* out);

}  // namespace ptv3
