// Index-side launches that the one-call backbone queues itself.
#pragma once
#include "bn.cuh"
#include "common.cuh"
#include "voxel_index.cuh"

namespace ptv3 {

// ptv3_pool_plan that also writes the cumulative scene sizes of the pooled level (n_scenes int64) and, unless NULL, its
// (batch, x, y, z) rows (16-byte aligned)
int pool_plan(const int64_t* code, const int64_t* order, const int32_t* grid_coord, const int64_t* batch, int k,
              int64_t n, int n_scenes, int pooling_depth, const int* row_perm, int64_t* cluster, int64_t* idx_ptr,
              int64_t* head, int64_t* pooled_code, int64_t* pooled_order, int64_t* pooled_inverse,
              int32_t* pooled_grid_coord, int64_t* pooled_batch, int64_t* meta, int64_t* meta_host,
              int64_t* pooled_offset, int32_t* pooled_indices, uint32_t* status, void* workspace, size_t workspace_bytes,
              cudaStream_t stream);

// ptv3_batch_indices (indices only) with a voxel index cleared and the network's BatchNorm layers done beside it
int batch_indices_and_norms(const int64_t* offset, int n_scenes, const int32_t* grid_coord, int64_t n, int32_t* indices,
                            const VoxelClear& index, const BnJobs& norms, cudaStream_t stream);

// ptv3_pad_plan with a voxel index cleared beside it
int pad_plan(const int64_t* offset, int n_scenes, int patch, int64_t n, int64_t n_pad, int n_seq, int64_t* pad,
             int64_t* unpad, int32_t* cu_seqlens, uint32_t* status, const VoxelClear& index, cudaStream_t stream);

// kernel map of a voxel set whose index exists already
int kmap_from_index(const VoxelIndex& vi, const int32_t* indices, int64_t n, int ksize, const int64_t* row_order,
                    int32_t* nbr, uint32_t* status, cudaStream_t stream);

// stem convolution (+ BatchNorm + GELU) on an existing voxel index; `scratch` holds
// conv_direct_scratch_bytes(n, ksize) bytes
size_t conv_direct_scratch_bytes(int64_t n, int ksize);
int conv_direct_from_index(const VoxelIndex& vi, const void* feat, const int32_t* indices, const void* weight,
                           const float* bn_scale, const float* bn_shift, void* out, const int64_t* row_order,
                           int64_t n, int c_in, int c_out, int ksize, int dtype, uint32_t* status, void* weight_scratch,
                           cudaStream_t stream);

}  // namespace ptv3
