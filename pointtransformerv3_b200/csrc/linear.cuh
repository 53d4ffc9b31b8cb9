// Linear layers as the one-call block and backbone queue them (linear_small.cu, linear_tc05.cu, gemm_tc05.cu,
// mlp_tc05.cu, block.cu): the entry points of the same names, with what the caller knows of the weights.
//
// `settled`: nothing in flight on the stream writes weights, biases or norm parameters.  The kernels then fetch
// them before they wait for the launch ahead of them.  That holds inside ptv3_backbone_fwd, whose first kernel on
// the stream is an ordinary launch: it starts when everything before it has finished, and every later kernel
// starts after it.  An entry point of its own cannot know: its weights may be what the call before it
// computes, and a distance of several launches does not help, because launches in between let theirs start early too.
//
// `planned`: nothing in flight writes the geometry that a convolution or attention reads (neighbours, orders, patch
// layout).  The kernels then look it up before that wait.  Inside ptv3_backbone_fwd it is made on the planning stream,
// for whose event the main stream waits before the first kernel of a level; only that kernel, the first one
// behind the event, must not count on it.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/ptv3_b200.h"

namespace ptv3 {

// Whether the short form (linear_small.cu) is the faster one for n rows, with GELU or a residual (`epilogue`) or
// without; bf16, 16-byte aligned rows
bool linear_small_wanted(int64_t n, int k, int n_out, bool epilogue);

// out = [residual +] act(x W^T + b) by the short form
int launch_linear_small(const void* x, const void* w, const void* bias, const void* residual, void* out, int64_t n, int k,
                        int n_out, int gelu, bool settled, uint32_t* status, cudaStream_t stream);

// fp32 Linear on split operands (split_f32.cuh); k and n_out multiples of 32.  The result goes to `out`, or as
// split rows to `split_out`.
int launch_linear_split(const void* xs, const void* ws, const float* bias, const float* residual, float* out,
                        void* split_out, int64_t n, int k, int n_out, int gelu, bool settled, uint32_t* status,
                        cudaStream_t stream);

int linear_fwd(const void* x, const void* weight, const void* bias, void* out, int64_t n, int k, int n_out, int dtype,
               bool settled, uint32_t* status, cudaStream_t stream);
int linear_ln_fwd(const void* x, const void* weight, const void* bias, const void* residual, const void* ln1_weight,
                  const void* ln1_bias, float ln1_eps, void* sum_out, const void* ln2_weight, const void* ln2_bias,
                  float ln2_eps, void* norm_out, int64_t n, int channels, int dtype, bool settled, uint32_t* status,
                  cudaStream_t stream);
int gemm_fwd(const void* x, const void* weight, const void* bias, const void* residual, void* out, int64_t n, int k,
             int n_out, int gelu, int dtype, bool settled, uint32_t* status, cudaStream_t stream);
int mlp_fwd(const void* x, const void* fc1_weight, const void* fc1_bias, const void* fc2_weight, const void* fc2_bias,
            const void* residual, void* out, int64_t n, int channels, int hidden, int dtype, bool settled,
            uint32_t* status, cudaStream_t stream);

// ptv3_add_layernorm_fwd in fp32 whose second norm leaves as split rows (split_f32.cuh)
int add_layernorm_split(const float* x, const float* residual, const float* ln1_weight, const float* ln1_bias, float ln1_eps,
                        float* sum_out, const float* ln2_weight, const float* ln2_bias, float ln2_eps, void* norm_split,
                        int64_t n, int channels, cudaStream_t stream);

// ptv3_attention_fwd in fp32 whose result leaves as split rows, where attention_splits says that it can
bool attention_splits(const void* qkv, int64_t n, int n_seq, int channels, int heads, int algo);
int attention_split(const void* qkv, const int64_t* order, const int64_t* pad, const int64_t* unpad,
                    const int32_t* cu_seqlens, void* split_out, int64_t n, int n_seq, int max_seqlen, int channels, int heads,
                    float scale, uint32_t* status, cudaStream_t stream);
int attention_fwd(const void* qkv, const int64_t* order, const int64_t* pad, const int64_t* unpad, const int32_t* cu_seqlens,
                  void* out, int64_t n, int n_seq, int max_seqlen, int channels, int heads, float scale, int dtype,
                  int algo, bool planned, uint32_t* status, cudaStream_t stream);
int subm_conv_fwd(const void* feat, const int32_t* nbr, const void* weight, const void* bias, void* out,
                  const int64_t* row_order, int64_t n, int c_in, int c_out, int kernel_volume, int dtype, int algo,
                  bool planned, uint32_t* status, cudaStream_t stream);

int block_fwd(const ptv3_block_args* a, bool settled, bool planned, cudaStream_t stream);
int pool_stage_fwd(const void* x, const void* weight, const void* bias, const float* coord, const int64_t* indices,
                   const int64_t* idx_ptr, int64_t n, int64_t m, int c_in, int c_out, const float* bn_scale,
                   const float* bn_shift, void* out, float* coord_out, int reduce, int dtype, bool settled,
                   uint32_t* status, void* workspace, size_t workspace_bytes, cudaStream_t stream);
int unpool_stage_fwd(const void* skip_feat, const void* child_feat, const void* w_skip, const void* b_skip,
                     const void* w_child, const void* b_child, const int64_t* cluster, int64_t n, int64_t m, int c_skip,
                     int c_child, int c_out, const float* skip_scale, const float* skip_shift, const float* child_scale,
                     const float* child_shift, void* out, void* skip_act, int dtype, bool settled, uint32_t* status,
                     void* workspace, size_t workspace_bytes, cudaStream_t stream);

}  // namespace ptv3
