// Linear layers on short inputs (linear_small.cu): bf16, 16-byte aligned rows.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ptv3 {

// Whether the short form is the faster one for n rows (see linear_small.cu for the measurements)
bool linear_small_wanted(int64_t n, int k, int n_out);
bool linear_ln_small_wanted(int64_t n, int c);

// out = [residual +] act(x W^T + b)
int launch_linear_small(const void* x, const void* w, const void* bias, const void* residual, void* out, int64_t n, int k,
                        int n_out, int gelu, uint32_t* status, cudaStream_t stream);
// sum = residual + LN1(x W^T + b) (without LN1 when ln1_w is NULL), norm = LN2(sum); sum_out may be NULL
int launch_linear_ln_small(const void* x, const void* w, const void* bias, const void* residual, const void* ln1_w,
                           const void* ln1_b, float eps1, void* sum_out, const void* ln2_w, const void* ln2_b, float eps2,
                           void* norm_out, int64_t n, int c, uint32_t* status, cudaStream_t stream);

// fp32 Linear on split operands (split_f32.cuh); k and n_out multiples of 32.  The result goes to `out`, or as
// split rows to `split_out`.
int launch_linear_split(const void* xs, const void* ws, const float* bias, const float* residual, float* out,
                        void* split_out, int64_t n, int k, int n_out, int gelu, uint32_t* status, cudaStream_t stream);

}  // namespace ptv3
