// Linear layers on short inputs (linear_small.cu): bf16, 16-byte aligned rows.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ptv3 {

// Whether the short form is the faster one for n rows (see linear_small.cu for the measurements)
bool linear_small_wanted(int64_t n, int k, int n_out);

// out = [residual +] act(x W^T + b)
int launch_linear_small(const void* x, const void* w, const void* bias, const void* residual, void* out, int64_t n, int k,
                        int n_out, int gelu, uint32_t* status, cudaStream_t stream);

// fp32 Linear on split operands (split_f32.cuh); k and n_out multiples of 32.  The result goes to `out`, or as
// split rows to `split_out`.
int launch_linear_split(const void* xs, const void* ws, const float* bias, const float* residual, float* out,
                        void* split_out, int64_t n, int k, int n_out, int gelu, uint32_t* status, cudaStream_t stream);

}  // namespace ptv3
