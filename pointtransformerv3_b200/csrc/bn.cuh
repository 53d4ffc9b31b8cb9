// BatchNorm in eval mode as scale and shift per channel, a block per layer (see ptv3_bn_affine).
#pragma once
#include "common.cuh"

namespace ptv3 {

constexpr int BN_JOBS = 48;          // 3.1 KB of the 4 KB of kernel parameters
struct BnJobs {
    ptv3_bn_args layer[BN_JOBS];
    float* out[BN_JOBS];
    int count;
};
static_assert(sizeof(BnJobs) <= 3584, "kernel parameters, with those of batch_indices_kernel");

// the first of `count` layers (at most BN_JOBS), checked; each has its scales and shifts behind one another in `out`
int bn_jobs(const ptv3_bn_args* layers, int count, float* out, BnJobs* jobs);

__device__ __forceinline__ float bn_value(const void* p, int dtype, int c, float absent)
{
    if (!p) return absent;
    return dtype == PTV3_DTYPE_F32 ? static_cast<const float*>(p)[c]
                                   : __bfloat162float(static_cast<const __nv_bfloat16*>(p)[c]);
}

__device__ __forceinline__ void bn_layer(const BnJobs& jobs, int i)
{
    const ptv3_bn_args& l = jobs.layer[i];
    float* out = jobs.out[i];
    for (int c = threadIdx.x; c < l.channels; c += blockDim.x) {
        const float scale = bn_value(l.weight, l.weight_dtype, c, 1.f) *
                            __frsqrt_rn(bn_value(l.var, l.var_dtype, c, 1.f) + l.eps);
        out[c] = scale;
        out[l.channels + c] = bn_value(l.bias, l.bias_dtype, c, 0.f) - bn_value(l.mean, l.mean_dtype, c, 0.f) * scale;
    }
}

}  // namespace ptv3
