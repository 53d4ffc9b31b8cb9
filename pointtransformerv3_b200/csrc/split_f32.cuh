// fp32 products on the bf16 tensor cores.
//
// A float is the exact sum of three bf16 values (8 + 8 + 8 significant bits): x = x1 + x2 + x3, each the
// rounded rest of what the ones before it leave.  Of the nine products of two such sums the six with
// i + j <= 4 are kept; the others are below 2^-24 of the whole, the rounding of one fp32 product.  A matrix
// product of floats then is one bf16 product over six times the inner dimension, accumulated in fp32:
//     A rows  [x1 x1 x1 x2 x2 x3]     B rows  [w1 w2 w3 w1 w2 w1]        (pieces of k columns each)
// The tensor core truncates where an fp32 addition rounds, once per 16 columns, so a long sum in one
// accumulator would lose more than a chain of FMAs: the leading piece goes to SPLIT_MAIN accumulators in turn,
// the five small ones to one of their own (their truncation is 2^-8 of the leading one's), and the epilogue
// adds them in fp32.  Against float64 the products come out as close as CUDA-core fp32.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mma_util.cuh"

namespace ptv3 {

constexpr int SPLIT_MAIN = 3, SPLIT_ACCS = SPLIT_MAIN + 1;

__device__ __forceinline__ void split3(float x, __nv_bfloat16& a, __nv_bfloat16& b, __nv_bfloat16& c)
{
    a = __float2bfloat16_rn(x);
    const float r = __fsub_rn(x, __bfloat162float(a));
    b = __float2bfloat16_rn(r);
    c = __float2bfloat16_rn(__fsub_rn(r, __bfloat162float(b)));
}

// eight values of an A row: `at` points at their column of the first piece, `k` is the width of a piece
__device__ __forceinline__ void split_store8(__nv_bfloat16* at, int k, const float* y)
{
    uint4 p[3];
    __nv_bfloat16* q = reinterpret_cast<__nv_bfloat16*>(p);
#pragma unroll
    for (int i = 0; i < 8; ++i) split3(y[i], q[i], q[8 + i], q[16 + i]);
    const int part[6] = {0, 0, 0, 1, 1, 2};
#pragma unroll
    for (int i = 0; i < 6; ++i) *reinterpret_cast<uint4*>(at + (int64_t)i * k) = p[part[i]];
}

// rows x k floats -> rows x 6k bf16; `weight`: in the order of a B row
int launch_split_f32(const float* x, int64_t rows, int k, bool weight, void* out, cudaStream_t stream);

}  // namespace ptv3
