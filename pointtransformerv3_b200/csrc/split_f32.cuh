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
// (The split and its six products: Henry, Tang and Heinecke, "Leveraging the bfloat16 Artificial Intelligence
// Datatype for Higher-Precision Computations", 2019; small products in accumulators of their own, because of the
// truncation: Ootomo and Yokota, "Recovering Single Precision Accuracy from Tensor Cores", 2022.)
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mma_util.cuh"

namespace ptv3 {

// Stored are the three parts where a piece is whole 64-column chunks (the products then read a part as
// often as they need it), all six pieces otherwise.
__host__ __device__ constexpr int split_stored(int k) { return k % 64 == 0 ? 3 : 6; }
// column of chunk `c` (64 columns of the six pieces) in a stored row of A or of B
__host__ __device__ __forceinline__ int split_column_a(int c, int k)
{
    if (k % 64) return c * 64;
    const int piece = c * 64 / k;
    return (piece < 3 ? 0 : piece < 5 ? 1 : 2) * k + c * 64 % k;
}
__host__ __device__ __forceinline__ int split_column_b(int c, int k)
{
    if (k % 64) return c * 64;
    const int piece = c * 64 / k;
    return (piece < 3 ? piece : piece < 5 ? piece - 3 : 0) * k + c * 64 % k;
}
// column of part p of a stored row of A; of a row of B it is p k either way
__host__ __device__ __forceinline__ int split_part_a(int p, int k) { return (k % 64 == 0 ? p : p == 0 ? 0 : 2 * p + 1) * k; }

constexpr int SPLIT_MAIN = 3, SPLIT_ACCS = SPLIT_MAIN + 1;

__device__ __forceinline__ void split3(float x, __nv_bfloat16& a, __nv_bfloat16& b, __nv_bfloat16& c)
{
    a = __float2bfloat16_rn(x);
    const float r = __fsub_rn(x, __bfloat162float(a));
    b = __float2bfloat16_rn(r);
    c = __float2bfloat16_rn(__fsub_rn(r, __bfloat162float(b)));
}

// eight values of an A row: `row` is the stored row, `c` their column, `k` the width of a piece
__device__ __forceinline__ void split_store8(__nv_bfloat16* row, int c, int k, const float* y, bool weight = false)
{
    uint4 p[3];
    __nv_bfloat16* q = reinterpret_cast<__nv_bfloat16*>(p);
#pragma unroll
    for (int i = 0; i < 8; ++i) split3(y[i], q[i], q[8 + i], q[16 + i]);
    if (k % 64 == 0) {
#pragma unroll
        for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(row + i * k + c) = p[i];
    } else {
        const int pa[6] = {0, 0, 0, 1, 1, 2}, pb[6] = {0, 1, 2, 0, 1, 0};
#pragma unroll
        for (int i = 0; i < 6; ++i) *reinterpret_cast<uint4*>(row + i * k + c) = p[weight ? pb[i] : pa[i]];
    }
}

// four values of an A row
__device__ __forceinline__ void split_store4(__nv_bfloat16* row, int c, int k, const float* y)
{
    uint2 p[3];
    __nv_bfloat16* q = reinterpret_cast<__nv_bfloat16*>(p);
#pragma unroll
    for (int i = 0; i < 4; ++i) split3(y[i], q[i], q[4 + i], q[8 + i]);
    if (k % 64 == 0) {
#pragma unroll
        for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(row + i * k + c) = p[i];
    } else {
        const int part[6] = {0, 0, 0, 1, 1, 2};
#pragma unroll
        for (int i = 0; i < 6; ++i) *reinterpret_cast<uint2*>(row + i * k + c) = p[part[i]];
    }
}

// rows x k floats -> rows x split_stored(k) k bf16, as A rows
int launch_split_f32(const float* x, int64_t rows, int k, void* out, cudaStream_t stream);
// ... as B rows, any number of weights
struct SplitWeight {
    const float* x;
    int64_t rows;
    int k;
    void* out;
};
int launch_split_weights(const SplitWeight* w, int count, cudaStream_t stream);

}  // namespace ptv3
