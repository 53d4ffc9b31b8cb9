#include "split_f32.cuh"
#include "common.cuh"

namespace ptv3 {

// a thread splits eight columns; bandwidth bound: 4 bytes in, 6 out
template <bool WEIGHT>
__global__ void __launch_bounds__(256) split_f32_kernel(const float* __restrict__ x, int64_t n8, int k,
                                                        __nv_bfloat16* __restrict__ out)
{
    // (the product behind the weight form fetches weights before it waits for anything)
    if (!WEIGHT) pdl_launch_next();
    pdl_wait();
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= n8) return;
    const int per = k / 8;
    const int64_t row = e / per;
    const int c = (int)(e - row * per) * 8;
    const float4 v0 = reinterpret_cast<const float4*>(x)[2 * e], v1 = reinterpret_cast<const float4*>(x)[2 * e + 1];
    const float y[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    split_store8(out + row * split_stored(k) * k, c, k, y, WEIGHT);
}

int launch_split_f32(const float* x, int64_t rows, int k, bool weight, void* out, cudaStream_t stream)
{
    const int64_t n8 = rows * (k / 8);
    const dim3 grid((unsigned)((n8 + 255) / 256));
    if (weight)
        launch_dependent(split_f32_kernel<true>, grid, dim3(256), 0, stream, x, n8, k, (__nv_bfloat16*)out);
    else
        launch_dependent(split_f32_kernel<false>, grid, dim3(256), 0, stream, x, n8, k, (__nv_bfloat16*)out);
    count_launches(1);
    return check_launch("fp32 split");
}

}  // namespace ptv3

extern "C" int ptv3_split_f32(const float* x, int64_t rows, int k, int weight, void* out, void* stream)
{
    using namespace ptv3;
    PTV3_REQUIRE(rows >= 0 && k >= 8 && k % 8 == 0, PTV3_ERR_INVALID_ARGUMENT, "ptv3_split_f32: bad sizes");
    if (rows == 0) return PTV3_OK;
    PTV3_REQUIRE(x && out && (((uintptr_t)x | (uintptr_t)out) & 15) == 0, PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_split_f32: tensors must be 16-byte aligned");
    return launch_split_f32(x, rows, k, weight != 0, out, (cudaStream_t)stream);
}
