#include "split_f32.cuh"
#include "common.cuh"

namespace ptv3 {

// rows of features: a thread splits eight columns; bandwidth bound: 4 bytes in, 6 out
__global__ void __launch_bounds__(256) split_f32_kernel(const float* x, int64_t n8, int k, __nv_bfloat16* out)
{
    pdl_launch_next();
    pdl_wait();
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= n8) return;
    const int per = k / 8;
    const int64_t row = e / per;
    const int c = (int)(e - row * per) * 8;
    const float4 v0 = reinterpret_cast<const float4*>(x)[2 * e], v1 = reinterpret_cast<const float4*>(x)[2 * e + 1];
    const float y[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    split_store8(out + row * split_stored(k) * k, c, k, y, false);
}

// Weights, many to a launch: a block takes 256 x 8 values of one of them.  Neither launched ahead of the work
// before it nor letting the kernel behind it start early: the Linear kernels fetch weights before they wait.
constexpr int SPLIT_JOBS = 144;          // those of the default network; 4 036 of the 4 096 bytes of kernel parameters
struct SplitJobs {
    const float* x[SPLIT_JOBS];
    __nv_bfloat16* out[SPLIT_JOBS];
    uint32_t n8[SPLIT_JOBS], first[SPLIT_JOBS];      // groups of eight values; first block
    int k[SPLIT_JOBS];
    int count;
};
static_assert(sizeof(SplitJobs) <= 4096, "kernel parameters");

__global__ void __launch_bounds__(256) split_weights_kernel(const __grid_constant__ SplitJobs jobs)
{
    int j = 0;
    for (int end = jobs.count; end - j > 1;) {
        const int mid = (j + end) / 2;
        if (jobs.first[mid] <= blockIdx.x) j = mid; else end = mid;
    }
    const uint32_t e = (blockIdx.x - jobs.first[j]) * 256 + threadIdx.x;
    if (e >= jobs.n8[j]) return;
    const int k = jobs.k[j];
    const uint32_t per = (uint32_t)k / 8, row = e / per;
    const float4* x = reinterpret_cast<const float4*>(jobs.x[j]) + 2 * (size_t)e;
    const float4 v0 = x[0], v1 = x[1];
    const float y[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    split_store8(jobs.out[j] + (size_t)row * split_stored(k) * k, (int)(e - row * per) * 8, k, y, true);
}

int launch_split_f32(const float* x, int64_t rows, int k, void* out, cudaStream_t stream)
{
    const int64_t n8 = rows * (k / 8);
    launch_dependent(split_f32_kernel, dim3((unsigned)((n8 + 255) / 256)), dim3(256), 0, stream, x, n8, k,
                     (__nv_bfloat16*)out);
    count_launches(1);
    return check_launch("fp32 split");
}

int launch_split_weights(const SplitWeight* w, int count, cudaStream_t stream)
{
    while (count > 0) {
        SplitJobs jobs;
        uint32_t blocks = 0;
        int c = 0;
        for (; c < count && c < SPLIT_JOBS; ++c) {
            const int64_t n8 = w[c].rows * (w[c].k / 8);
            PTV3_REQUIRE(n8 > 0 && n8 < (1ll << 32), PTV3_ERR_INVALID_ARGUMENT, "fp32 split: a weight of %lld x %d",
                         (long long)w[c].rows, w[c].k);
            if (blocks + (uint64_t)((n8 + 255) / 256) >= (1ull << 31)) break;
            jobs.x[c] = w[c].x;
            jobs.out[c] = (__nv_bfloat16*)w[c].out;
            jobs.n8[c] = (uint32_t)n8;
            jobs.first[c] = blocks;
            jobs.k[c] = w[c].k;
            blocks += (uint32_t)((n8 + 255) / 256);
        }
        jobs.count = c;
        split_weights_kernel<<<blocks, 256, 0, stream>>>(jobs);
        count_launches(1);
        const int rc = check_launch("fp32 split of weights");
        if (rc != PTV3_OK) return rc;
        w += c;
        count -= c;
    }
    return PTV3_OK;
}

}  // namespace ptv3

extern "C" int ptv3_split_f32(const float* x, int64_t rows, int k, int weight, void* out, void* stream)
{
    using namespace ptv3;
    PTV3_REQUIRE(rows >= 0 && k >= 8 && k % 8 == 0, PTV3_ERR_INVALID_ARGUMENT, "ptv3_split_f32: bad sizes");
    if (rows == 0) return PTV3_OK;
    PTV3_REQUIRE(x && out && (((uintptr_t)x | (uintptr_t)out) & 15) == 0, PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_split_f32: tensors must be 16-byte aligned");
    if (!weight) return launch_split_f32(x, rows, k, out, (cudaStream_t)stream);
    const SplitWeight w{x, rows, k, out};
    return launch_split_weights(&w, 1, (cudaStream_t)stream);
}
