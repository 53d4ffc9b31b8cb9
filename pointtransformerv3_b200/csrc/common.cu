#include "common.cuh"
#include <stdarg.h>
#include <atomic>
#include <chrono>
#include "../../include/ptv3_b200.h"

namespace ptv3 {

static thread_local char g_err[512] = "";
static std::atomic<long long> g_launches{0};

static __global__ void status_report_kernel(const uint32_t* status, int64_t* host)
{
    host[0] = *status;
    __threadfence_system();
    *reinterpret_cast<volatile int64_t*>(&host[1]) = 1;
    __threadfence_system();
}

void count_launches(int n) { g_launches.fetch_add(n, std::memory_order_relaxed); }
long long launches() { return g_launches.load(std::memory_order_relaxed); }

void set_error(const char* fmt, ...)
{
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

int check_launch(const char* what)
{
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("%s: %s", what, cudaGetErrorString(e));
        return PTV3_ERR_CUDA;
    }
    return PTV3_OK;
}

}  // namespace ptv3

extern "C" const char* ptv3_last_error(void) { return ptv3::g_err; }
extern "C" int ptv3_version(void) { return 1; }
extern "C" long long ptv3_launch_count(void) { return ptv3::launches(); }
namespace ptv3 {
int host_wait(const int64_t* word, cudaStream_t stream)
{
    const volatile int64_t* w = word;
    if (*w) return PTV3_OK;
    const auto began = std::chrono::steady_clock::now();
    for (uint32_t i = 1; !*w; ++i) {
        if ((i & 4095) == 0 && std::chrono::steady_clock::now() - began > std::chrono::seconds(2)) {
            if (cudaStreamSynchronize(stream) != cudaSuccess) return check_launch("ptv3_host_wait");
            PTV3_REQUIRE(*w, PTV3_ERR_CUDA, "the kernels of this call finished without reporting their result");
        }
    }
    return PTV3_OK;
}
}  // namespace ptv3

extern "C" int ptv3_host_wait(const int64_t* word, void* stream)
{
    PTV3_REQUIRE(word, PTV3_ERR_INVALID_ARGUMENT, "ptv3_host_wait: null pointer");
    return ptv3::host_wait(word, (cudaStream_t)stream);
}
extern "C" int ptv3_status_report(const uint32_t* status, int64_t* host, void* stream)
{
    PTV3_REQUIRE(status && host, PTV3_ERR_INVALID_ARGUMENT, "ptv3_status_report: null pointer");
    ptv3::status_report_kernel<<<1, 1, 0, (cudaStream_t)stream>>>(status, host);
    ptv3::count_launches(1);
    return ptv3::check_launch("ptv3_status_report");
}
extern "C" int ptv3_status_reset(uint32_t* status, void* stream)
{
    PTV3_REQUIRE(status != nullptr, PTV3_ERR_INVALID_ARGUMENT, "ptv3_status_reset: null pointer");
    if (cudaMemsetAsync(status, 0, sizeof(uint32_t), (cudaStream_t)stream) != cudaSuccess)
        return ptv3::check_launch("ptv3_status_reset");
    return PTV3_OK;
}
